"""Host arrays of the weighting that lie one after another without being one
array."""

import ctypes as C
import mmap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [(), (0,), (1,), (0, 1)])
def test_neighbouring_arrays_pinned_apart(pinned):
    """The weights of two channels in one mapping whose halves are pinned each by
    itself, or one of them alone: the result of ordinary arrays, in place too."""
    import gpuvmem_gb300 as gv
    import torch
    n, M, cell = 1 << 20, 64, 0.05 / 3600.0
    half = 4 * n
    rt = torch.cuda.cudart()
    torch.cuda.synchronize()
    mem = mmap.mmap(-1, 2 * half)
    w = np.frombuffer(mem, np.float32)
    rng = np.random.default_rng(1)
    uvw = rng.normal(0, 150.0, (2 * n, 3))
    weights = (rng.random(2 * n) + 0.5).astype(np.float32)
    freqs = np.array([220e9, 230e9], np.float32)
    off = np.array([0, n, 2 * n], np.int64)
    ref = gv.apply_weighting("uniform", 0.0, M, M, -cell, cell, freqs, off, uvw, weights)
    w[:] = weights
    for h in pinned:
        assert int(rt.cudaHostRegister(w.ctypes.data + h * half, half, 0)) == 0
    try:
        cd, outs = (gv.ChannelDesc * 2)(), (C.c_void_p * 2)()
        for c in range(2):
            cd[c] = gv.ChannelDesc(float(freqs[c]), n,
                                   uvw[c * n:].ctypes.data_as(C.POINTER(C.c_double)), None,
                                   w[c * n:].ctypes.data_as(C.POINTER(C.c_float)))
            outs[c] = w[c * n:].ctypes.data
        gv.check(gv.lib().gv_apply_weighting(gv.WEIGHTING["uniform"], 0.0, M, M, -cell, cell, 2,
                                             cd, outs, None))
        assert np.array_equal(w, ref, equal_nan=True)
    finally:
        torch.cuda.synchronize()
        for h in pinned:
            rt.cudaHostUnregister(w.ctypes.data + h * half)
