"""Sequential FP32 sums in parallel (seqsum.cuh), through the weighting schemes
and the set-up's weight sum, bit for bit against the sequential restatement."""

import dataclasses

import numpy as np
import pytest

import weights_oracle as W
from gpuvmem_gb300 import synth

pytestmark = pytest.mark.gpu

RPDEG = np.pi / 180.0


def _weights(kind, n, rng):
    return {"equal": np.full(n, 1e6), "uniform": rng.random(n) + 0.5,
            "wide": 10.0 ** rng.uniform(-6, 6, n),  # leaves binades, rounds halves
            "halves": rng.integers(0, 64, n) / 8.0,
            "zeros": np.where(rng.random(n) < 0.9, 0.0, 1e6 * rng.random(n)),
            "negative": rng.normal(0, 1, n), "tiny": rng.random(n) * 1e-35}[kind].astype(np.float32)


@pytest.mark.parametrize("kind", ["equal", "uniform", "wide", "halves", "zeros", "negative", "tiny"])
@pytest.mark.parametrize("counts", [(1,), (8191, 0, 8193), (30000, 1, 17000)])
def test_schemes(kind, counts):
    import gpuvmem_gb300 as gv
    rng = np.random.default_rng([len(counts), len(kind)])
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    V, M, cell = int(off[-1]), 64, 0.05 / 3600.0
    freqs = np.linspace(220e9, 240e9, len(counts)).astype(np.float32)
    uvw = rng.normal(0, 150.0, (V, 3))  # some beyond the grid's edge
    w = _weights(kind, V, rng)
    du = 1.0 / (M * (RPDEG * -cell))
    dv = 1.0 / (M * (RPDEG * cell))
    for scheme in ("uniform", "briggs"):
        with np.errstate(divide="ignore", invalid="ignore", over="ignore", under="ignore"):
            ref = W.apply(scheme, uvw, w, freqs, off, M, M, du, dv, 0.5)
        got = gv.apply_weighting(scheme, 0.5, M, M, -cell, cell, freqs, off, uvw, w)
        assert np.array_equal(got, ref, equal_nan=True), (scheme, kind)
        # channels whose arrays do not follow one another
        chans = [(uvw[a:b].copy(), w[a:b].copy()) for a, b in zip(off[:-1], off[1:])]
        import ctypes as C
        cd = (gv.ChannelDesc * len(counts))()
        out = [np.empty(n, np.float32) for n in counts]
        outs = (C.c_void_p * len(counts))(*[o.ctypes.data for o in out])
        for c, (u, x) in enumerate(chans):
            cd[c] = gv.ChannelDesc(float(freqs[c]), counts[c],
                                   u.ctypes.data_as(C.POINTER(C.c_double)), None,
                                   x.ctypes.data_as(C.POINTER(C.c_float)))
        gv.check(gv.lib().gv_apply_weighting(gv.WEIGHTING[scheme], 0.5, M, M, -cell, cell,
                                             len(counts), cd, outs, None))
        assert np.array_equal(np.concatenate(out), ref, equal_nan=True)


@pytest.mark.parametrize("kind", ["equal", "uniform", "wide", "halves"])
def test_set_up_sum(kind):
    import gpuvmem_gb300 as gv
    data = synth.generate(synth.small_config(n=64, nchan=3, seed=4, n_ant=20, n_times=60))
    w = _weights(kind, data.weight.size, np.random.default_rng(8))
    prob = gv.Problem(dataclasses.replace(data, weight=w), [gv.term("Chi2", 1.0)])
    ref = np.float32(0.0)
    for c in range(3):
        o, e = data.chan_off[c], data.chan_off[c + 1]
        ref = np.float32(ref + np.cumsum(w[o:e], dtype=np.float32)[-1])
    assert np.float32(prob.info.sum_weights).tobytes() == ref.tobytes()
