"""Problems at the edges of what the non-uniform FFT of DChi2 (dchi2_engine 0)
takes: values that a flagged visibility may hold, channels without any."""

import dataclasses

import numpy as np
import pytest

from gpuvmem_gb300 import synth

pytestmark = pytest.mark.gpu


def _data(n=128, nchan=1, seed=1):
    return synth.generate(synth.small_config(n=n, nchan=nchan, seed=seed, n_ant=9, n_times=31))


def _gradient(data, engine=0, **kw):
    import gpuvmem_gb300 as gv
    import torch
    prob = gv.Problem(data, [gv.term("Chi2", 1.0)], engine=engine, **kw)
    img = prob.initial_image()
    img[0] += (200.0 * torch.rand(img[0].shape, generator=torch.Generator().manual_seed(3)) ** 6).cuda()
    prob.chi2(img)
    return prob.dchi2(img)


@pytest.mark.parametrize("n", [64, 128])
def test_flagged_visibility_without_a_w(n):
    """A NaN in the w of a visibility of weight 0 changes nothing."""
    import torch
    data = _data(n)
    w = data.weight.copy()
    w[17] = 0.0
    uvw = data.uvw_m.copy()
    ref = _gradient(dataclasses.replace(data, weight=w, uvw_m=uvw))
    uvw = uvw.copy()
    uvw[17, 2] = np.nan
    got = _gradient(dataclasses.replace(data, weight=w, uvw_m=uvw))
    assert ref.any() and torch.equal(got, ref)


@pytest.mark.parametrize("empty", [0, 1, 2])
def test_channel_without_visibilities(empty):
    """It adds nothing to a normalised gradient (1/V is not taken), as in the
    GEMM engine; the other channels' sums agree with it to the GEMM's accuracy."""
    data = _data(128, nchan=3)
    off = data.chan_off
    keep = np.ones(data.weight.size, bool)
    keep[off[empty]:off[empty + 1]] = False
    sizes = np.diff(off)
    sizes[empty] = 0
    data = dataclasses.replace(data, uvw_m=data.uvw_m[keep], vo=data.vo[keep],
                               weight=data.weight[keep],
                               chan_off=np.concatenate([[0], np.cumsum(sizes)]).astype(off.dtype))
    got, ref = (_gradient(data, engine=e, normalize=True)[0] for e in (0, 2))
    assert ref.abs().max() > 0
    assert (got - ref).abs().max() <= 1e-5 * ref.abs().max()
