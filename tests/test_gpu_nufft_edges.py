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


def _pairs_of_the_series(data):
    """Pairs of terms after which the w series leaves no more than 3e-7
    (2 (A/2)^2p / (2p)! with A the largest phase), or 0 beyond 4."""
    lam = np.repeat(299792458.0 / np.asarray(data.freqs, np.float64), np.diff(data.chan_off))
    w = np.abs(data.uvw_m[:, 2] / lam).max()
    half = [max(x, data.N - 1 - x) * abs(d) * np.pi / 180.0
            for x, d in ((int(data.xobs), data.DELTAX), (int(data.yobs), data.DELTAY))]
    r2 = half[0] ** 2 + half[1] ** 2
    a = 2.0 * np.pi * w * r2 / (1.0 + np.sqrt(1.0 - r2))
    for p in range(1, 5):
        if 2.0 * np.prod([0.5 * a / k for k in range(1, 2 * p + 1)]) <= 3e-7:
            return p
    return 0


def test_engine_that_runs():
    """The pairs reported are the series' own, from 1 to 4, and 0 where more are
    needed or a direct engine is asked for."""
    import gpuvmem_gb300 as gv
    seen = set()
    for wscale in (0.0, 1.0, 30.0, 300.0, 1500.0, 2600.0, 1e5):
        data = _data(128, seed=5)
        data = dataclasses.replace(data, uvw_m=data.uvw_m * np.array([1.0, 1.0, wscale]))
        want = _pairs_of_the_series(data)
        prob = gv.Problem(data, [gv.term("Chi2", 1.0)])
        assert prob.dchi2_pairs == want
        seen.add(want)
        prob.close()
    assert seen == {0, 1, 2, 3, 4}
    for engine in (1, 2):
        assert gv.Problem(_data(128), [gv.term("Chi2", 1.0)], engine=engine).dchi2_pairs == 0


@pytest.mark.parametrize("n", [16, 64, 256, 1024])
def test_default_engine(n):
    import gpuvmem_gb300 as gv
    prob = gv.Problem(_data(n, nchan=2), [gv.term("Chi2", 1.0)])
    assert 1 <= prob.dchi2_pairs <= 4


def _with_pairs(data, uvscale, pairs):
    """The data with their uv scaled, and their w so that the series takes `pairs`."""
    for wscale in 10.0 ** np.arange(-4.0, 4.0, 0.05):
        d = dataclasses.replace(data, uvw_m=data.uvw_m * np.array([uvscale, uvscale, wscale]))
        if _pairs_of_the_series(d) == pairs:
            return d
    raise AssertionError(f"no scale of w takes {pairs} pairs")


def _against_simt(data, pairs):
    """Tolerance as for the other comparisons with the SIMT sums."""
    import gpuvmem_gb300 as gv
    from test_gpu_nufft import TOL
    prob = gv.Problem(data, [gv.term("Chi2", 1.0)])
    assert prob.dchi2_pairs == pairs
    prob.close()
    got, ref = (_gradient(data, engine=e)[0] for e in (0, 1))
    assert ref.abs().max() > 0
    assert (got - ref).abs().max() <= TOL * ref.abs().max()


@pytest.mark.parametrize("n,pairs,uvscale", [(1024, 1, 1.0), (1024, 4, 6.0), (2048, 2, 1.0),
                                             (2048, 3, 6.0), (4096, 1, 1.0), (4096, 2, 0.3)])
def test_large_sides(n, pairs, uvscale):
    """The largest sides as a non-uniform FFT: the small arrays' own w needs more
    pairs than there are from 2048^2 on."""
    _against_simt(_with_pairs(_data(n, nchan=2), uvscale, pairs), pairs)


def test_channel_groups():
    """4096^2 with all rows of the grid and four pairs: 1.07 GB a channel, so that
    five channels go in two groups of at most 4 GB."""
    _against_simt(_with_pairs(_data(4096, nchan=5), 6.0, 4), 4)
