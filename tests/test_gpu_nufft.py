"""DChi2 as a non-uniform FFT (dchi2_engine 0) against the direct sums of the
SIMT engine on the same problem, which agree with 64 bits to 2.5e-7.

Tolerance: the spreading kernel leaves 2e-7 and the w series 3e-7; FP32
spreading and two FFTs add some 5e-7 of the 2-norm, up to 8 times that in the
corners, where the kernel's correction is largest: 5e-6 of the largest value,
half the gradient's parity gate."""

import dataclasses

import numpy as np
import pytest

from gpuvmem_gb300 import synth

pytestmark = pytest.mark.gpu

TOL = 5e-6


def _pair(n, nchan=1, seed=1, wscale=1.0, uvscale=1.0, x0=None, empty=None, **kw):
    import gpuvmem_gb300 as gv
    data = synth.generate(synth.small_config(n=n, nchan=nchan, seed=seed, n_ant=9, n_times=31))
    uvw = data.uvw_m * np.array([uvscale, uvscale, wscale])
    rng = np.random.default_rng(seed)
    w = (data.weight * rng.uniform(0.5, 1.5, data.weight.size)).astype(np.float32)
    w[rng.random(w.size) < 0.05] = 0.0
    if empty is not None:
        w[data.chan_off[empty]:data.chan_off[empty + 1]] = 0.0
    data = dataclasses.replace(data, uvw_m=uvw, weight=w)
    if x0 is not None:
        data = dataclasses.replace(data, xobs=float(x0[0]), yobs=float(x0[1]))
    terms = [gv.term("Chi2", 1.0)]
    return [gv.Problem(data, terms, engine=e, **kw) for e in (0, 1)]


def _image(prob, seed, alpha):
    import torch
    g = torch.Generator().manual_seed(seed)
    img = prob.initial_image()
    img[0] += (200.0 * torch.rand(img[0].shape, generator=g) ** 6).cuda()
    if alpha:
        img[1] = torch.rand(img[1].shape, generator=g).cuda() - 0.3
    return img


def _close(a, b, scale=None):
    scale = b.abs().max().item() if scale is None else scale
    assert scale > 0
    err = (a - b).abs().max().item() / scale
    assert err <= TOL, err


@pytest.mark.parametrize("n", [16, 32, 64, 128, 256, 512, 1024, 2048, 4096])
def test_gradient_every_side(n):
    pa, pb = _pair(n, nchan=2, seed=n)
    ia, ib = _image(pa, 3, False), _image(pb, 3, False)
    assert pa.chi2(ia) == pytest.approx(pb.chi2(ib), rel=1e-9)
    _close(pa.dchi2(ia)[0], pb.dchi2(ib)[0])


@pytest.mark.parametrize("wscale", [0.0, 1.0, 30.0, 300.0, 1500.0, 2600.0])
def test_w_series(wscale):
    """No w-term, then 1 to 4 pairs of terms."""
    pa, pb = _pair(128, seed=5, wscale=wscale)
    ia, ib = _image(pa, 4, False), _image(pb, 4, False)
    pa.chi2(ia)
    pb.chi2(ib)
    _close(pa.dchi2(ia)[0], pb.dchi2(ib)[0])


def test_beyond_the_w_series():
    """A w-term that 4 pairs do not cover keeps the direct-sum engine that the
    problem reports."""
    import gpuvmem_gb300 as gv
    pa, _ = _pair(128, seed=5, wscale=1e5)
    pb = gv.Problem(pa.data, [gv.term("Chi2", 1.0)], engine=pa.info.dchi2_engine)
    ia, ib = _image(pa, 4, False), _image(pb, 4, False)
    pa.chi2(ia)
    pb.chi2(ib)
    _close(pa.dchi2(ia)[0], pb.dchi2(ib)[0])


@pytest.mark.parametrize("uvscale", [0.05, 3.0, 6.0, 12.0])
@pytest.mark.parametrize("n", [32, 128])
def test_coverage(n, uvscale):
    """From a few central cells to beyond the grid's edge, where cells wrap
    round its period and visibilities fall off the grid."""
    pa, pb = _pair(n, seed=7, uvscale=uvscale)
    assert pa.info.nvis_in_grid == pb.info.nvis_in_grid > 0
    ia, ib = _image(pa, 5, False), _image(pb, 5, False)
    pa.chi2(ia)
    pb.chi2(ib)
    _close(pa.dchi2(ia)[0], pb.dchi2(ib)[0])


@pytest.mark.parametrize("x0", [(0, 0), (127, 3), (61.5, 70.25)])
def test_centre(x0):
    pa, pb = _pair(128, seed=9, x0=x0)
    ia, ib = _image(pa, 6, False), _image(pb, 6, False)
    pa.chi2(ia)
    pb.chi2(ib)
    _close(pa.dchi2(ia)[0], pb.dchi2(ib)[0])


@pytest.mark.parametrize("normalize", [False, True])
def test_channels_planes_and_modes(normalize):
    """Three channels, the middle one without a kept visibility: both planes'
    chain rules, the raw channel sums, dirty image, PSF and error maps."""
    import torch
    rng = np.random.default_rng(2)
    gcf = rng.uniform(0.5, 2.0, (128, 128)).astype(np.float32)
    pa, pb = _pair(128, nchan=3, seed=11, empty=1, normalize=normalize, gcf=gcf)
    ia, ib = _image(pa, 7, True), _image(pb, 7, True)
    for flag in (0, 1):
        pa.chi2(ia, flag)
        pb.chi2(ib, flag)
        ga, gb = pa.dchi2(ia, flag), pb.dchi2(ib, flag)
        # the channels' terms of the alpha plane cancel: scale of the I_nu0 sums
        scale = None
        if flag:
            scale = sum((pb.dchi2_channel(c).abs() * (ib[0] * pb.info.fg_scale * 0.02)).max().item()
                        for c in (0, 2))
        _close(ga[flag], gb[flag], scale)
        assert not ga[1 - flag].any()
    for c in (0, 2):
        _close(pa.dchi2_channel(c), pb.dchi2_channel(c))
    assert not pa.dchi2_channel(1).any()
    _close(pa.dirty_image(), pb.dirty_image())
    _close(pa.psf_image(), pb.psf_image())
    ea, eb = pa.error_images(ia), pb.error_images(ib)
    torch.testing.assert_close(ea[0], eb[0], rtol=1e-5, atol=0.0)


def test_repeats_bit_for_bit():
    import torch
    pa, _ = _pair(256, nchan=2, seed=13)
    ia = _image(pa, 8, False)
    pa.chi2(ia)
    g = pa.dchi2(ia)
    for _ in range(3):
        assert torch.equal(pa.dchi2(ia), g)


@pytest.mark.parametrize("nchan,wscale", [(1, 0.0), (1, 1.0), (3, 1.0), (5, 2.0)])
def test_columns_shared_out(nchan, wscale):
    """Sides from 1024 up share the columns' planes out between blocks: one
    plane a column (nothing shared, fewer units than blocks), two (a column in
    two pieces at most) and more than a block's run."""
    import torch
    pa, pb = _pair(1024, nchan=nchan, seed=21, wscale=wscale)
    ia, ib = _image(pa, 9, True), _image(pb, 9, True)
    pa.chi2(ia)
    pb.chi2(ib)
    # one channel is at the reference frequency: its alpha gradient is zero
    for flag in (0, 1) if nchan > 1 else (0,):
        ga, gb = pa.dchi2(ia, flag_opt=flag), pb.dchi2(ib, flag_opt=flag)
        _close(ga[flag], gb[flag])
        assert torch.equal(ga, pa.dchi2(ia, flag_opt=flag))
