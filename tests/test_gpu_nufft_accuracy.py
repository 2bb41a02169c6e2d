"""Dirty images and PSFs of the default DChi2 engine, the non-uniform FFT,
against 64-bit sums over the visibilities.

Tolerance, of the 2-norm: the spreading kernel's truncation leaves 1.5e-7 of
visibilities that do not add up, the FP32 FFTs 1.2e-7 (emulated in 64 bits with
the one and the other); 3e-7 for the two and the w series together, however many
visibilities a tile or a channel holds."""

import dataclasses

import numpy as np
import pytest

from gpuvmem_gb300 import synth

pytestmark = pytest.mark.gpu

TOL = 3e-7
RAD = np.pi / 180.0


def _data(n, nchan, n_ant, n_times, uvscale, wscale):
    """Uneven weights, and noise of the size of the visibilities."""
    d = synth.generate(synth.small_config(n=n, nchan=nchan, seed=1, n_ant=n_ant, n_times=n_times))
    rng = np.random.default_rng(1)
    w = (d.weight * rng.uniform(0.5, 1.5, d.weight.size)).astype(np.float32)
    vo = (d.vo + rng.normal(0, np.abs(d.vo).mean(), d.vo.shape)).astype(np.float32)
    return dataclasses.replace(d, uvw_m=d.uvw_m * np.array([uvscale, uvscale, wscale]), weight=w,
                               vo=vo)


def _sums(d, pix):
    """sum w Re(conj(Vo) e^{2 pi i (x u + y v + (z - 1) w)}) and the same with Vo
    = 1, over the visibilities on the grid, at some pixels."""
    import torch
    n = d.N
    x = torch.from_numpy((pix % n - int(d.xobs)) * d.DELTAX * RAD).cuda()
    y = torch.from_numpy((pix // n - int(d.yobs)) * d.DELTAY * RAD).cuda()
    r2 = x * x + y * y
    z1 = -r2 / (1.0 + torch.sqrt(1.0 - r2))
    out = torch.zeros((2, pix.size), dtype=torch.float64, device="cuda")
    lam = np.float32(299792458.0) / np.repeat(d.freqs.astype(np.float32), np.diff(d.chan_off))
    uvw = d.uvw_m / lam.astype(np.float64)[:, None]
    flip = np.where(uvw[:, 0] > 0.0, -1.0, 1.0)
    u, v, w = uvw[:, 0] * flip, uvw[:, 1] * flip, uvw[:, 2]
    keep = np.ones(u.size, bool)
    for a, delta in ((u, d.DELTAX), (v, d.DELTAY)):
        c = a * (n * delta * RAD)
        c = np.where(c < 0.0, c + n, c)
        keep &= (c >= 0.0) & (c < n)
    wt = d.weight * keep
    for b in range(0, u.size, 4096):
        s = slice(b, b + 4096)
        tu, tv, tw, tf, tt = (torch.from_numpy(np.ascontiguousarray(a[s], np.float64)).cuda()
                              for a in (u, v, w, flip, wt))
        vo = torch.from_numpy(d.vo[s].astype(np.float64)).cuda()
        ph = x[:, None] * tu + y[:, None] * tv + z1[:, None] * tw
        ph = 2.0 * np.pi * (ph - ph.round())
        c, sn = torch.cos(ph), torch.sin(ph)
        out[0] += c @ (tt * vo[:, 0]) + sn @ (tt * vo[:, 1] * tf)
        out[1] += c @ tt
    return out


def _check(*config, pixels=1000):
    import gpuvmem_gb300 as gv
    import torch
    d = _data(*config)
    prob = gv.Problem(d, [gv.term("Chi2", 1.0)])
    assert prob.dchi2_pairs > 0
    rng = np.random.default_rng(0)
    pix = np.unique(np.append(rng.choice(d.N * d.N, min(pixels, d.N * d.N), replace=False),
                              int(d.yobs) * d.N + int(d.xobs)))
    at = torch.from_numpy(pix).cuda()
    for got, ref in zip((prob.dirty_image(), prob.psf_image()), _sums(d, pix)):
        err = ((got.flatten()[at].double() - ref).norm() / ref.norm()).item()
        assert err <= TOL, err


@pytest.mark.parametrize("n,nchan,n_ant,n_times,uvscale,wscale", [
    (16, 1, 30, 240, 1.0, 1.0),
    (32, 1, 30, 240, 6.0, 1.0),       # round the grid's edge
    (128, 4, 20, 120, 1.0, 1.0),
    (128, 1, 30, 240, 1.0, 1500.0),   # three and four pairs
    (128, 1, 30, 240, 1.0, 2600.0),
    (256, 1, 30, 240, 1.0, 1.0),
    (1024, 2, 20, 60, 1.0, 1.0),
])
def test_sizes(n, nchan, n_ant, n_times, uvscale, wscale):
    _check(n, nchan, n_ant, n_times, uvscale, wscale)


@pytest.mark.parametrize("n,uvscale", [(64, 1.0), (64, 0.05), (512, 0.05)])
def test_many_pieces_a_tile(n, uvscale):
    """2.1M visibilities in one channel, thousands of pieces in the densest tiles."""
    _check(n, 1, 60, 1200, uvscale, 1.0, pixels=600)


def test_many_channels():
    """2048 channels of 100 visibilities: the terms of a PSF have one sign, so
    that rounding errors of a sum over channels add up."""
    _check(32, 2048, 5, 10, 1.0, 1.0)
