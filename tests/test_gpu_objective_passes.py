"""The objective's row and column passes at every side, and several images in
one launch, against the FP64 oracle and the single evaluation."""

import dataclasses

import numpy as np
import pytest

import oracle as O
from gpuvmem_gb300 import synth

pytestmark = pytest.mark.gpu

TERMS = [(O.FI_CHI2, 1.0, 0, 0, 0.0, 0.0, 0.0), (O.FI_ENTROPY, 0.01, 0, 0, 0.001, -1.0, 0.0)]


def _image(shape, floor, seed, alpha=False):
    rng = np.random.default_rng(seed)
    img = np.zeros(shape, np.float32)
    img[0] = floor + 500.0 * rng.uniform(0, 1, shape[1:]) ** 6
    if alpha:
        img[1] = rng.uniform(-1, 1, shape[1:])
    return img


@pytest.mark.parametrize("uvscale", [0.1, 1.0, 6.0])
@pytest.mark.parametrize("n", [16, 32, 64, 128, 256, 512, 1024, 2048, 4096])
def test_chi2_every_side(n, uvscale):
    """From a few needed columns to cells at the grid's edge.  The model's FP32
    transform is some 3e-7 off, and so is its part of chi2: 2e-6."""
    import torch
    import gpuvmem_gb300 as gv
    data = synth.generate(synth.small_config(n=n, nchan=2, seed=n, n_ant=7, n_times=13))
    data = dataclasses.replace(data, uvw_m=data.uvw_m * np.array([uvscale, uvscale, 1.0]))
    orc = O.Oracle(data, TERMS)
    prob = gv.Problem(data, [tuple(t) for t in TERMS])
    img = _image((2, n, n), 0.001, n, alpha=n <= 256)
    ref, img_c = orc.chi2(img.copy())
    d = torch.from_numpy(img.copy()).cuda()
    assert abs(prob.chi2(d) - ref) <= 2e-6 * abs(ref)
    np.testing.assert_array_equal(d.cpu().numpy(), img_c)


@pytest.mark.parametrize("n,nchan", [(64, 1), (256, 3), (2048, 4)])
@pytest.mark.parametrize("count", [1, 2, 16, 17, 35])
def test_many_images(n, nchan, count):
    """Counts around the 16 images of a launch, priors on and off, a tensor
    and a list: each value is the single evaluation's."""
    import torch
    import gpuvmem_gb300 as gv
    if n == 2048 and count not in (1, 17):
        pytest.skip("the large side at two counts")
    data = synth.generate(synth.small_config(n=n, nchan=nchan, seed=3, n_ant=8, n_times=20))
    prob = gv.Problem(data, [tuple(t) for t in TERMS] + [gv.term("TotalSquaredVariation", 1e-4)])
    imgs = torch.stack([torch.from_numpy(_image((2, n, n), 0.001, 10 + k, alpha=True))
                        for k in range(min(count, 5))]).cuda()
    imgs = imgs[torch.arange(count) % imgs.shape[0]].contiguous()
    before = imgs.clone()
    for it in (0, 1):
        prob.set_iteration(it)
        for batch in (imgs, [i for i in imgs]):
            got = prob.objective_many(batch, flag_opt=1)
            assert torch.equal(imgs, before)
            single = [prob.objective(imgs[k].clone(), 1)[0] for k in range(min(count, 5))]
            assert got == [single[k % 5] for k in range(count)]
