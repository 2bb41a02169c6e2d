"""Candidates of a problem with thousands of channels: channels times images pass
65,535, the limit of a grid's second dimension."""

import pytest

from gpuvmem_gb300 import synth

pytestmark = pytest.mark.gpu


def test_candidates_of_5000_channels():
    import gpuvmem_gb300 as gv
    import torch
    data = synth.generate(synth.small_config(n=16, nchan=5000, seed=2, n_ant=4, n_times=2))
    prob = gv.Problem(data, [gv.term("Chi2", 1.0)])
    imgs = prob.initial_image()[None].repeat(16, 1, 1, 1)
    imgs[:, 0] += torch.rand((16, 16, 16), device="cuda") ** 6
    many = prob.objective_many(imgs)
    assert many == [prob.objective(i.clone())[0] for i in imgs]
