"""Batches whose planes (batch x channels) pass 65,535, the limit of a grid's
second dimension: 256 skies of a network with 256 channels at its deepest level,
and a bias gradient of more channels than that."""

import numpy as np
import pytest

import cnn_oracle as CO
from test_gpu_cnn_tiles import _layers

pytestmark = pytest.mark.gpu

SIDE, BASE, LEVELS = 32, 16, 5


def test_network_of_65536_planes():
    """Each channel takes one tap of weight 1 (the last layer all channels), of
    integer images: activations are exact in FP32 whatever the order of a sum, so
    the whole batch, its halves and the oracle give the same numbers.  Only the
    sums over pixels of the weight gradients round: at most 2^18 terms."""
    import torch
    from gpuvmem_gb300 import unet
    batch = 256
    net = unet.UNet(SIDE, in_channels=2, base_channels=BASE, levels=LEVELS, max_batch=batch, seed=3)
    rng = np.random.default_rng(1)
    theta = np.zeros(net.nparams, np.float32)
    for cin, cout, ks, w, _ in _layers(BASE, LEVELS):
        for n in range(cout):
            taps = rng.permutation(cin * ks * ks)[:1 if ks == 3 else None]
            theta[w + n * cin * ks * ks + taps] = 1.0
    net.set_params(torch.from_numpy(theta).cuda())
    x = torch.from_numpy(rng.integers(-2, 5, (batch, 2, SIDE, SIDE)).astype(np.float32)).cuda()
    t = torch.from_numpy(rng.integers(-2, 3, (batch, 1, SIDE, SIDE)).astype(np.float32)).cuda()
    out = net.forward(x)
    assert out.any()
    ends = x[[0, batch - 1]].cpu().numpy()
    ref = CO.UNet(SIDE, 2, BASE, LEVELS).forward(theta.astype(np.float64), ends)
    ref = ref[0] if isinstance(ref, tuple) else ref
    assert np.array_equal(out[[0, batch - 1]].cpu().numpy(), ref.astype(np.float32))
    loss = net.loss_grad(x, t)
    g = net.grads()
    losses, halves = [], []
    for h in (slice(0, batch // 2), slice(batch // 2, batch)):
        assert torch.equal(net.forward(x[h]), out[h])
        losses.append(net.loss_grad(x[h], t[h]))
        halves.append(net.grads())
    assert loss == pytest.approx(sum(losses) / 2, rel=1e-12)
    mean = (halves[0] + halves[1]) / 2
    assert (g - mean).abs().max() <= 1e-5 * mean.abs().max()


def test_bias_gradient_of_65536_channels():
    import torch
    from gpuvmem_gb300 import unet
    cout = 65537
    g = torch.Generator().manual_seed(2)
    x = torch.randint(-1, 2, (1, 1, 8, 8), generator=g).float().cuda()
    dz = torch.randint(-1, 2, (1, cout, 8, 8), generator=g).float().cuda()
    w = torch.ones((cout, 1, 1, 1), device="cuda")
    dx, dw, db = unet.conv2d_backward(x, w, dz, 1)
    assert torch.equal(db, dz.sum((0, 2, 3)))
    assert torch.equal(dw.view(-1), (dz * x).sum((0, 2, 3)))
    assert torch.equal(dx, dz.sum(1, keepdim=True))


def test_weight_gradient_of_more_weights_than_the_splits_scratch():
    """512 x 1024 channels: 4.7M weights, beyond the 4M floats that the splits
    otherwise share.  Operands -1, 0 and 1: exact sums."""
    import torch
    from gpuvmem_gb300 import unet
    g = torch.Generator().manual_seed(4)
    x = torch.randint(-1, 2, (1, 512, 8, 8), generator=g).float().cuda()
    dz = torch.randint(-1, 2, (1, 1024, 8, 8), generator=g).float().cuda()
    w = torch.randint(-1, 2, (1024, 512, 3, 3), generator=g).float().cuda()
    dx, dw, db = unet.conv2d_backward(x, w, dz, 3)
    ref = torch.nn.functional.conv2d(x.double().transpose(0, 1), dz.double().transpose(0, 1),
                                     padding=1).transpose(0, 1)
    assert torch.equal(dw.double(), ref)
    assert torch.equal(db, dz.sum((0, 2, 3)))
    assert torch.equal(dx.double(), torch.nn.functional.conv_transpose2d(dz.double(), w.double(),
                                                                         padding=1))
