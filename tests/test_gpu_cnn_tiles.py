"""The staging of the convolution GEMMs' tiles where its units and tiles end:
channel counts whose taps straddle the chunks of 64 k, ragged column tiles,
1 x 1 taps, and networks whose packed weights are taken in tiles of every
width, against the FP64 oracle."""

import numpy as np
import pytest

import cnn_oracle as CO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Cin,Cout,H,ks", [
    (1, 1, 1, 8, 3),       # nine k, one column
    (1, 43, 130, 8, 3),    # 387 k: a last chunk of three; columns of two tiles and two more
    (3, 15, 17, 24, 3),    # 135 k; row tiles that end inside a plane and in the next batch
    (1, 70, 3, 8, 1),      # 1 x 1: a last chunk of six
    (2, 5, 66, 40, 1),
])
def test_conv_tiles_match_oracle(B, Cin, Cout, H, ks):
    import torch
    from gpuvmem_gb300 import unet
    rng = np.random.default_rng(Cin + 1000 * Cout + H)

    def exact(shape, scale=1.0):
        return CO.bf16(rng.normal(0, scale, shape).astype(np.float32)).astype(np.float32)

    x, w, dz = exact((B, Cin, H, H)), exact((Cout, Cin, ks, ks), 0.2), exact((B, Cout, H, H))
    b = rng.normal(0, 0.1, Cout).astype(np.float32)
    tx, tw, tb, tz = (torch.from_numpy(a).cuda() for a in (x, w, b, dz))
    got = [unet.conv2d_forward(tx, tw, tb, ks, False)] + list(unet.conv2d_backward(tx, tw, tz, ks))
    ref = [CO.conv_forward(x, w, b, ks, False)] + list(CO.conv_backward(x, w, dz, ks))
    # operands are exact in BF16: only the FP32 accumulation of at most 4800
    # products, whose error grows like the root of their number
    for g, r in zip(got, ref):
        assert np.abs(g.cpu().numpy() - r).max() <= 1e-5 * max(1.0, np.abs(r).max())


def _layers(base, levels):
    """(cin, cout, taps a side, offset of the weights, of the bias), in order."""
    width = [base << l for l in range(levels)]
    shapes = []
    for l in range(levels):
        shapes += [(width[l - 1] if l else 2, width[l], 3), (width[l], width[l], 3)]
    for l in range(levels - 2, -1, -1):
        shapes += [(width[l + 1] + width[l], width[l], 3), (width[l], width[l], 3)]
    shapes.append((width[0], 1, 1))
    off = 0
    for cin, cout, ks in shapes:
        w = off
        off += cout * cin * ks * ks + cout
        yield cin, cout, ks, w, off - cout


@pytest.mark.parametrize("side,base,levels,batch", [(16, 64, 3, 2), (64, 8, 4, 1), (8, 128, 2, 4)])
def test_networks_of_every_tile_width_match_oracle(side, base, levels, batch):
    """Each channel takes a few taps with weights +-1 of integer images (the last
    layer all channels): every activation and its gradient is exact in FP32, so
    that BF16 rounds the same numbers here and in the oracle and no result
    hangs on a tie.  Only the sums over pixels of the weight gradients round."""
    import torch
    from gpuvmem_gb300 import unet
    net = unet.UNet(side, in_channels=2, base_channels=base, levels=levels, max_batch=batch, seed=3)
    ref = CO.UNet(side, 2, base, levels)
    rng = np.random.default_rng(1)
    theta = np.zeros(net.nparams, np.float32)
    for cin, cout, ks, w, b in _layers(base, levels):
        for n in range(cout):
            taps = rng.permutation(cin * ks * ks)[:4 if ks == 3 else None]
            theta[w + n * cin * ks * ks + taps] = rng.choice([-1.0, 1.0], taps.size, p=[0.3, 0.7])
    assert b + 1 == net.nparams
    net.set_params(torch.from_numpy(theta).cuda())
    x = rng.integers(-2, 5, (batch, 2, side, side)).astype(np.float32)
    t = rng.integers(-2, 3, (batch, 1, side, side)).astype(np.float32)
    loss_ref, g_ref, out_ref = ref.loss_grad(theta.astype(np.float64), x, t)
    tx, tt = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    assert np.array_equal(net.forward(tx).cpu().numpy(), out_ref.astype(np.float32))
    loss = net.loss_grad(tx, tt)
    g = net.grads().cpu().numpy()
    assert abs(loss - loss_ref) <= 1e-6 * loss_ref
    # FP32 sums of at most 4096 terms
    assert np.abs(g - g_ref).max() <= 1e-5 * np.abs(g_ref).max()
    # a second pass gives the same bits: the weight gradients' stream is joined
    net.loss_grad(tx, tt)
    assert np.array_equal(net.grads().cpu().numpy(), g)
