"""Convolutions of tensors with more than 2^31 elements.  All operands are -1, 0
or 1 and the sums stay below 2^24, so every result is exact in FP32; batches
but the first and the last are zero."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

B, C, H = 33, 64, 1024  # 33 * 64 * 2^20 elements: 2^31 lies in the last batch


def _ternary(shape, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(-1, 2, shape, generator=g, device="cuda").float()


def _ends(channels, seed):
    import torch
    x = torch.zeros((B, channels, H, H), dtype=torch.float32, device="cuda")
    x[0], x[-1] = _ternary(x.shape[1:], seed), _ternary(x.shape[1:], seed + 1)
    return x


def test_forward_result():
    import torch
    from gpuvmem_gb300 import unet
    x, w, b = _ends(1, 1), _ternary((C, 1, 3, 3), 3), _ternary((C,), 4)
    y = unet.conv2d_forward(x, w, b, 3, False)
    for k in (0, B - 1):
        ref = torch.nn.functional.conv2d(x[k:k + 1].double(), w.double(), b.double(), padding=1)
        assert torch.equal(y[k:k + 1].double(), ref)
    assert torch.equal(y[1:-1], b[None, :, None, None].expand_as(y[1:-1]))


def test_forward_and_backward_operands():
    import torch
    from gpuvmem_gb300 import unet
    x, dz = _ends(C, 5), _ends(C, 7)
    w, b = _ternary((C, C, 3, 3), 9), _ternary((8,), 10)
    y = unet.conv2d_forward(x, w[:8], b, 3, False)
    dx, dw, db = unet.conv2d_backward(x, w, dz, 3)
    dw_ref, db_ref = torch.zeros_like(w, dtype=torch.float64), torch.zeros(C, dtype=torch.float64)
    for k in (0, B - 1):
        xk, zk = x[k:k + 1].double(), dz[k:k + 1].double()
        ref = torch.nn.functional.conv2d(xk, w[:8].double(), b.double(), padding=1)
        assert torch.equal(y[k:k + 1].double(), ref)
        ref = torch.nn.functional.conv_transpose2d(zk, w.double(), padding=1)
        assert torch.equal(dx[k:k + 1].double(), ref)
        # one tap at a time: products of the shifted planes
        xp = torch.nn.functional.pad(xk[0], (1, 1, 1, 1))
        for t in range(9):
            s = xp[:, t // 3:t // 3 + H, t % 3:t % 3 + H].reshape(C, -1)
            dw_ref[:, :, t // 3, t % 3] += zk[0].reshape(C, -1) @ s.T
        db_ref += zk.sum((0, 2, 3)).cpu()
    assert not dx[1:-1].any()
    assert torch.equal(dw.double(), dw_ref)
    assert np.array_equal(db.double().cpu().numpy(), db_ref.numpy())


@pytest.fixture(autouse=True)
def _give_back():
    import torch
    yield
    torch.cuda.empty_cache()
