"""The U-Net's pooling, upsampling and head passes, and the convolution's masked
output, against the library operations that they stand for: the same roundings
in the same order, so the same bits.  Odd sizes, ties, zeros, NaN and infinities.
"""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1, 8), (2, 3, 5, 8), (1, 7, 37, 24), (3, 16, 33, 32), (1, 2, 300, 64), (2, 5, 9, 200)]


def _data(torch, shape, seed, special=True):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(shape, generator=g, device="cuda").mul(2).round().mul(0.5).to(torch.bfloat16)  # many ties and zeros
    if special and x.numel() > 64:
        flat = x.reshape(-1)
        at = torch.randint(0, flat.numel(), (8,), generator=g, device="cuda")
        flat[at[:3]], flat[at[3:5]], flat[at[5:]] = float("nan"), float("inf"), float("-inf")
    return x


def _same(torch, a, b):
    return torch.equal(torch.nan_to_num(a.float(), nan=123.0), torch.nan_to_num(b.float(), nan=123.0)) and \
        torch.equal(a.isnan(), b.isnan())


@pytest.mark.parametrize("B,h,w,C", SIZES)
def test_pool_and_upcat(cuda, B, h, w, C):
    torch = cuda
    from iterative_tomographic_reconstruction_algorithms_b200 import nn
    F, bf = torch.nn.functional, torch.bfloat16
    X = _data(torch, (B, 2 * h, 2 * w, C), 1)
    Y = torch.empty((B, h, w, C), dtype=bf, device="cuda")
    assert nn.lib.tomo_nn_pool(nn._p(X), B, h, w, C, nn._p(Y), nn._stream(X)) == 0
    Xt = X.permute(0, 3, 1, 2).detach().requires_grad_(True)
    Yt = F.max_pool2d(Xt, 2)
    assert _same(torch, Y, Yt.permute(0, 2, 3, 1))
    # backward, with the skip's gradient a slice of wider pixels
    dP, wide = _data(torch, Y.shape, 2, False), _data(torch, (B, 2 * h, 2 * w, C + 16), 3, False)
    dS = wide[..., 16:]
    dZ = torch.empty_like(X)
    assert nn.lib.tomo_nn_pool_bwd(nn._p(X), nn._p(dP), nn._p(dS), C + 16, B, h, w, C, nn._p(dZ), nn._stream(X)) == 0
    Yt.backward(dP.permute(0, 3, 1, 2))
    ref = torch.where(X > 0, Xt.grad.permute(0, 2, 3, 1) + dS, torch.zeros_like(X))
    assert _same(torch, dZ, ref)
    # upsampling beside a skip, and its gradient
    U = _data(torch, (B, h, w, C), 4)
    cat = torch.empty((B, 2 * h, 2 * w, 2 * C), dtype=bf, device="cuda")
    assert nn.lib.tomo_nn_upcat(nn._p(U), nn._p(X), B, h, w, C, C, nn._p(cat), nn._stream(X)) == 0
    Ut = U.permute(0, 3, 1, 2).detach().requires_grad_(True)
    up = F.interpolate(Ut, scale_factor=2, mode="nearest")
    assert _same(torch, cat, torch.cat([up.permute(0, 2, 3, 1), X], dim=-1))
    d = torch.randn(cat.shape, device="cuda").to(bf)
    dU = torch.empty_like(U)
    assert nn.lib.tomo_nn_up_bwd(nn._p(d), 2 * C, nn._p(U), B, h, w, C, nn._p(dU), nn._stream(X)) == 0
    up.backward(d[..., :C].permute(0, 3, 1, 2))
    assert _same(torch, dU, torch.where(U > 0, Ut.grad.permute(0, 2, 3, 1), torch.zeros_like(U)))


@pytest.mark.parametrize("P,C", [(1, 8), (37, 32), (5000, 40), (777, 1024)])
def test_head_gradient(cuda, P, C):
    torch = cuda
    from iterative_tomographic_reconstruction_algorithms_b200 import nn
    g = torch.Generator(device="cuda").manual_seed(P)
    d = torch.randn(P, generator=g, device="cuda")
    W = torch.randn((8, 1, C), generator=g, device="cuda")
    X = _data(torch, (P, C), 5)
    _, Wt = nn.prepare_weights(W)
    dZ = torch.empty((P, 8), dtype=torch.bfloat16, device="cuda")
    assert nn.lib.tomo_nn_pad8(nn._p(d), P, nn._p(dZ), nn._stream(d)) == 0
    assert torch.equal(dZ[:, 0], d.to(torch.bfloat16)) and not dZ[:, 1:].any()
    dX = torch.empty_like(X)
    assert nn.lib.tomo_nn_head_bwd(nn._p(dZ), nn._p(Wt), nn._p(X), P, C, nn._p(dX), nn._stream(d)) == 0
    ref = nn.gemm(dZ, Wt.reshape(C, 8), out_dtype=torch.bfloat16)
    assert torch.equal(dX, torch.where(X > 0, ref, torch.zeros_like(ref)))  # one product per element: exact


@pytest.mark.parametrize("B,H,W,Cin,Cout", [(1, 5, 7, 16, 8), (2, 17, 9, 32, 32), (1, 33, 18, 64, 200), (1, 8, 16, 24, 12)])
def test_masked_convolution(cuda, B, H, W, Cin, Cout):
    torch = cuda
    from iterative_tomographic_reconstruction_algorithms_b200 import nn
    X, Wd = _data(torch, (B, H, W, Cin), 6, False), _data(torch, (Cout, 3, 3, Cin), 7, False)
    mask = _data(torch, (B, H, W, Cout), 8)
    out = torch.empty_like(mask)
    assert nn.lib.tomo_nn_conv3x3_masked(nn._p(X), B, H, W, Cin, nn._p(Wd), Cout, nn._p(mask), nn._p(out),
                                         nn._stream(X)) == 0
    full = nn.conv3x3(X, Wd)
    assert torch.equal(out, torch.where(mask > 0, full, torch.zeros_like(full)))
