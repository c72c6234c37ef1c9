"""The tensor-core kernels' pipelines over many rounds: convolutions whose CTAs go
through several groups of tiles (accumulator sets and patch slots used again, both
issuing warps at work), and weight gradients whose pixels are split into ranges
that start inside an image or a row and are added afterwards; against FP64 torch
on the same BF16 operands.

Tolerances.  Convolution: 9 Cin / 16 <= 72 groups of 16 products (225 for 392
channels) are added into an FP32 accumulator, each addition off by at most 2^-23
of a running sum within the largest output's magnitude, so 72 x 2^-23 = 8.6e-6
of it.  Weight gradient: a range holds at most P / (16 S) + 4 groups and S <= 8
ranges are added in FP32: (P / (16 S) + 4 + S) x 2^-23 of the largest entry.
"""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W,Cin,Cout", [
    # resident weights, two issuing warps: 5, 9 and 3 groups per CTA, odd sides
    (1, 320, 321, 32, 32), (2, 270, 331, 16, 24), (3, 143, 131, 64, 32),
    # resident, one issuing warp; two taps to an MMA (9 groups for 8 patch slots)
    (1, 290, 293, 32, 96), (2, 300, 299, 8, 32), (2, 177, 203, 24, 40),
    # streamed weights, two tiles to a stage; several output blocks; two channel passes
    (2, 270, 250, 128, 64), (1, 199, 201, 64, 200), (1, 270, 260, 392, 40)])
def test_conv3x3_many_groups(cuda, B, H, W, Cin, Cout):
    torch = cuda
    import torch.nn.functional as F
    from iterative_tomographic_reconstruction_algorithms_b200 import nn
    g = torch.Generator().manual_seed(B * H + W + Cin + Cout)
    X = torch.randn((B, H, W, Cin), generator=g).to(torch.bfloat16).cuda()
    Wt = torch.randn((Cout, 3, 3, Cin), generator=g).to(torch.bfloat16).cuda()
    b = torch.randn((Cout,), generator=g).cuda()
    ref = F.conv2d(X.double().permute(0, 3, 1, 2), Wt.double().permute(0, 3, 1, 2), b.double(), padding=1).permute(0, 2, 3, 1)
    tol = (9 * Cin / 16 if Cin > 128 else 72) * 2.0 ** -23 * float(ref.abs().max())
    Y = nn.conv3x3(X, Wt, b, out_dtype=torch.float32)
    Yr = nn.conv3x3(X, Wt, b, relu=True)
    nn.check_status()
    assert float((Y.double() - ref).abs().max()) <= tol
    assert torch.equal(Yr, Y.clamp(min=0).to(torch.bfloat16))
    # masked form: the result kept where the mask is > 0
    if Cout % 8 == 0:
        mask = torch.randn((B, H, W, Cout), generator=g).to(torch.bfloat16).cuda()
        Yn = nn.conv3x3(X, Wt)
        Wd = Wt.reshape(Cout, 9, Cin)
        Ym = nn._conv3x3_dx(X, Wd, mask)
        nn.check_status()
        assert torch.equal(Ym, torch.where(mask > 0, Yn, torch.zeros_like(Yn)))


@pytest.mark.parametrize("B,H,W,Cin,Cout,taps", [
    (1, 160, 128, 32, 32, 9),    # rows of whole 64-pixel blocks
    (2, 121, 136, 32, 32, 9),    # blocks that go over the end of a row, two images
    (3, 91, 72, 16, 40, 9),
    (2, 160, 48, 64, 64, 9),     # strips of 16
    (4, 512, 8, 8, 32, 9),       # strips of 8
    (1, 300, 56, 96, 130, 9),
    (2, 136, 92, 32, 24, 9),     # width not a multiple of 8
    (3, 72, 100, 128, 128, 9),
    (2, 96, 104, 64, 8, 1)])     # 1x1
def test_wgrad_split_ranges(cuda, B, H, W, Cin, Cout, taps):
    torch = cuda
    import torch.nn.functional as F
    from iterative_tomographic_reconstruction_algorithms_b200 import nn
    P = B * H * W
    assert P >= 3 * 4096
    g = torch.Generator().manual_seed(B * H + W + Cin + Cout)
    X = torch.randn((B, H, W, Cin), generator=g).to(torch.bfloat16).cuda()
    dY = torch.randn((B, H, W, Cout), generator=g).to(torch.bfloat16).cuda()
    k = 3 if taps == 9 else 1
    w = torch.zeros((Cout, Cin, k, k), dtype=torch.float64, device="cuda", requires_grad=True)
    b = torch.zeros((Cout,), dtype=torch.float64, device="cuda", requires_grad=True)
    F.conv2d(X.double().permute(0, 3, 1, 2), w, b, padding=k // 2).backward(dY.double().permute(0, 3, 1, 2))
    ref = w.grad.permute(0, 2, 3, 1).reshape(Cout, taps, Cin)
    dW, db = nn.wgrad(X, dY, taps)
    nn.check_status()
    # the split: ranges of at least 4096 pixels, about 296 blocks of work in all
    bn = 32 if Cout <= 32 else 64 if Cout <= 64 else 128 if Cout <= 128 else 256
    tiles = ((taps * Cin + 127) // 128) * ((Cout + bn - 1) // bn)
    S = min(max(1, 296 // tiles), P // 4096, 64)
    assert S >= 2
    tol = (P / (16 * S) + 4 + S) * 2.0 ** -23
    assert float((dW.double() - ref).abs().max()) <= tol * float(ref.abs().max())
    assert float((db.double() - b.grad).abs().max()) <= 1e-6 * float(b.grad.abs().max())
    again, _ = nn.wgrad(X, dY, taps)
    assert torch.equal(again, dW)
