"""The convolution weight gradient's kernel at the edges of its tiles and splits.

The sizes cross the 8-pixel tile width, both tile heights, the 128-channel
output blocks, the 256-channel input blocks, the tap groups and odd channel
counts; FP64 torch on the same BF16 operands is the reference.

Tolerance: a CTA adds at most P / 16 <= 100 groups of 16 products into an FP32
accumulator, each addition off by at most 2^-23 of the running sum, which stays
within the largest entry's magnitude: 100 x 2^-23 = 1.2e-5 of it.
"""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W,Cin,Cout,taps", [
    (1, 8, 1, 8, 1, 9), (1, 1, 8, 8, 8, 1), (2, 17, 20, 24, 12, 9), (1, 16, 9, 40, 130, 9), (1, 33, 8, 96, 32, 9),
    (2, 7, 12, 264, 64, 9), (1, 9, 24, 384, 128, 9), (1, 24, 40, 128, 192, 9), (1, 40, 40, 64, 200, 1),
    (3, 16, 32, 32, 32, 9)])
def test_wgrad_tile_edges(cuda, B, H, W, Cin, Cout, taps):
    torch = cuda
    import torch.nn.functional as F
    from iterative_tomographic_reconstruction_algorithms_b200 import nn
    g = torch.Generator().manual_seed(B * H + W + Cin + Cout)
    X = torch.randn((B, H, W, Cin), generator=g).to(torch.bfloat16)
    dY = torch.randn((B, H, W, Cout), generator=g).to(torch.bfloat16)
    k = 3 if taps == 9 else 1
    w = torch.zeros((Cout, Cin, k, k), dtype=torch.float64, requires_grad=True)
    b = torch.zeros((Cout,), dtype=torch.float64, requires_grad=True)
    F.conv2d(X.double().permute(0, 3, 1, 2), w, b, padding=k // 2).backward(dY.double().permute(0, 3, 1, 2))
    ref = w.grad.permute(0, 2, 3, 1).reshape(Cout, taps, Cin)
    dW, db = nn.wgrad(X.cuda(), dY.cuda(), taps)
    nn.check_status()
    assert float((dW.double().cpu() - ref).abs().max()) <= 1.2e-5 * float(ref.abs().max())
    assert float((db.double().cpu() - b.grad).abs().max()) <= 1e-6 * float(b.grad.abs().max())
    again, _ = nn.wgrad(X.cuda(), dY.cuda(), taps)
    assert torch.equal(again, dW)
    # operands that do not start on a 16-byte boundary
    Xo = torch.empty(X.numel() + 1, dtype=torch.bfloat16, device="cuda")[1:].view(X.shape)
    Yo = torch.empty(dY.numel() + 1, dtype=torch.bfloat16, device="cuda")[1:].view(dY.shape)
    off, _ = nn.wgrad(Xo.copy_(X), Yo.copy_(dY), taps)
    assert torch.equal(off, dW)


@pytest.mark.parametrize("B,H,W,Cin,Cout", [
    (1, 5, 64, 32, 32), (1, 5, 72, 32, 32), (2, 9, 88, 8, 40), (1, 7, 120, 64, 64), (1, 3, 200, 96, 130), (2, 4, 136, 16, 24),
    (3, 11, 80, 48, 16), (1, 1, 104, 8, 8), (2, 2, 760, 32, 32)])
def test_wgrad_rows_ending_among_a_block(cuda, B, H, W, Cin, Cout):
    """64-pixel blocks that go over the end of a row at each multiple of 8; fewer than 100
    groups of 16 pixels per accumulator, as above."""
    test_wgrad_tile_edges(cuda, B, H, W, Cin, Cout, 9)
