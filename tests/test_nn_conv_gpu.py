"""The 3x3 convolution kernel at the edges of its tiles, channel blocks and launch forms.

The sizes cross the 8 x 16 pixel tile, every row width of the staged patch (8,
16, 32 and 64 channels), resident and streamed weights, one and two tiles to a
weight stage, several output blocks, and the pass boundary at 384 channels;
FP64 torch on the same BF16 operands is the reference.

Tolerance: an output adds 9 Cin / 16 <= 225 groups of 16 products into an FP32
accumulator, each addition off by at most 2^-23 of the running sum, which stays
within the largest output's magnitude: 225 x 2^-23 = 2.7e-5 of it.
"""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W,Cin,Cout", [
    (1, 1, 1, 8, 1), (1, 17, 9, 8, 32), (2, 16, 8, 16, 20), (1, 15, 23, 24, 40), (1, 33, 17, 32, 96), (2, 20, 12, 40, 8),
    (1, 18, 30, 64, 192), (1, 31, 8, 96, 130), (3, 160, 136, 128, 64), (1, 40, 40, 192, 64), (1, 16, 24, 256, 256),
    (1, 9, 10, 384, 128), (1, 12, 11, 392, 36)])
def test_conv3x3_tile_edges(cuda, B, H, W, Cin, Cout):
    torch = cuda
    import torch.nn.functional as F
    from iterative_tomographic_reconstruction_algorithms_b200 import nn
    g = torch.Generator().manual_seed(B * H + W + Cin + Cout)
    X = torch.randn((B, H, W, Cin), generator=g).to(torch.bfloat16)
    Wt = torch.randn((Cout, 3, 3, Cin), generator=g).to(torch.bfloat16)
    b = torch.randn((Cout,), generator=g)
    ref = F.conv2d(X.double().permute(0, 3, 1, 2), Wt.double().permute(0, 3, 1, 2), b.double(), padding=1).permute(0, 2, 3, 1)
    Y = nn.conv3x3(X.cuda(), Wt.cuda(), b.cuda(), out_dtype=torch.float32)
    Yr = nn.conv3x3(X.cuda(), Wt.cuda(), b.cuda(), relu=True)
    Yn = nn.conv3x3(X.cuda(), Wt.cuda(), out_dtype=torch.float32)
    nn.check_status()
    assert float((Y.double().cpu() - ref).abs().max()) <= 2.7e-5 * float(ref.abs().max())
    assert torch.equal(Yr, Y.clamp(min=0).to(torch.bfloat16))
    assert float((Yn.double().cpu() + b.double() - ref).abs().max()) <= 2.7e-5 * float(ref.abs().max())
    with pytest.raises(RuntimeError):  # a source off the 16-byte boundary is refused
        off = torch.empty(X.numel() + 1, dtype=torch.bfloat16, device="cuda")[1:].view(X.shape)
        nn.conv3x3(off, Wt.cuda())


def test_conv3x3_wait_limit(cuda):
    """With the pipeline wait limit at 0 the kernel's roles give up, it drains
    its copies and MMAs, sets the status bit and returns."""
    torch = cuda
    from iterative_tomographic_reconstruction_algorithms_b200 import nn
    X = torch.randn((1, 40, 40, 128), device="cuda").to(torch.bfloat16)
    W = torch.randn((64, 3, 3, 128), device="cuda").to(torch.bfloat16)
    want = nn.conv3x3(X, W)
    nn.check_status()
    try:
        nn.set_wait_limit(0)
        nn.conv3x3(X, W)
        with pytest.raises(RuntimeError, match="wait gave up"):
            nn.check_status()
    finally:
        nn.set_wait_limit(-1)
    assert torch.equal(nn.conv3x3(X, W), want)
    nn.check_status()
