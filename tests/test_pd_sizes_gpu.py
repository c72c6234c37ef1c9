"""The pixel-driven pair where its kernels change shape with the image side:
how many warps share a bin's lines and a tile's angles, ragged tiles, and the
smallest images; against the FP64 oracle.

Tolerances (relative L2).  Forward: products of two lines, at most 12, are added
in float before they go to double: 12 x 2^-24 = 7.2e-7.  Adjoint: a pixel adds
4 products per angle in float: 4 x 31 x 2^-24 = 7.4e-6.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 31, 33, 128, 161, 320, 321, 384, 385, 448, 449, 640, 641])
def test_pd_pair_at_kernel_boundaries(cuda, oracle, n):
    torch = cuda
    from iterative_tomographic_reconstruction_algorithms_b200 import class_projectors_radon as cpr
    na = 31
    deg = np.sort(np.concatenate([[0.0, 45.0, 89.9, 90.0, 135.0, 179.9], np.linspace(1.3, 178.0, na - 6)]))
    tp = cpr.projectors(n, deg, oper="pd")
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, n)).astype(np.float32)
    y = rng.standard_normal((na, n)).astype(np.float32)
    A, At = tp.A(torch.from_numpy(x).cuda()), tp.At(torch.from_numpy(y).cuda())
    ref, reft = oracle.radon("pd", 0, x, tp.angles), oracle.radon("pd", 1, y, tp.angles)
    assert np.linalg.norm(A.cpu().numpy() - ref) <= 7.2e-7 * np.linalg.norm(ref) + 1e-30
    assert np.linalg.norm(At.cpu().numpy() - reft) <= 7.4e-6 * np.linalg.norm(reft) + 1e-30
    # slices of one call have the bits of single calls
    x2 = torch.from_numpy(np.stack([x[::-1].copy(), x])).cuda()
    y2 = torch.from_numpy(np.stack([y[::-1].copy(), y])).cuda()
    assert torch.equal(tp.A(x2)[1], A) and torch.equal(tp.At(y2)[1], At)
