"""The slant-stacking pair where its kernels change shape with the image side
(warps sharing a ray's steps or a tile's angles, ragged and border-only tiles)
and at angles next to an axis, against the FP64 oracle.

Tolerances (relative L2).  Forward: a ray adds 2 n products in float, in runs of
at least n / 4: 2 n x 2^-24.  Adjoint: a pixel adds 2 products per angle: 2 x 31
x 2^-24 = 3.7e-6.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 31, 33, 128, 160, 161, 384, 385, 448, 449, 640, 641])
def test_ss_pair_at_kernel_boundaries(cuda, oracle, n):
    torch = cuda
    from iterative_tomographic_reconstruction_algorithms_b200 import class_projectors_radon as cpr
    na = 31
    # nothing within 1/nh of 180 degrees: those rays miss the square, where the oracle has no value
    deg = np.sort(np.concatenate([[0.0, 0.3, 1.1, 44.9, 45.0, 89.6, 90.0, 90.2, 135.0], np.linspace(2.3, 150.0, na - 9)]))
    tp = cpr.projectors(n, deg, oper="ss")
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, n)).astype(np.float32)
    y = rng.standard_normal((na, n)).astype(np.float32)
    A, At = tp.A(torch.from_numpy(x).cuda()), tp.At(torch.from_numpy(y).cuda())
    ref, reft = oracle.radon("ss", 0, x, tp.angles), oracle.radon("ss", 1, y, tp.angles)
    assert np.linalg.norm(A.cpu().numpy() - ref) <= 2 * n * 2.0 ** -24 * np.linalg.norm(ref) + 1e-30
    assert np.linalg.norm(At.cpu().numpy() - reft) <= 3.7e-6 * np.linalg.norm(reft) + 1e-30
    # slices of one call have the bits of single calls
    x2 = torch.from_numpy(np.stack([x[::-1].copy(), x])).cuda()
    y2 = torch.from_numpy(np.stack([y[::-1].copy(), y])).cuda()
    assert torch.equal(tp.A(x2)[1], A) and torch.equal(tp.At(y2)[1], At)
