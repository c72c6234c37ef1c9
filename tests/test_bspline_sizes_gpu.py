"""The B-spline pair where its kernels change shape with the image side, the
special bins (bin 0, next to 0 and to powers of two) at axis angles, and tables
that take the general kernels; against the FP64 oracle.

Tolerances (relative L2).  Forward: six products of a line are added in float,
lines in double: 7 x 2^-24 = 4.2e-7.  Adjoint: a pixel adds 5 products per angle
in float: 5 x 24 x 2^-24 = 7.2e-6.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,support,samples", [
    (2, 4, 2048), (4, 4, 2048), (5, 4, 2048), (31, 4, 2048), (64, 4, 2048), (65, 4, 2048), (130, 4, 64), (257, 4, 2048),
    (512, 4, 2048), (769, 4, 1024), (1025, 4, 2048), (48, 4, 1000), (49, 6, 2048), (48, 4, 4096)])
def test_bspline_pair_at_kernel_boundaries(cuda, oracle, n, support, samples):
    torch = cuda
    from iterative_tomographic_reconstruction_algorithms_b200 import class_projectors_bspline as cpb
    na = 24  # 0, 45, 90 and 135 degrees among them
    tp = cpb.projectors(n, np.arange(na), proj_support_y=support, nsamples_y=samples)
    rng = np.random.default_rng(n + samples)
    x = rng.standard_normal((n, n)).astype(np.float32)
    y = rng.standard_normal((na, n)).astype(np.float32)
    A, At = tp.A(torch.from_numpy(x).cuda()), tp.At(torch.from_numpy(y).cuda())
    ref = oracle.bspline(0, x, tp.angles, tp.lut, tp.param_spline)
    reft = oracle.bspline(1, y, tp.angles, tp.lut, tp.param_spline)
    assert np.linalg.norm(A.cpu().numpy() - ref) <= 4.2e-7 * np.linalg.norm(ref) + 1e-30
    assert np.linalg.norm(At.cpu().numpy() - reft) <= 7.2e-6 * np.linalg.norm(reft) + 1e-30
    # slices of one call have the bits of single calls
    x2 = torch.from_numpy(np.stack([x[::-1].copy(), x])).cuda()
    y2 = torch.from_numpy(np.stack([y[::-1].copy(), y])).cuda()
    assert torch.equal(tp.A(x2)[1], A) and torch.equal(tp.At(y2)[1], At)
