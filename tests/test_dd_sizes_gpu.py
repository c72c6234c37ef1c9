"""The distance-driven pair where its kernels change shape: a forward item's
boundaries in one warp or split over four, the adjoint's rows per lane (few or
many tiles in the plan), ragged groups, tiles and pre-pass chunks.  Shapes and
batches keep every sum's order, so they agree bit for bit; the bits are compared
with the FP64 oracle.

Tolerances (relative L2): forward sums in double, each term a float distance
(n x 2^-24 of a pixel at most, of a chord of about n / 2 pixels or of one):
16 x 2^-24 + n x 2^-24 / 8; adjoint: two float terms per angle, 2 na x 2^-24,
and the same distances.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 32, 63, 127, 128, 129, 254, 255, 513])
def test_dd_pair_at_kernel_boundaries(cuda, oracle, n):
    torch = cuda
    from iterative_tomographic_reconstruction_algorithms_b200 import class_projectors_radon as cpr
    na = 37
    deg = np.sort(np.concatenate([[0.0, 45.0, 89.9, 90.0, 135.0, 179.9], np.linspace(1.3, 178.0, na - 6)]))
    tp = cpr.projectors(n, deg, oper="dd")
    rng = np.random.default_rng(n)
    x = rng.random((n, n)).astype(np.float32) + 0.5
    y = rng.random((na, n)).astype(np.float32) + 0.5
    xg, yg = torch.from_numpy(x).cuda()[None], torch.from_numpy(y).cuda()[None]
    p = tp.plan(1, 0)
    A, At = p.forward(xg), p.adjoint(yg)
    for shape in ("w2w", "w8b", "w4s"):
        p.set_tuning(shape, None)
        assert torch.equal(p.forward(xg), A), shape
    nz = 800 // (((n + 31) // 32) * ((n + 15) // 16)) + 1  # enough tiles for 4 x 4 pixels per lane
    assert torch.equal(tp.A(xg.expand(nz, n, n).contiguous())[-1], A[0])
    assert torch.equal(tp.At(yg.expand(nz, na, n).contiguous())[-1], At[0])
    ref, reft = oracle.radon("dd", 0, x, tp.angles), oracle.radon("dd", 1, y, tp.angles)
    u = 2.0 ** -24
    assert np.linalg.norm(A[0].cpu().numpy() - ref) <= (16 + n / 8) * u * np.linalg.norm(ref) + 1e-30
    assert np.linalg.norm(At[0].cpu().numpy() - reft) <= (16 + 2 * na + n / 8) * u * np.linalg.norm(reft) + 1e-30
