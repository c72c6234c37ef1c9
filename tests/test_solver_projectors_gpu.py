"""The forms of the pixel-driven and slant-stacking kernels that the solvers
launch (one chain per bin and pixel, in the reference's order), across the sizes
where their layout changes: one MLEM step against the FP64 oracle's.

Tolerance: all data are positive, so relative errors add.  A bin sums at most 4 n
terms in a chain, a pixel 4 na, and a weight, a difference of coordinates of about
n, is off by about n x 2^-24 of one; the step has two adjoints and a forward:
(16 n + 16 na + 64) x 2^-24.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 33, 384, 385, 1024, 1025])
@pytest.mark.parametrize("oper", ["pd", "ss"])
def test_mlem_step_at_kernel_boundaries(cuda, oracle, oper, n):
    from iterative_tomographic_reconstruction_algorithms_b200 import class_projectors_radon as cpr
    from iterative_tomographic_reconstruction_algorithms_b200.solvers import Solver
    deg = np.array([3.0, 41.0, 45.0, 77.5, 101.0, 135.0, 168.0])
    tp = cpr.projectors(n, deg, oper=oper)
    rng = np.random.default_rng(n)
    x = rng.random((n, n)).astype(np.float32) + 0.5
    b = rng.random((len(deg), n)).astype(np.float32) + 0.5
    got, _ = Solver(tp, "em", b).run(x, 1)

    def fix(a, eps):
        return np.where(a == 0, eps, a)
    f32 = np.float32
    bn = fix(oracle.radon(oper, 0, x, tp.angles), 2.220446049250313e-16)
    d = fix(oracle.radon(oper, 1, np.ones_like(b), tp.angles), 1e-10)
    ref = x * (oracle.radon(oper, 1, (b / bn).astype(f32), tp.angles) / d)
    tol = (16 * n + 16 * len(deg) + 64) * 2.0 ** -24
    assert np.linalg.norm(got - ref) <= tol * np.linalg.norm(ref)
