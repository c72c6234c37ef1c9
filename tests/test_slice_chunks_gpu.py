"""Calls on many slices: a plan's scratch stays within 512 MiB (or one slice's)
however many slices it serves; they go through it in chunks, and each slice has
the bits of a call on it alone.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _projector(oper, n, na):
    deg = np.linspace(0, 170, na, endpoint=False)
    if oper == "bspline":
        from iterative_tomographic_reconstruction_algorithms_b200 import class_projectors_bspline as cpb
        return cpb.projectors(n, deg)
    from iterative_tomographic_reconstruction_algorithms_b200 import class_projectors_radon as cpr
    return cpr.projectors(n, deg, oper=oper)


@pytest.mark.parametrize("oper", ["pd", "ss", "bspline"])
def test_plan_memory_is_bounded(cuda, oper):
    torch = cuda
    tp = _projector(oper, 512, 400)
    dev = torch.cuda.current_device()
    tp.plan(1, dev)  # tables of one slice, and the library itself
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    tp.plan(400, dev)
    used = before - torch.cuda.mem_get_info()[0]
    # 512 MiB of scratch; ray limits (ss) and tables with their weights (bspline) below 32 MiB, blocks of 2 MiB
    assert used <= 560 * MIB


@pytest.mark.parametrize("oper,n,na,nz", [("pd", 256, 5200, 72), ("ss", 256, 5200, 72), ("bspline", 256, 1500, 70)])
def test_slices_in_chunks(cuda, oper, n, na, nz):
    """Two full chunks of 31 or 32 slices, and a rest."""
    torch = cuda
    tp = _projector(oper, n, na)
    g = torch.Generator().manual_seed(n)
    x = torch.randn((nz, n, n), generator=g).cuda()
    y = torch.randn((nz, na, n), generator=g).cuda()
    A, At = tp.A(x), tp.At(y)
    for z in list(range(0, nz, 9)) + list(range(25, 37)) + [nz - 1]:
        assert torch.equal(A[z], tp.A(x[z])) and torch.equal(At[z], tp.At(y[z])), z


@pytest.mark.parametrize("oper,n,na,nz", [("pd", 256, 5200, 40), ("ss", 256, 5200, 40)])
def test_solver_over_chunks(cuda, oper, n, na, nz):
    """The fused iteration reads b, the weights and x, and writes its residual's parts, at
    the chunk's place.  The residual adds 5.3e7 squares of float values in 64 bits; 1e-6 covers
    the rounding of A x (2 n x 2^-24 of each bin at most, of either sign)."""
    torch = cuda
    from iterative_tomographic_reconstruction_algorithms_b200.solvers import Solver
    tp = _projector(oper, n, na)
    g = torch.Generator().manual_seed(n)
    b = (torch.rand((nz, na, n), generator=g) + 0.5).cuda()
    x0 = torch.ones((nz, n, n), device="cuda")
    x, r = Solver(tp, "sirt", b).run(x0, 2)
    for z in (0, 17, 30, 39):
        xz, _ = Solver(tp, "sirt", b[z]).run(x0[z], 2)
        assert torch.equal(x[z], xz), z
    want = float(((tp.A(x0).double() - b.double()) ** 2).sum())
    assert any(abs(v - want) <= 1e-6 * want for v in (r[0], r[0] ** 2))
