"""One plan used from several streams: every call shares the plan's tables and
scratch, so calls on different streams have to run one after another.  Results
are compared bit for bit with the same calls on one stream (the kernels sum in
fixed orders).
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, NA = 300, 280
OPERS = ("dd", "rd", "pd", "ss", "bspline", "grid")


def _projector(oper):
    if oper == "bspline":
        from iterative_tomographic_reconstruction_algorithms_b200 import class_projectors_bspline as cpb
        return cpb.projectors(N, np.linspace(0, 180, NA, endpoint=False))
    if oper == "grid":
        from iterative_tomographic_reconstruction_algorithms_b200 import class_projectors_grid as cpg
        return cpg.projectors(N, np.linspace(0, 180, NA, endpoint=False), verbose=False)
    from iterative_tomographic_reconstruction_algorithms_b200 import class_projectors_radon as cpr
    return cpr.projectors(N, np.linspace(0, 170, NA, endpoint=False), oper=oper)


def _inputs(torch, k):
    g = torch.Generator().manual_seed(7)
    xs = [torch.randn((N, N), generator=g).cuda() for _ in range(k)]
    ys = [torch.randn((NA, N), generator=g).cuda() for _ in range(k)]
    return xs, ys


@pytest.mark.parametrize("oper", OPERS)
def test_calls_on_several_streams(cuda, oper):
    torch = cuda
    tp = _projector(oper)
    xs, ys = _inputs(torch, 3)
    want = [(tp.A(x), tp.At(y)) for x, y in zip(xs, ys)]
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    got = []
    for it in range(8):
        for k, s in enumerate(streams):
            with torch.cuda.stream(s):
                if (it + k) % 2:
                    got.append((k, 0, tp.A(xs[k])))
                got.append((k, 1, tp.At(ys[k])))
    torch.cuda.synchronize()
    for k, d, out in got:
        assert torch.equal(out, want[k][d]), (k, d)


@pytest.mark.parametrize("oper", ["pd", "ss", "bspline", "dd"])
def test_graphs_and_calls_on_several_streams(cuda, oper):
    """Captured calls, replayed on streams of their own beside plain ones; and a capture over two streams."""
    torch = cuda
    tp = _projector(oper)
    xs, ys = _inputs(torch, 3)
    want = [tp.At(y) for y in ys]
    graphs, outs = [], []
    for y in ys[:2]:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            outs.append(tp.At(y))
        graphs.append(g)
    fork, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(fork):
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            b0 = tp.At(ys[0])
        b1 = tp.At(ys[1])
        torch.cuda.current_stream().wait_stream(side)
    streams = [torch.cuda.Stream() for _ in range(4)]
    torch.cuda.synchronize()
    plain = []
    for _ in range(6):
        for g, s in zip(graphs + [fork], streams):
            with torch.cuda.stream(s):
                g.replay()
        with torch.cuda.stream(streams[3]):
            plain.append(tp.At(ys[2]))
    torch.cuda.synchronize()
    assert torch.equal(outs[0], want[0]) and torch.equal(outs[1], want[1])
    assert torch.equal(b0, want[0]) and torch.equal(b1, want[1])
    assert all(torch.equal(p, want[2]) for p in plain)


@pytest.mark.parametrize("oper", ["pd", "ss", "dd"])
def test_solver_beside_calls(cuda, oper):
    torch = cuda
    from iterative_tomographic_reconstruction_algorithms_b200.solvers import Solver
    tp = _projector(oper)
    xs, ys = _inputs(torch, 2)
    b = ys[0].abs()
    want_at, ones = tp.At(ys[1]), torch.ones((N, N), device="cuda")
    solver = Solver(tp, "sirt", b)
    want, _ = solver.run(ones, 5)
    s0, s1 = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for use_graph in (True, False):
        got = []
        with torch.cuda.stream(s1):
            got += [tp.At(ys[1]) for _ in range(4)]
        with torch.cuda.stream(s0):
            x, _ = solver.run(ones, 5, use_graph)
        with torch.cuda.stream(s1):
            got.append(tp.At(ys[1]))
        torch.cuda.synchronize()
        assert torch.equal(x, want) and all(torch.equal(a, want_at) for a in got)
