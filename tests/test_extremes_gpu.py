"""The projector pairs at the ends of the float range: values next to the largest
float whose projections are finite, and infinite values that meet a weight of
exactly 0, against the FP64 oracle (the reference's float geometry and bin
decisions, summed in FP64).

Tolerance of the large values: all terms have one sign, so relative errors add.
Forward: every product is rounded (2^-24), their sum once more.  Adjoint: a pixel
adds up to 8 products in float.  9 x 2^-24 in both.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BIG = 3.2e38  # the largest float is 3.4e38
REL = 9 * 2.0 ** -24


def _pair(oper, n, deg, oracle):
    from iterative_tomographic_reconstruction_algorithms_b200 import class_projectors_radon as cpr
    tp = cpr.projectors(n, np.array(deg), oper=oper)
    return tp, lambda d, a: oracle.radon(oper, d, a, tp.angles)


def _compare(torch, fn, ref, a):
    got = fn(torch.from_numpy(a).cuda()).cpu().numpy()
    with np.errstate(over="ignore"):
        ref = np.where(np.isfinite(ref), ref.astype(np.float32), ref)  # beyond the largest float: infinite
    for test in (np.isnan, np.isposinf, np.isneginf):
        assert np.array_equal(test(got), test(ref)), test.__name__
    fin = np.isfinite(ref)
    assert np.all(np.abs(got[fin] - ref[fin]) <= REL * np.abs(ref[fin]) + 1e-30)
    return fin


@pytest.mark.parametrize("oper,n", [("pd", 40), ("pd", 330), ("pd", 641), ("ss", 40), ("ss", 450), ("ss", 641)])
def test_values_next_to_the_largest_float(cuda, oracle, oper, n):
    tp, orc = _pair(oper, n, [20.0, 61.0, 100.0, 155.0], oracle)
    for place in ((n // 2 + 3, n // 3), (n // 4, n // 2)):
        x = np.zeros((n, n), np.float32)
        x[place] = BIG
        assert _compare(cuda, tp.A, orc(0, x), x).sum() > 3 * n
    for place in ((0, n // 2 + 5), (1, n // 3), (3, n // 2 - 1)):
        y = np.zeros((4, n), np.float32)
        y[place] = BIG
        assert _compare(cuda, tp.At, orc(1, y), y).sum() > n * (n - 2)


@pytest.mark.parametrize("oper,n", [("pd", 32), ("pd", 33), ("pd", 450), ("ss", 32), ("ss", 33), ("ss", 450)])
def test_infinite_values_at_zero_weights(cuda, oracle, oper, n):
    """At 45 degrees (pd) the pixels of the diagonal land on a bin's centre exactly, where the
    other neighbour has weight 0: 0 x infinity is NaN.  At 0 degrees (ss) every ray does."""
    deg = [20.0, 45.0, 100.0] if oper == "pd" else [0.0, 20.0, 100.0]
    tp, orc = _pair(oper, n, deg, oracle)
    x = np.zeros((n, n), np.float32)
    x[n - 1 - n // 3, n // 3] = np.inf
    ref = orc(0, x)
    assert np.isnan(ref).any()
    _compare(cuda, tp.A, ref, x)
    for sign in (1.0, -1.0):
        y = np.zeros((3, n), np.float32)
        y[:, n // 2] = sign * np.inf
        ref = orc(1, y)
        assert np.isnan(ref).any()
        _compare(cuda, tp.At, ref, y)


@pytest.mark.parametrize("n", [32, 33, 384, 385, 1900])
def test_ss_small_weights_at_the_centre(cuda, oracle, n):
    """Next to the centre a crossing has bits below those of the pixel's coordinate: a single bin
    of 1 gives every pixel its weight, each right to 9 x 2^-24 of itself however small."""
    deg = np.concatenate([np.linspace(3.1, 87.3, 9), np.linspace(92.2, 148.7, 6)])
    tp, orc = _pair("ss", n, deg, oracle)
    for b in (n // 2 - 1, n // 2, n // 2 + 1):
        y = np.zeros((len(deg), n), np.float32)
        for v in range(0, len(deg), 1 if n < 100 else 4):
            y[:] = 0.0
            y[v, b] = 1.0
            assert _compare(cuda, tp.At, orc(1, y), y).all()


def _bspline(n, oracle):
    from iterative_tomographic_reconstruction_algorithms_b200 import class_projectors_bspline as cpb
    tp = cpb.projectors(n, np.arange(24))  # 0, 45, 90 and 135 degrees among them
    return tp, lambda d, a: oracle.bspline(d, a, tp.angles, tp.lut, tp.param_spline)


@pytest.mark.parametrize("n", [40, 41, 300, 1100])
def test_bspline_values_next_to_the_largest_float(cuda, oracle, n):
    """Forward: neighbouring values that overflow a line's float sum in places where the bin is
    finite (off by the rounding of at most 12 products).  Adjoint: bin 0, whose value counts twice."""
    tp, orc = _bspline(n, oracle)
    x = np.zeros((n, n), np.float32)
    x[n // 2 + 3, n // 3:n // 3 + 6] = [3.1e38, 3.1e38, 3.1e38, -3.1e38, -3.1e38, -3.1e38]
    ref = orc(0, x)
    lim = float(np.finfo(np.float32).max)
    keep = np.abs(np.abs(ref) / lim - 1) > 1e-4  # away from the edge itself
    got = tp.A(cuda.from_numpy(x).cuda()).cpu().numpy()
    assert np.array_equal(np.isfinite(got)[keep], (np.abs(ref) < lim)[keep])
    fin = keep & (np.abs(ref) < lim)
    assert np.all(np.abs(got[fin] - ref[fin]) <= 13 * 2.0 ** -24 * 3.1e38)
    for v in (0, 3, 6, 12, 17):
        y = np.zeros((24, n), np.float32)
        y[v, 0] = BIG
        fin = _compare(cuda, tp.At, orc(1, y), y)
        assert fin.sum() > n * (n - 5)


@pytest.mark.parametrize("n", [40, 41])
def test_bspline_infinite_values(cuda, oracle, n):
    tp, orc = _bspline(n, oracle)
    rng = np.random.default_rng(n)
    for value in (np.inf, -np.inf, np.nan):
        x = rng.standard_normal((n, n)).astype(np.float32)
        x[n // 3, n // 2 - 2] = value
        y = rng.standard_normal((24, n)).astype(np.float32)
        y[5, 0], y[7, n // 2], y[0, 1] = value, value, -value
        for d, fn, a in ((0, tp.A, x), (1, tp.At, y)):
            ref, got = orc(d, a), fn(cuda.from_numpy(a).cuda()).cpu().numpy()
            for test in (np.isnan, np.isposinf, np.isneginf):
                assert np.array_equal(test(got), test(ref)), (value, d, test.__name__)


def test_bspline_table_that_is_not_finite(cuda, oracle):
    """Such a table takes the general kernels, where only the taps that read it are touched."""
    from iterative_tomographic_reconstruction_algorithms_b200 import _lib
    n = 40
    tp, _ = _bspline(n, oracle)
    lut = np.array(tp.lut, np.float32)
    lut[3, lut.shape[1] // 2 + 700] = np.nan
    x = np.random.default_rng(1).standard_normal((n, n)).astype(np.float32)
    ref = oracle.bspline(0, x, tp.angles, lut, tp.param_spline)
    assert np.isnan(ref).any() and np.isfinite(ref).any()
    plan = _lib.Plan(_lib.KIND_BSPLINE, n, tp.angles, lut=lut, lut_size=lut.shape[1], support=float(tp.param_spline[1]))
    got = plan.forward(cuda.from_numpy(x[None]).cuda()).cpu().numpy()[0]
    assert np.array_equal(np.isnan(got), np.isnan(ref))


@pytest.mark.parametrize("n", [41, 251, 600])
def test_grid_adjoint_next_to_the_largest_float(cuda, n):
    """A sum of the 1-D transform that passes the largest float makes NaN of the whole slice in the 2-D
    one: its butterflies add no more than the results do.  (The unnormalised 2-D transform may
    still pass it at single pixels, as the reference's does.)  Elsewhere the pixels are those of
    2^-60 of the value, times 2^60: powers of two round nothing, and the FFTs' log2(pdim) = 11 rounds
    and windows of 25 products stay within 1e-5 of the largest entry."""
    torch = cuda
    from iterative_tomographic_reconstruction_algorithms_b200 import class_projectors_grid as cpg
    tp = cpg.projectors(n, np.array([3.0, 31.0, 77.0, 118.0, 162.0]), verbose=False)
    lim = float(np.finfo(np.float32).max)
    for v, b in ((0, n // 2), (2, n // 3), (3, n - 7)):
        y = np.zeros((5, n), np.float32)
        y[v, b] = BIG
        small = tp.At(torch.from_numpy(y * np.float32(2.0 ** -60)).cuda()).cpu().numpy().astype(np.float64) * 2.0 ** 60
        got = tp.At(torch.from_numpy(y).cuda()).cpu().numpy().astype(np.float64)
        inside = np.isfinite(got) & (np.abs(small) < lim)
        assert inside.sum() > 0.9 * n * n
        assert np.abs(got[inside] - small[inside]).max() <= 1e-5 * np.abs(small[inside]).max()
