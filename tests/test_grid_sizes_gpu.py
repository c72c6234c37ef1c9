"""The gridding pair over Fourier grids of different factors (FFT passes of radix 8,
4, 2, 3, 5, 7 and of a prime without a butterfly) and over angle sets that fill the
adjoint's angle buckets unevenly.  The forward is compared with a NumPy restatement
of gridrec_v4_forwproj.c:213-398 (weights and window bounds in float32 as there,
transforms and sums in float64), the matched adjoint with it by dot products.

Tolerances as for the same comparisons elsewhere: 1e-5 relative L2 against the
reference's float arithmetic, 1e-5 of |A x| |y| for the dot products.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu
f32 = np.float32


def _weights(tp, dist, tbl):
    x = (dist * tbl).astype(f32)
    if int(tp.param_nofilt[4]) == 0:
        return tp.lut[(x + f32(0.49999997)).astype(f32).astype(int)]
    i = np.floor(x).astype(int)
    return (1 - x + i) * tp.lut[i] + (x - i) * tp.lut[i + 1]


def _forward(tp, img):
    n, (N, _) = tp.npix, tp.deapod.shape
    half, pad = N // 2, (N - n) // 2
    H = np.zeros((N, N))
    H[pad:pad + n, pad:pad + n] = (tp.deapod[pad:pad + n, pad:pad + n] * img[::-1].T)
    H = np.fft.ifft2(np.fft.fftshift(H)) * N * N
    lconv = f32(2 * 7.0 / np.pi)
    h, tbl = lconv * f32(0.5), f32(2 * int(tp.param_nofilt[5])) * (f32(1) / lconv)
    w = np.arange(half)
    phase = np.exp(1j * w * f32(2 * np.pi * (n * 0.5 + (pad if N != n else 0)) / N))
    out = np.zeros((len(tp.angles), n))
    for k, deg in enumerate(tp.angles):
        s, c = f32(np.sin(float(deg) * np.pi / 180)), f32(np.cos(float(deg) * np.pi / 180))
        U, V = ((float(t) * w + half).astype(f32) for t in (c, s))
        c1, c2 = np.zeros(half, complex), np.zeros(half, complex)
        ok0 = (np.ceil(U - h) >= 0) & (np.ceil(V - h) >= 0)
        for du in range(-4, 5):
            for dv in range(-4, 5):
                iu, iv = np.rint(U).astype(int) + du, np.rint(V).astype(int) + dv
                ok = ok0 & (iu >= np.ceil(U - h)) & (iu <= np.floor(h + U)) & (iv >= np.ceil(V - h)) & \
                    (iv <= np.floor(V + h)) & (iu < N) & (iv < N)
                i, j, q = iu[ok], iv[ok], w[ok]
                wt = _weights(tp, np.abs(U[ok] - i.astype(f32)), tbl) * _weights(tp, np.abs(V[ok] - j.astype(f32)), tbl)
                c1[q] += H[i, j] * wt
                m = (i != 0) & (j != 0) & (q != 0)
                c2[q[m]] += H[N - i[m], N - j[m]] * wt[m]
        row = np.zeros(N, complex)
        row[N - w[1:]], row[0] = (np.conj(phase) * c1)[1:], c1[0]
        row[w[1:]] = (phase * c2)[1:]
        out[k] = np.fft.fft(row).real[pad:pad + n] / N
    return out


ANGLES = {"even": np.linspace(0, 180, 24, endpoint=False), "clustered": np.sort(np.r_[np.linspace(40, 41, 40), 90.0, 179.0]),
          "one": np.array([37.0]), "repeated": np.array([0.0, 0.0, 45.0, 45.0, 45.0, 135.0])}


@pytest.mark.parametrize("n,os_,angles", [
    (16, 2.0, "even"), (33, 2.0, "one"), (40, 1.5, "clustered"), (64, 1.25, "repeated"), (64, 1.75, "even"),
    (60, 2.75, "even"), (100, 1.375, "clustered"), (24, 2.125, "even"), (128, 4.0, "even")])
def test_grid_pair_sizes(cuda, n, os_, angles):
    from iterative_tomographic_reconstruction_algorithms_b200 import class_projectors_grid as cpg
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, n)).astype(f32)
    for interp in ("nn", "lin"):
        tp = cpg.projectors(n, ANGLES[angles], kernel="pswf", oversampl=os_, interp=interp, W=7.0, verbose=False,
                            adjoint="matched")
        a = tp.A(x)
        assert rel_l2(a, _forward(tp, x)) <= 1e-5
        y = rng.standard_normal(a.shape).astype(f32)
        dot = float(np.vdot(a.astype(float), y)) - float(np.vdot(x.astype(float), tp.At(y)))
        assert abs(dot) <= 1e-5 * float(np.linalg.norm(a.astype(float)) * np.linalg.norm(y.astype(float)))
        b2 = tp.At(np.stack([y[::-1].copy(), y]))
        assert np.array_equal(b2[1], tp.At(y))  # slices of one call have the bits of single calls
