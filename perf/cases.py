"""The work that users of this framework have it do, as cases that can be timed and compared.

Paths (a case's ``path``):

* ``pair``   one ``A x`` and one ``At b`` of a projector class (``oper``: pd, rd, dd, ss, bspline, grid) on CUDA
             tensors: what every reference solver loop, autograd step and FBP does.  ``nz`` slices share one call.
* ``solver`` a whole fused reconstruction (``solvers.Solver``: SIRT or MLEM) from a constant start.
* ``batch``  SIRT on slices of uneven size in one batched plan.
* ``unet``   the warm-start network: one training step's forward and backward (``train``) or inference.
* ``conv``   one 3x3 convolution layer, forward and both gradients, through the functions of ``nn``.
"""
import ctypes
import math

import numpy as np
import torch

from iterative_tomographic_reconstruction_algorithms_b200 import _lib, nn
from iterative_tomographic_reconstruction_algorithms_b200 import class_projectors_bspline as cp_bspline
from iterative_tomographic_reconstruction_algorithms_b200 import class_projectors_grid as cp_grid
from iterative_tomographic_reconstruction_algorithms_b200 import class_projectors_radon as cp_radon
from iterative_tomographic_reconstruction_algorithms_b200.solvers import Solver

PI = math.pi
OPERS = ("pd", "rd", "dd", "ss", "bspline", "grid")


def listed():
    return [
        # a quick look at a small slice (the ray-driven configuration's size): latency and launches count
        dict(name="dd pair 256x304", path="pair", oper="dd", n=256, na=304, nz=1),
        # one full-size slice, the benchmark's default workload
        dict(name="dd pair 2048x1800", path="pair", oper="dd", n=2048, na=1800, nz=1),
        # the class's default projector at the size of the statistical solvers' configuration
        dict(name="pd pair 768x720", path="pair", oper="pd", n=768, na=720, nz=1),
        # an odd detector and an odd angle count, as centred or cropped scans give them
        dict(name="rd pair 769x513", path="pair", oper="rd", n=769, na=513, nz=1),
        # slant stacking on a few slices of a volume at once
        dict(name="ss pair 4x641x600", path="pair", oper="ss", n=641, na=600, nz=4),
        # the cubic B-spline pair that regularised solvers use
        dict(name="bspline pair 768x720", path="pair", oper="bspline", n=768, na=720, nz=1),
        # the gridding pair of the ADMM-TV configuration (Kaiser-Bessel, width 6, oversampling 2)
        dict(name="grid pair 1536x1500", path="pair", oper="grid", n=1536, na=1500, nz=1),
        # a whole plain SIRT reconstruction, ray-driven, 100 iterations
        dict(name="sirt rd 256x304", path="solver", algo="sirt", oper="rd", n=256, na=304, nz=1, iters=100),
        # a whole MLEM reconstruction, distance-driven, 50 iterations (512^2 object in 768 bins)
        dict(name="mlem dd 768x720", path="solver", algo="em", oper="dd", n=768, na=720, nz=1, iters=50),
        # SIRT on a mixed bag of regions of interest, one launch per application
        dict(name="sirt batch 16", path="batch", slices=16, mix=1, largest=1024, iters=5),
        # a training step of the warm-start network at its configuration (batch 4, 768^2, 32 channels, 4 levels)
        dict(name="unet step 4x768", path="unet", batch=4, side=768, base=32, levels=4, train=True),
        # one of that network's inner layers
        dict(name="conv 4x192x192x128", path="conv", batch=4, h=192, w=192, cin=128, cout=128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choices(("pair", "solver", "batch", "unet", "conv"), weights=(7, 2, 1, 2, 2))[0]
    if path == "pair":
        oper = rng.choice(OPERS)
        top = {"dd": 2048, "grid": 1536, "ss": 1280, "rd": 768, "pd": 1280, "bspline": 1024}[oper]
        n = _log_int(rng, 96, top)
        na = max(30, int(n * rng.uniform(0.4, 1.2)))
        nz = rng.choice((1, 1, 1, 2, 3)) if n <= 0.6 * top else 1
        return dict(path=path, oper=oper, n=n, na=na, nz=nz)
    if path == "solver":
        n = _log_int(rng, 128, 512)
        return dict(path=path, algo=rng.choice(("sirt", "em")), oper=rng.choice(("dd", "dd", "pd", "ss")), n=n,
                    na=int(n * rng.uniform(0.4, 1.2)), nz=rng.choice((1, 1, 2)), iters=rng.randint(10, 40))
    if path == "batch":
        return dict(path=path, slices=rng.randint(3, 16), mix=rng.randint(2, 1 << 20),
                    largest=rng.choice((512, 1024)), iters=rng.randint(2, 5))
    if path == "unet":
        return dict(path=path, batch=rng.randint(1, 4), side=8 * rng.randint(8, 88), base=32, levels=4,
                    train=rng.random() < 0.6)
    lvl = rng.randint(0, 3)
    return dict(path=path, batch=rng.randint(1, 4), h=8 * rng.randint(3, 80 >> lvl), w=8 * rng.randint(3, 80 >> lvl),
                cin=32 << rng.randint(max(0, lvl - 1), lvl), cout=32 << lvl)


# ---- inputs ----
def _device():
    return torch.device("cuda", torch.cuda.current_device()) if torch.cuda.is_available() else torch.device("cpu")


def _rng(case, seed, k=0):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, k])


def _ellipses(g, count=10):
    """(x0, y0, a, b, phi, rho) of a random-ellipse phantom on [-1, 1]^2, densities >= 0."""
    rad, ang = 0.7 * np.sqrt(g.uniform(0, 1, count)), g.uniform(0, 2 * PI, count)
    return np.stack([rad * np.cos(ang), rad * np.sin(ang), g.uniform(0.05, 0.5, count), g.uniform(0.05, 0.5, count),
                     g.uniform(0, PI, count), g.uniform(0.05, 1.0, count)], 1)


def _image(ell, n, dev):
    """The phantom's pixel values, rows downwards, float32; the square is the middle 2/3 of the canvas."""
    c = (torch.arange(n, dtype=torch.float64, device=dev) + 0.5 - n // 2) / (n / 3.0)
    X, Y = c[None, :], c[:, None]
    img = torch.zeros((n, n), dtype=torch.float64, device=dev)
    for x0, y0, a, b, phi, rho in ell:
        u = ((X - x0) * math.cos(phi) + (Y - y0) * math.sin(phi)) / a
        v = (-(X - x0) * math.sin(phi) + (Y - y0) * math.cos(phi)) / b
        img += (u * u + v * v <= 1.0).to(torch.float64) * rho
    return img.to(torch.float32)


def _normals(oper, na):
    """Unit normals (along columns, along rows) of every sinogram row's detector axis."""
    deg = np.linspace(0.0, 180.0, na, endpoint=False) * PI / 180.0
    if oper == "dd":
        a = np.fft.fftshift(deg)[::-1]
        s, c = np.sin(a), np.cos(a)
        f = np.where(a > PI / 2, 1.0, -1.0)
        return f * s, -f * c
    if oper == "rd":
        return -np.cos(deg), np.sin(deg)
    if oper == "pd":
        a = np.fft.fftshift(deg)
        f = np.where(np.cos(a) >= 0, 1.0, -1.0)
        return f * np.sin(a), f * np.cos(a)
    if oper == "ss":
        a = deg[::-1]
        return np.cos(a), np.sin(a)
    return np.cos(deg), -np.sin(deg)


def _sinogram(ell, oper, n, na, dev, scale=1.0):
    """The phantom's line integrals per detector bin (float64), rows as ``oper`` orders them."""
    nx, ny = (torch.from_numpy(np.ascontiguousarray(v)).to(dev)[:, None] for v in _normals(oper, na))
    unit = n / 3.0
    t = (torch.arange(n, dtype=torch.float64, device=dev) + (0.0 if oper in ("pd", "rd", "ss", "bspline") else 0.5) - n // 2)[None, :] / unit
    out = torch.zeros((na, n), dtype=torch.float64, device=dev)
    for x0, y0, a, b, phi, rho in ell:
        p, q = nx * math.cos(phi) + ny * math.sin(phi), -nx * math.sin(phi) + ny * math.cos(phi)
        w2 = (a * p) ** 2 + (b * q) ** 2
        d = t - (nx * x0 + ny * y0)
        out += rho * 2.0 * a * b * torch.sqrt(torch.clamp(w2 - d * d, min=0.0)) / w2
    return out * (unit * scale)


def _projector(oper, n, na):
    deg = np.linspace(0.0, 180.0, na, endpoint=False)
    if oper == "bspline":
        return cp_bspline.projectors(n, deg)
    if oper == "grid":
        return cp_grid.projectors(n, deg, kernel="kb", oversampl=2.0, W=6.0, errs=1e-3, interp="lin", verbose=False)
    return cp_radon.projectors(n, deg, oper=oper)


def _pair_inputs(case, seed, dev):
    n, na, nz, oper = case["n"], case["na"], case["nz"], case["oper"]
    xs, bs = [], []
    for z in range(nz):
        g = _rng(case, seed, z)
        ell = _ellipses(g)
        xs.append(_image(ell, n, dev))
        b = _sinogram(ell, oper, n, na, dev)
        noise = torch.from_numpy(g.standard_normal((na, n), dtype=np.float32)).to(dev).double()
        bs.append((b + 0.01 * b.max() * noise).to(torch.float32))
    return torch.stack(xs).contiguous(), torch.stack(bs).contiguous()


def _batch_geoms(case):
    """Sides from {256, 512, 1024, 2048} with weights 4:3:2:1 up to ``largest``, 1.5 angles and bins per side pixel."""
    g = np.random.default_rng(case["mix"])
    sides, w = [256, 512, 1024, 2048], [4, 3, 2, 1]
    keep = [i for i, s in enumerate(sides) if s <= case["largest"]]
    p = np.array([w[i] for i in keep], float)
    pick = g.choice([sides[i] for i in keep], size=case["slices"], p=p / p.sum())
    return [(int(math.ceil(1.5 * s)), int(round(1.5 * s))) for s in pick]


def _conv_inputs(case, seed, dev):
    g = torch.Generator(device=dev).manual_seed(int(seed))
    B, H, W, ci, co = case["batch"], case["h"], case["w"], case["cin"], case["cout"]
    X = torch.relu(torch.randn((B, H, W, ci), generator=g, device=dev)).to(torch.bfloat16)
    Wt = torch.randn((co, 3, 3, ci), generator=g, device=dev) * math.sqrt(2.0 / (9 * ci))
    b = 0.1 * torch.randn((co,), generator=g, device=dev)
    dY = torch.randn((B, H, W, co), generator=g, device=dev).to(torch.bfloat16)
    return X, Wt, b, dY


def prepare(case, seed):
    dev, path = _device(), case["path"]
    if path == "pair":
        x, b = _pair_inputs(case, seed, dev)
        tp = _projector(case["oper"], case["n"], case["na"])
        tp.plan(case["nz"], dev.index)
        return {"path": path, "tp": tp, "x": x, "b": b}
    if path == "solver":
        n, na = case["n"], case["na"]
        tp = _projector(case["oper"], n, na)
        b = torch.stack([_sinogram(_ellipses(_rng(case, seed, z)), case["oper"], n, na, dev, 0.01) for z in range(case["nz"])])
        b = b.clamp(min=0.0).to(torch.float32).contiguous()
        x0 = torch.full((case["nz"], n, n), 0.005, device=dev)
        return {"path": path, "solver": Solver(tp, case["algo"], b), "x0": x0, "iters": case["iters"]}
    if path == "batch":
        geoms = _batch_geoms(case)
        deg = [np.linspace(0.0, 180.0, na, endpoint=False) for _, na in geoms]
        plan = _lib.BatchPlan([(n, cp_radon.shim_angles("dd", (d * PI / 180.0).astype(np.float32))) for (n, _), d in zip(geoms, deg)])
        b = [_sinogram(_ellipses(_rng(case, seed, k)), "dd", n, na, dev, 0.01).to(torch.float32) for k, (n, na) in enumerate(geoms)]
        b = plan.pack(b, "sino")
        return {"path": path, "solver": Solver(plan, "sirt", b), "x0": torch.zeros((plan.img_total,), device=dev), "iters": case["iters"]}
    if path == "unet":
        net = nn.UNet(levels=case["levels"], base=case["base"], seed=int(seed)).to(dev)
        g = torch.Generator(device=dev).manual_seed(int(seed))
        with torch.no_grad():
            net.head_w.copy_(0.05 * torch.randn(net.head_w.shape, generator=g, device=dev))
        side, ims = case["side"], []
        for k in range(case["batch"]):
            ims.append(_image(_ellipses(_rng(case, seed, k)), side, dev))
        t = torch.stack(ims)
        blur = torch.nn.functional.avg_pool2d(t[:, None], 5, stride=1, padding=2)[:, 0]
        noise = 0.1 * torch.randn(t.shape, generator=g, device=dev)
        return {"path": path, "net": net, "x": blur, "fbp": t + noise, "t": t, "train": case["train"]}
    X, Wt, b, dY = _conv_inputs(case, seed, dev)
    return {"path": path, "X": X, "W": Wt, "b": b, "dY": dY}


def run(state):
    path = state["path"]
    if path == "pair":
        tp = state["tp"]
        return {"Ax": tp.A(state["x"]), "Atb": tp.At(state["b"])}
    if path in ("solver", "batch"):
        x, res = state["solver"].run(state["x0"], state["iters"])
        return {"x": x, "residuals": res}
    if path == "unet":
        net = state["net"]
        if not state["train"]:
            with torch.no_grad():
                return {"out": net(state["x"], state["fbp"])}
        for p in net.parameters():
            p.grad = None
        out = net(state["x"], state["fbp"])
        loss = ((out - state["t"]) ** 2).sum() / (state["t"] ** 2).sum()
        loss.backward()
        return {"out": out.detach(), "loss": loss.detach(), "grads": [p.grad for p in net.parameters()]}
    X, W, dY = state["X"], state["W"], state["dY"]
    co, _, _, ci = W.shape
    Wb, Wd = nn.prepare_weights(W.reshape(co, 9, ci))
    Y = nn.conv3x3(X, Wb.reshape(co, 3, 3, ci), state["b"], relu=True)
    dX = nn.conv3x3(dY, Wd.reshape(ci, 3, 3, co))
    dW, db = nn.wgrad(X, dY, 9)
    return {"Y": Y, "dX": dX, "dW": dW, "db": db}


# ---- what a pass cannot do without ----
# multiply-adds per (pixel, angle) and direction: the operands a projector's definition names
_TERMS = {"pd": 4, "rd": 6, "dd": 2, "ss": 2, "bspline": 5}


def _pair_work(oper, n, na, nz):
    bytes_ = 8.0 * nz * (n * n + na * n)
    if oper == "grid":
        p = 4
        while p < 2 * n:
            p *= 2
        taps = (6 * 6 + 5 * 5) * 8.0 * na * p / 2  # window gathers of both directions, complex by real
        return bytes_, nz * (2 * 5.0 * p * p * 2 * math.log2(p) + 2 * 5.0 * na * p * math.log2(p) + taps)
    return bytes_, 2.0 * 2.0 * _TERMS[oper] * n * n * na * nz


def _conv_flops(px, ci, co):
    return 2.0 * 9 * ci * co * px


def work(case):
    path = case["path"]
    if path == "pair":
        b, f = _pair_work(case["oper"], case["n"], case["na"], case["nz"])
    elif path == "solver":
        b, f = _pair_work(case["oper"], case["n"], case["na"], case["nz"])
        b, f = b, f * case["iters"]
    elif path == "batch":
        parts = [_pair_work("dd", n, na, 1) for n, na in _batch_geoms(case)]
        b, f = sum(p[0] for p in parts), sum(p[1] for p in parts) * case["iters"]
    elif path == "unet":
        px, base, L, f = float(case["batch"] * case["side"] ** 2), case["base"], case["levels"], 0.0
        cin = 8
        for i in range(L):
            f += (_conv_flops(px, cin, base << i) + _conv_flops(px, base << i, base << i)) / 4 ** i
            cin = base << i
        for i in reversed(range(L - 1)):
            f += (_conv_flops(px, (base << (i + 1)) + (base << i), base << i) + _conv_flops(px, base << i, base << i)) / 4 ** i
        f *= 3 if case["train"] else 1
        b = px * 4 * (4 if case["train"] else 3)
    else:
        px = float(case["batch"] * case["h"] * case["w"])
        f = 3 * _conv_flops(px, case["cin"], case["cout"])
        b = 2.0 * px * 2 * (case["cin"] + case["cout"]) + 2 * 4.0 * 9 * case["cin"] * case["cout"]
    return {"bytes": b, "flops": f}


# ---- the same results in 64 bits ----
# The operators' bins and weights are defined by float32 geometry (the angle's float32 sine and cosine and the
# float32 expressions of the projector's definition); the sums over them are exact ones, here in 64 bits.
_libm = ctypes.CDLL("libm.so.6")
for _f in ("sinf", "cosf"):
    getattr(_libm, _f).restype = ctypes.c_float
    getattr(_libm, _f).argtypes = [ctypes.c_float]


def _sc(theta):
    return np.float32(_libm.sinf(float(theta))), np.float32(_libm.cosf(float(theta)))


def _fma(a, b, c):
    """a * b + c of float32 operands, rounded once to float32."""
    return (a.double() * float(b) + c.double()).float() if not isinstance(b, torch.Tensor) else (a.double() * b.double() + c.double()).float()


def _rad(oper, na):
    a = (np.linspace(0.0, 180.0, na, endpoint=False) * PI / 180.0).astype(np.float32)
    return np.fft.fftshift(a) if oper in ("pd", "dd") else a


def _exact_pd(x, b, n, na, dev):
    nh = n // 2
    fwd, adj = torch.zeros((na, n), dtype=torch.float64, device=dev), torch.zeros((n, n), dtype=torch.float64, device=dev)
    ar = torch.arange(n, dtype=torch.float32, device=dev)
    img = x.flip(0).double()  # loop row i is stored at row n - 1 - i
    spread = 32
    lane = (torch.arange(n, device=dev) % spread)[:, None] * (n + 2)
    for v, th in enumerate(_rad("pd", na)):
        s, c = _sc(th)
        rc = np.float32(1.0) / c
        acc = torch.zeros(spread * (n + 2), dtype=torch.float64, device=dev)
        row = torch.zeros(n + 2, dtype=torch.float64, device=dev)
        row[1:n] = b[v, 1:n].double()  # bin 0 and bins outside take no part; place n + 1 collects them
        for d in (-0.25, 0.25):
            X, Y = (ar - nh + 0.5 + d)[None, :], (ar - nh + 0.5 + d)[:, None]
            xs = X * s.item()
            t = _fma(-Y, float(c), xs).abs()
            keep = (Y > xs * rc.item()) if float(th) != PI / 2 else torch.zeros_like(t, dtype=torch.bool)
            if float(th) == 0.0:
                keep = keep | (Y > 0.0)
            t = torch.where(keep, t, -t)
            T = nh - t
            lo, hi = torch.floor(T), torch.ceil(T)
            for k, w in ((lo, ((t + hi) - nh).abs()), (hi, (T - lo).abs())):
                idx = torch.where((k >= 1) & (k < n), k, torch.full_like(k, n + 1)).long()
                w = 0.5 * w.double()
                acc.index_add_(0, (idx + lane).reshape(-1), (w * img).reshape(-1))
                adj += w * row[idx]
        fwd[v] = acc.view(spread, n + 2).sum(0)[:n]
        fwd[v, 0] = 0.0
    return fwd, adj.flip(0)


def _exact_dd(x, b, n, na, dev):
    nh = n // 2
    fwd, adj = torch.zeros((na, n), dtype=torch.float64, device=dev), torch.zeros((n, n), dtype=torch.float64, device=dev)
    u = torch.arange(n + 1, dtype=torch.float32, device=dev) - nh
    for v, th in enumerate(_rad("dd", na)):
        s, c = _sc(th)
        out = na - 1 - v
        y = b[out].double()
        if abs(float(s)) < 1e-7:
            fwd[out] = x.double().sum(1)
            adj += y[:, None]
            continue
        if abs(float(c)) < 1e-7:
            fwd[out] = x.double().sum(0)
            adj += y[None, :]
            continue
        rows = float(th) > PI / 2
        r = np.float32(1.0) / (s if rows else c)
        k = (c if rows else s) * r
        L = (x if rows else x.t()).double()
        q = (u[:n] + 0.5) * float(k)
        P, D = u[None, :] - q[:, None], u * float(r)
        # the last overlap piece of a line, up to the first boundary numbered n, is not credited
        first_p = P[:, n] <= D[n]
        before_p = torch.searchsorted(D, P[:, n].contiguous()) - 1
        at_p = torch.maximum(P[:, n - 1], torch.where(before_p >= 0, D[before_p.clamp(min=0)], torch.full_like(q, -1e30)))
        below_d = (torch.searchsorted(P.contiguous(), D[n].expand(n, 1).contiguous(), right=True) - 1)[:, 0]
        at_d = torch.maximum(D[n - 1], torch.where(below_d >= 0, torch.gather(P, 1, below_d.clamp(min=0)[:, None])[:, 0], torch.full_like(q, -1e30)))
        cut = torch.where(first_p, at_p, at_d).double()[:, None]
        P, Dd = P.double(), D.double()
        # forward: the line's integral up to each detector boundary
        S = torch.zeros((n, n + 1), dtype=torch.float64, device=dev)
        S[:, 1:] = torch.cumsum(L * (P[:, 1:] - P[:, :-1]), 1)
        B = torch.minimum(Dd[None, :].expand(n, n + 1), cut).contiguous()
        kk = (torch.searchsorted(P.contiguous(), B, right=True) - 1).clamp(0, n - 1)
        pk = torch.gather(P, 1, kk)
        F = torch.gather(S, 1, kk) + (torch.minimum(B, P[:, n:]) - pk).clamp(min=0.0) * torch.gather(L, 1, kk)
        fwd[out] = (F[:, 1:] - F[:, :-1]).sum(0)
        # adjoint: the detector row's integral up to each pixel boundary
        G = torch.zeros(n + 1, dtype=torch.float64, device=dev)
        G[1:] = torch.cumsum(y * (Dd[1:] - Dd[:-1]), 0)
        E = torch.minimum(torch.minimum(P, cut), Dd[n]).contiguous()
        m = (torch.searchsorted(Dd, E, right=True) - 1).clamp(0, n - 1)
        I = G[m] + (E - Dd[m]).clamp(min=0.0) * y[m]
        W = I[:, 1:] - I[:, :-1]
        adj += W if rows else W.t()
    return fwd, adj


def _round_away(v):
    return torch.where(v >= 0, torch.floor(v.double() + 0.5), torch.ceil(v.double() - 0.5))


def _exact_ss(x, b, n, na, dev):
    nh = n // 2
    fwd, adj = torch.zeros((na, n), dtype=torch.float64, device=dev), torch.zeros((n, n), dtype=torch.float64, device=dev)
    t = torch.arange(-nh, nh, dtype=torch.float32, device=dev)
    m = torch.arange(-nh, nh, dtype=torch.float32, device=dev)
    for v, th in enumerate(_rad("ss", na)):
        s, c = _sc(th)
        out, fn, fn1 = na - 1 - v, float(nh), float(nh - 1)
        steep = abs(float(s)) <= 0.70710678118654757
        a, den = (s, c) if steep else (c, s)
        if abs(float(s)) < 1e-5 or abs(float(c)) < 1e-5:
            lo, hi = torch.full_like(t, -fn), torch.full_like(t, fn1)
        else:
            o, e = (c, s) if steep else (s, c)  # limits of the major coordinate
            e0, e1 = _fma(torch.full_like(t, fn), o, t) / float(e), _fma(torch.full_like(t, -fn1), o, t) / float(e)
            q = torch.sort(torch.stack([e0, e1, torch.full_like(t, -fn), torch.full_like(t, fn1)]), 0)[0]
            lo, hi = q[1], q[2]
        lo, hi = _round_away(lo), _round_away(hi)
        rb, wt = np.float32(1.0) / den, 1.0 / abs(float(den))
        f = _fma(-m[:, None], float(a), t[None, :].expand(2 * nh, 2 * nh)) * float(rb)
        fl = torch.floor(f)
        on = (m[:, None] >= lo[None, :]) & (m[:, None] < hi[None, :])
        M = (x if steep else x.t())[: 2 * nh].double()
        row = b[out, : 2 * nh].double()[None, :]
        W = torch.zeros((2 * nh, n), dtype=torch.float64, device=dev)
        acc = torch.zeros(2 * nh, dtype=torch.float64, device=dev)
        for tap, w in ((0, (fl + 1.0) - f), (1, f - fl)):
            q = fl.long() + nh + tap
            ok = on & (q >= 0) & (q < n)
            w = torch.where(ok, wt * w.double(), torch.zeros((), dtype=torch.float64, device=dev))
            q = q.clamp(0, n - 1)
            acc += (w * torch.gather(M, 1, q)).sum(0)
            W.scatter_add_(1, q, w * row)
        fwd[out, : 2 * nh] = acc
        if steep:
            adj[: 2 * nh] += W
        else:
            adj[:, : 2 * nh] += W.t()
    return fwd, adj


def _exact_bspline(x, b, n, na, dev, lut):
    """``lut``: the table of the spline's Radon transform, which the projector takes as data."""
    support, size = 4.0, lut.shape[1]
    step, ds, mid = np.float32((size * 0.5) / (support * 0.5)), int(0.5 * support + 0.5), 0.5 * n
    fwd, adj = torch.zeros((na, n), dtype=torch.float64, device=dev), torch.zeros((n, n), dtype=torch.float64, device=dev)
    ar = torch.arange(n, dtype=torch.float32, device=dev)
    deg = ((np.arange(na) * 180.0) / np.float32(na)).astype(np.float32)
    lut = torch.from_numpy(lut).to(dev)
    spread = 32
    lane = (torch.arange(n, device=dev) % spread)[:, None] * (n + 1)
    for v in range(na):
        s, c = _sc(np.float32(float(deg[v]) * (PI / 180.0)))
        ky, kx = (-ar + mid)[:, None], (ar - mid)[None, :]
        ps = _fma(kx.expand(n, n), float(c), (ky * float(s)).expand(n, n))
        acc = torch.zeros(spread * (n + 1), dtype=torch.float64, device=dev)
        row = torch.cat([b[v].double(), torch.zeros(1, dtype=torch.float64, device=dev)])
        for k in range(-ds, ds + 1):
            yi = torch.trunc((k + ps).double() + mid)
            li = torch.trunc(((yi - mid).float() - ps) * float(step)).long() + size // 2
            ok = (yi >= 0) & (yi < n) & (li >= 0) & (li < size - 1)
            w = torch.where(ok, lut[v][li.clamp(0, size - 1)].double(), torch.zeros((), dtype=torch.float64, device=dev))
            idx = torch.where(ok, yi, torch.full_like(yi, n)).long()
            acc.index_add_(0, (idx + lane).reshape(-1), (w * x.double()).reshape(-1))
            adj += w * row[idx]
        fwd[v] = acc.view(spread, n + 1).sum(0)[:n]
    return fwd, adj


def _exact_rd(x, b, n, na, dev):
    """Every sub-ray's walk, all rays one step at a time."""
    nh = n // 2
    fwd, adj = torch.zeros(na * n, dtype=torch.float64, device=dev), torch.zeros(n * n, dtype=torch.float64, device=dev)
    img, sino = x.double().reshape(-1), b.double().reshape(-1)
    p1s, p2s, idxs = [], [], []
    i = np.array([k for k in range(1, 6 * n) if k % 6])
    for v, th in enumerate(_rad("rd", na)):
        s, c = _sc(th)
        if abs(float(s)) < 1e-7:
            cols = x.double().sum(0)
            fwd[v * n + n - 1 - torch.arange(1, n, device=dev)] = cols[1:]
            adj.view(n, n)[:, 1:] += b[v].double()[n - 1 - torch.arange(1, n, device=dev)][None, :]
            continue
        if abs(float(c)) < 1e-7:
            fwd[v * n:(v + 1) * n] = x.double().sum(1)
            adj.view(n, n)[:] += b[v].double()[:, None]
            continue
        f32, fn = np.float32, np.float32(nh)
        t = np.abs(i.astype(np.float64) / 6.0 - nh).astype(f32)
        left = float(th) < PI / 2
        t = np.where((i >= 3 * n) if left else (i < 3 * n), -t, t) if float(th) != PI / 2 else t
        rc, rs = f32(1) / c, f32(1) / s
        if left:
            y1, x1, y2, x2 = (-fn * s + t) * rc, (-fn * c - t) * rs, (fn * s + t) * rc, (fn * c - t) * rs
            e1, e2 = -fn, fn
        else:
            y1, x1, y2, x2 = (fn * s - t) * rc, (-fn * c + t) * rs, (-fn * s - t) * rc, (fn * c + t) * rs
            e1, e2 = fn, -fn
        in1, in2 = (y1 >= -fn) & (y1 <= fn), (y2 >= -fn) & (y2 <= fn)
        p1s.append(np.stack([np.where(in1, e1, x1), np.where(in1, y1, -fn)]))
        p2s.append(np.stack([np.where(in2, e2, x2), np.where(in2, y2, fn)]))
        idxs.append(v * n + i // 6)
    p1 = torch.from_numpy(np.concatenate(p1s, 1).astype(np.float32)).to(dev)
    p2 = torch.from_numpy(np.concatenate(p2s, 1).astype(np.float32)).to(dev)
    idx = torch.from_numpy(np.concatenate(idxs)).to(dev)
    y = sino[idx]
    e = p2 - p1
    inc = torch.sqrt(_fma(e[0], e[0], e[1] * e[1]))
    pix = _round_away(p1)
    d = torch.where(p2 > p1, 1.0, -1.0).double()
    p1, e = p1.double(), e.double()
    alpha = torch.zeros_like(inc)
    acc = torch.zeros(idx.numel(), dtype=torch.float64, device=dev)
    for _ in range(4 * n + 16):
        a = ((pix + 0.5 * d - p1) / e).float()
        ax, ay = a[0], a[1]
        live = alpha <= 1.0
        new = torch.where(ax < ay, ax, ay)
        pix[0] += torch.where(live & (ax <= ay), d[0], torch.zeros_like(d[0]))
        pix[1] += torch.where(live & (ay <= ax), d[1], torch.zeros_like(d[1]))
        l = 0.2 * ((new - alpha) * inc).double()
        ii, jj = pix[0].long() + nh, pix[1].long() + nh
        at = torch.where(live & (ii > 0) & (ii < n) & (jj > 0) & (jj < n), ii * n + jj, torch.full_like(ii, -1))
        ok = at >= 0
        l = torch.where(ok, l, torch.zeros_like(l))
        at = at.clamp(min=0)
        acc += l * img[at]
        adj.index_add_(0, at, l * y)
        alpha = torch.where(live, new, alpha)
        if _ % 64 == 0 and not bool((alpha <= 1.0).any()):
            break
    fwd.index_add_(0, idx, acc)
    return fwd.view(na, n), adj.view(n, n)


def exact(case, seed):
    dev, path = _device(), case["path"]
    if path == "pair":
        oper, n, na, nz = case["oper"], case["n"], case["na"], case["nz"]
        most = {"pd": 1.3e9, "dd": 8e9, "ss": 2e9, "bspline": 1.2e9, "rd": 4e8}.get(oper, 0)
        if n * n * na * nz > most:
            return None  # the gridding pair: a chain of float32 tables and transforms with no 64-bit form of its own
        x, b = _pair_inputs(case, seed, dev)
        if oper == "bspline":
            lut = _projector(oper, n, na).lut
            both = [_exact_bspline(x[z], b[z], n, na, dev, lut) for z in range(nz)]
        else:
            fn = {"pd": _exact_pd, "dd": _exact_dd, "ss": _exact_ss, "rd": _exact_rd}[oper]
            both = [fn(x[z], b[z], n, na, dev) for z in range(nz)]
        return {"Ax": torch.stack([p[0] for p in both]), "Atb": torch.stack([p[1] for p in both])}
    if path == "conv":
        X, Wt, bias, dY = _conv_inputs(case, seed, dev)
        if X.numel() * case["cout"] > 2.5e9:
            return None
        x, w = X.double().permute(0, 3, 1, 2), Wt.to(torch.bfloat16).double().permute(0, 3, 1, 2)
        g = dY.double().permute(0, 3, 1, 2)

        def shifts(a):
            return torch.nn.functional.pad(a, (1, 1, 1, 1))
        H, W_ = x.shape[2:]
        xp, gp = shifts(x), shifts(g)
        Y, dX, dW = 0.0, 0.0, torch.empty(Wt.shape, dtype=torch.float64, device=dev)
        for ky in range(3):
            for kx in range(3):
                xs = xp[:, :, ky:ky + H, kx:kx + W_]
                Y = Y + torch.einsum("oc,bchw->bhwo", w[:, :, ky, kx], xs)
                dX = dX + torch.einsum("oc,bohw->bhwc", w[:, :, ky, kx], gp[:, :, 2 - ky:2 - ky + H, 2 - kx:2 - kx + W_])
                dW[:, ky, kx, :] = torch.einsum("bohw,bchw->oc", g, xs)
        Y = torch.relu(Y + bias.double())
        return {"Y": Y, "dX": dX, "dW": dW.reshape(dW.shape[0], 9, -1), "db": g.sum((0, 2, 3))}
    return None  # whole calls: rounding travels through their layers and iterations
