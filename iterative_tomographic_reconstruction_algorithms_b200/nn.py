"""Learned warm start: tensor-core convolution kernels and a small U-Net.

The network maps a cheap reconstruction (2 SIRT iterations) to a start close
to the converged SIRT result; the plain solver then continues from it.  All
convolutions -- forward, input gradient and weight gradient -- are the
hand-written tcgen05 BF16 kernels of ``libtomo_nn.so`` (``csrc/nn_conv.cu``,
``csrc/nn_wgrad.cu``, ``csrc/nn_gemm.cu``) with FP32 accumulation and FP32 master
weights; pooling, upsampling beside the skip connection and their gradients are
passes of its own (``csrc/nn_resample.cu``).  Activations are BF16 NHWC.

Layers (``UNet(levels=4, base=32)``): per level two 3x3 convolutions + ReLU,
2x2 max-pooling down, nearest 2x upsampling up with the skip connection
concatenated, a final 1x1 convolution, and the input added back (the network
predicts a correction).
"""
from __future__ import annotations

import ctypes
import math
import os
from pathlib import Path

import torch

PKG_DIR = Path(__file__).resolve().parent
LIB_PATH = PKG_DIR / "libtomo_nn.so"

__all__ = ["gemm", "conv3x3", "wgrad", "UNet", "Adam", "check_status"]


def _load():
    if not LIB_PATH.exists():
        raise ImportError(f"{LIB_PATH} is missing: build it with `make -C {PKG_DIR / 'csrc'}`")
    lib = ctypes.CDLL(str(LIB_PATH), mode=os.RTLD_GLOBAL)
    vp, i, f, sz = ctypes.c_void_p, ctypes.c_int, ctypes.c_float, ctypes.c_size_t
    lib.tomo_nn_gemm.argtypes = [vp, i, vp, i, i, i, i, vp, vp, i, vp, i, vp]
    lib.tomo_nn_conv3x3.argtypes = [vp, i, i, i, i, vp, i, vp, vp, vp, i, vp]
    lib.tomo_nn_wgrad_workspace.argtypes = [i, i, i, i, i, i]
    lib.tomo_nn_wgrad_workspace.restype = sz
    lib.tomo_nn_wgrad.argtypes = [vp, vp, i, i, i, i, i, i, vp, vp, vp, sz, vp]
    lib.tomo_nn_prepare_weights.argtypes = [vp, i, i, i, vp, vp, vp]
    lib.tomo_nn_conv3x3_masked.argtypes = [vp, i, i, i, i, vp, i, vp, vp, vp]
    lib.tomo_nn_pool.argtypes = [vp, i, i, i, i, vp, vp]
    lib.tomo_nn_pool_bwd.argtypes = [vp, vp, vp, i, i, i, i, i, vp, vp]
    lib.tomo_nn_upcat.argtypes = [vp, vp, i, i, i, i, i, vp, vp]
    lib.tomo_nn_up_bwd.argtypes = [vp, i, vp, i, i, i, i, vp, vp]
    lib.tomo_nn_pad8.argtypes = [vp, ctypes.c_longlong, vp, vp]
    lib.tomo_nn_head_bwd.argtypes = [vp, vp, vp, ctypes.c_longlong, i, vp, vp]
    lib.tomo_nn_relu_bwd.argtypes = [vp, vp, sz, vp]
    lib.tomo_nn_adam.argtypes = [vp, vp, vp, vp, sz, f, f, f, f, i, vp]
    lib.tomo_nn_status.argtypes = [ctypes.POINTER(ctypes.c_uint)]
    return lib


lib = _load()


def _check(rc, what):
    if rc != 0:
        raise RuntimeError(f"{what} failed with status {rc}")


def _stream(t):
    return ctypes.c_void_p(torch.cuda.current_stream(t.device).cuda_stream)


def _p(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def set_wait_limit(spins: int) -> None:
    """Polls of a tensor-core pipeline wait before it gives up (tomo_nn.h:
    tomo_nn_set_wait_limit); a negative value restores the default."""
    lib.tomo_nn_set_wait_limit.argtypes = [ctypes.c_int]
    _check(lib.tomo_nn_set_wait_limit(int(spins)), "tomo_nn_set_wait_limit")


def check_status():
    """Raises if a tensor-core wait gave up in any kernel since the last check."""
    flags = ctypes.c_uint()
    _check(lib.tomo_nn_status(ctypes.byref(flags)), "tomo_nn_status")
    if flags.value:
        raise RuntimeError(f"tensor-core kernel reported status {flags.value:#x} (a wait gave up)")


def gemm(A, B, bias=None, relu=False, out_dtype=torch.float32):
    """A [M, K] . B [N, K]^T (BF16 CUDA tensors, K % 8 == 0) -> [M, N]."""
    M, K = A.shape
    N = B.shape[0]
    out = torch.empty((M, N), dtype=out_dtype, device=A.device)
    f32 = out_dtype == torch.float32
    _check(lib.tomo_nn_gemm(_p(A), A.stride(0), _p(B), B.stride(0), M, N, K, _p(out) if f32 else None,
                            None if f32 else _p(out), N, _p(bias), int(relu), _stream(A)), "tomo_nn_gemm")
    return out


def conv3x3(X, Wb, bias=None, relu=False, out_dtype=torch.bfloat16):
    """X [B, H, W, Cin] BF16, Wb [Cout, 3, 3, Cin] BF16 -> [B, H, W, Cout]."""
    B, H, W, Cin = X.shape
    Cout = Wb.shape[0]
    out = torch.empty((B, H, W, Cout), dtype=out_dtype, device=X.device)
    f32 = out_dtype == torch.float32
    _check(lib.tomo_nn_conv3x3(_p(X), B, H, W, Cin, _p(Wb), Cout, _p(out) if f32 else None,
                               None if f32 else _p(out), _p(bias), int(relu), _stream(X)), "tomo_nn_conv3x3")
    return out


def wgrad(X, dY, taps):
    """Weight and bias gradients of a 3x3 (taps=9) or 1x1 (taps=1) convolution."""
    B, H, W, Cin = X.shape
    Cout = dY.shape[-1]
    dW = torch.empty((Cout, taps, Cin), dtype=torch.float32, device=X.device)
    db = torch.empty((Cout,), dtype=torch.float32, device=X.device)
    nbytes = lib.tomo_nn_wgrad_workspace(B, H, W, Cin, Cout, taps)
    work = torch.empty((nbytes,), dtype=torch.uint8, device=X.device)
    _check(lib.tomo_nn_wgrad(_p(X), _p(dY), B, H, W, Cin, Cout, taps, _p(dW), _p(db), _p(work), nbytes,
                             _stream(X)), "tomo_nn_wgrad")
    return dW, db


def prepare_weights(W, with_transpose=True):
    """FP32 [Cout, taps, Cin] -> (BF16 copy, BF16 [Cin, taps, Cout] with the taps reversed)."""
    Cout, taps, Cin = W.shape
    Wb = torch.empty_like(W, dtype=torch.bfloat16)
    Wd = torch.empty((Cin, taps, Cout), dtype=torch.bfloat16, device=W.device) if with_transpose else None
    _check(lib.tomo_nn_prepare_weights(_p(W), Cout, Cin, taps, _p(Wb), _p(Wd), _stream(W)),
           "tomo_nn_prepare_weights")
    return Wb, Wd


def _conv3x3_dx(dZ, Wd, X=None):
    """Input gradient [B, H, W, Cin]; with X, where the input X is > 0 (through the ReLU that made it)."""
    B, H, W, Cin = dZ.shape
    Cout = Wd.shape[0]
    if X is None:
        return conv3x3(dZ, Wd.reshape(Cout, 3, 3, Cin))
    out = torch.empty((B, H, W, Cout), dtype=torch.bfloat16, device=dZ.device)
    _check(lib.tomo_nn_conv3x3_masked(_p(dZ), B, H, W, Cin, _p(Wd), Cout, _p(X), _p(out), _stream(dZ)),
           "tomo_nn_conv3x3_masked")
    return out


def _bf16(d):
    return d.to(torch.bfloat16).contiguous()


# The network's layers.  A layer's incoming gradient has already gone through
# the ReLU at its output: whoever consumes that output has it at hand and
# applies it while writing the gradient.

class _Conv3x3(torch.autograd.Function):
    """3x3 convolution + bias + ReLU; mask_dx: the input is a ReLU's output."""

    @staticmethod
    def forward(ctx, X, W, b, need_dx, mask_dx):
        Wb, Wd = prepare_weights(W.detach().reshape(W.shape[0], 9, W.shape[-1]), with_transpose=need_dx)
        Y = conv3x3(X, Wb.reshape(W.shape), b.detach(), relu=True)
        ctx.save_for_backward(X, Wd if need_dx else None)
        ctx.need_dx, ctx.mask_dx = need_dx, mask_dx
        return Y

    @staticmethod
    def backward(ctx, dY):
        X, Wd = ctx.saved_tensors
        dZ = _bf16(dY)
        dW, db = wgrad(X, dZ, 9)
        dX = _conv3x3_dx(dZ, Wd, X if ctx.mask_dx else None) if ctx.need_dx else None
        return dX, dW.reshape(dW.shape[0], 3, 3, dW.shape[-1]), db, None, None


class _Conv3x3Pool(torch.autograd.Function):
    """3x3 convolution + bias + ReLU of a ReLU's output, and its 2x2 max-pooling."""

    @staticmethod
    def forward(ctx, X, W, b):
        Wb, Wd = prepare_weights(W.detach().reshape(W.shape[0], 9, W.shape[-1]))
        Y = conv3x3(X, Wb.reshape(W.shape), b.detach(), relu=True)
        B, H, W_, C = Y.shape
        P = torch.empty((B, H // 2, W_ // 2, C), dtype=torch.bfloat16, device=Y.device)
        _check(lib.tomo_nn_pool(_p(Y), B, H // 2, W_ // 2, C, _p(P), _stream(Y)), "tomo_nn_pool")
        ctx.save_for_backward(X, Y, Wd)
        return Y, P

    @staticmethod
    def backward(ctx, dS, dP):
        X, Y, Wd = ctx.saved_tensors
        B, H, W, C = Y.shape
        dP, dS = _bf16(dP), dS.to(torch.bfloat16)
        ld = dS.stride(2)
        # the skip's gradient comes as a slice of the concatenation's channels
        if dS.stride() != (H * W * ld, W * ld, ld, 1) or ld < C or ld % 8 or dS.data_ptr() % 16:
            dS, ld = dS.contiguous(), C
        dZ = torch.empty_like(Y)
        _check(lib.tomo_nn_pool_bwd(_p(Y), _p(dP), _p(dS), ld, B, H // 2, W // 2, C, _p(dZ), _stream(Y)),
               "tomo_nn_pool_bwd")
        dW, db = wgrad(X, dZ, 9)
        return _conv3x3_dx(dZ, Wd, X), dW.reshape(dW.shape[0], 3, 3, dW.shape[-1]), db


class _UpCat(torch.autograd.Function):
    """A ReLU's output upsampled by 2 (nearest) beside the skip's channels."""

    @staticmethod
    def forward(ctx, X, S):
        B, h, w, Cu = X.shape
        Cs = S.shape[-1]
        Y = torch.empty((B, 2 * h, 2 * w, Cu + Cs), dtype=torch.bfloat16, device=X.device)
        _check(lib.tomo_nn_upcat(_p(X), _p(S), B, h, w, Cu, Cs, _p(Y), _stream(X)), "tomo_nn_upcat")
        ctx.save_for_backward(X)
        return Y

    @staticmethod
    def backward(ctx, dY):
        X, = ctx.saved_tensors
        B, h, w, Cu = X.shape
        d = _bf16(dY)
        dX = torch.empty_like(X)
        _check(lib.tomo_nn_up_bwd(_p(d), d.shape[-1], _p(X), B, h, w, Cu, _p(dX), _stream(d)), "tomo_nn_up_bwd")
        return dX, d[..., Cu:]


class _Head(torch.autograd.Function):
    """First output of a 1x1 convolution with 8 outputs on a ReLU's output, + bias, FP32 [B, H, W]."""

    @staticmethod
    def forward(ctx, X, W, b):
        Bn, H, W_, Cin = X.shape
        Wb, Wt = prepare_weights(W.detach().reshape(W.shape[0], 1, Cin), with_transpose=True)
        Y = gemm(X.reshape(-1, Cin), Wb.reshape(W.shape[0], Cin)[:1], bias=b.detach())
        ctx.save_for_backward(X, Wt)
        return Y.reshape(Bn, H, W_)

    @staticmethod
    def backward(ctx, dY):
        X, Wt = ctx.saved_tensors
        Bn, H, W_, Cin = X.shape
        d = dY.to(torch.float32).contiguous()
        dZ = torch.empty((Bn, H, W_, 8), dtype=torch.bfloat16, device=X.device)
        _check(lib.tomo_nn_pad8(_p(d), d.numel(), _p(dZ), _stream(d)), "tomo_nn_pad8")
        dW, db = wgrad(X, dZ, 1)
        if Cin <= 1024:
            dX = torch.empty_like(X)
            _check(lib.tomo_nn_head_bwd(_p(dZ), _p(Wt), _p(X), d.numel(), Cin, _p(dX), _stream(d)), "tomo_nn_head_bwd")
        else:  # its weights no longer fit that kernel's shared memory
            dX = gemm(dZ.reshape(-1, 8), Wt.reshape(Cin, 8), out_dtype=torch.bfloat16).reshape(X.shape)
            _check(lib.tomo_nn_relu_bwd(_p(X), _p(dX), dX.numel(), _stream(d)), "tomo_nn_relu_bwd")
        return dX, dW.reshape(dW.shape[0], Cin), db


class UNet(torch.nn.Module):
    """U-Net with ``levels`` resolutions and ``base`` channels at the top level.

    ``forward(x)``: x FP32 [B, H, W] (H, W divisible by 2^(levels-1)) -> FP32
    [B, H, W] = x + correction.  Input channels are padded to 8 with zeros.
    """

    CIN = 8

    def __init__(self, levels: int = 4, base: int = 32, seed: int = 0):
        super().__init__()
        g = torch.Generator().manual_seed(seed)
        self.levels = levels
        ch = [base * 2 ** i for i in range(levels)]
        self.enc, self.dec = torch.nn.ParameterList(), torch.nn.ParameterList()

        def conv(cin, cout, store):
            w = torch.randn((cout, 3, 3, cin), generator=g) * math.sqrt(2.0 / (9 * cin))
            store.append(torch.nn.Parameter(w))
            store.append(torch.nn.Parameter(torch.zeros(cout)))

        cin = self.CIN
        for c in ch:
            conv(cin, c, self.enc)
            conv(c, c, self.enc)
            cin = c
        for c in reversed(ch[:-1]):
            conv(cin + c, c, self.dec)
            conv(c, c, self.dec)
            cin = c
        self.head_w = torch.nn.Parameter(torch.zeros((8, cin)))
        self.head_b = torch.nn.Parameter(torch.zeros(8))

    def forward(self, x, extra=None):
        """``extra``: optional further input channels, FP32 [B, H, W] or [B, H, W, k] (k <= 7)."""
        B, H, W = x.shape
        if H % 2 ** (self.levels - 1) or W % 2 ** (self.levels - 1):
            raise RuntimeError(f"sides {H} x {W} are not multiples of {2 ** (self.levels - 1)}")
        h = torch.zeros((B, H, W, self.CIN), dtype=torch.bfloat16, device=x.device)
        h[..., 0] = x.to(torch.bfloat16)
        if extra is not None:
            e = extra if extra.dim() == 4 else extra[..., None]
            h[..., 1:1 + e.shape[-1]] = e.to(torch.bfloat16)
        skips = []
        for lvl in range(self.levels):
            w1, b1, w2, b2 = self.enc[4 * lvl:4 * lvl + 4]
            h = _Conv3x3.apply(h, w1, b1, lvl > 0, False)
            if lvl < self.levels - 1:
                skip, h = _Conv3x3Pool.apply(h, w2, b2)
                skips.append(skip)
            else:
                h = _Conv3x3.apply(h, w2, b2, True, True)
        for j in range(self.levels - 1):
            w1, b1, w2, b2 = self.dec[4 * j:4 * j + 4]
            h = _UpCat.apply(h, skips[-1 - j])
            h = _Conv3x3.apply(h, w1, b1, True, False)
            h = _Conv3x3.apply(h, w2, b2, True, True)
        return x + _Head.apply(h, self.head_w, self.head_b)


class Adam:
    """Adam on FP32 parameters with the ``tomo_nn_adam`` kernel."""

    def __init__(self, params, lr=1e-3, betas=(0.9, 0.999), eps=1e-8):
        self.params = [p for p in params]
        self.lr, self.b1, self.b2, self.eps = lr, betas[0], betas[1], eps
        self.m = [torch.zeros_like(p) for p in self.params]
        self.v = [torch.zeros_like(p) for p in self.params]
        self.t = 0

    def zero_grad(self):
        for p in self.params:
            p.grad = None

    @torch.no_grad()
    def step(self):
        self.t += 1
        for p, m, v in zip(self.params, self.m, self.v):
            if p.grad is None:
                continue
            g = p.grad.contiguous()
            _check(lib.tomo_nn_adam(_p(p), _p(g), _p(m), _p(v), p.numel(), self.lr, self.b1, self.b2, self.eps,
                                    self.t, _stream(p)), "tomo_nn_adam")
