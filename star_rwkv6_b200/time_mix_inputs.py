"""Input stage of the time-mix block: from the block input x to the five tensors that feed the r, k, v, w, g
projections (TimeMix.call, rwkv6_model.py:128-146):

    x_shift = shift(x) - x                              (TimeShift, rwkv6_model.py:37-44)
    x_mix   = x + x_shift * time_mix_x
    l_i     = tanh(x_mix A_i) B_i + b_i                 (DecomposerDense, rwkv6_model.py:11-24), i in r, k, v, w, g
    x_i     = x + x_shift * l_i

The interpolation steps are fused kernels (x is read once, no shifted copy is materialised).  For bf16 with the usual rank
of 32 the products with B_i run inside the second one (``wkv6_lora_mix_forward / _backward``), so that the l_i exist in
registers only; otherwise they are a batched library product in front of ``wkv6_shift_mix_forward / _backward``.
"""
from __future__ import annotations

import ctypes

import torch

from ._lib import check, lib
from .layer_norm import _dense16
from .ops import _DT, _check_cuda, _ptr, _stream


def _shift_mix_fwd(x, m, vector: bool):
    B, T, C = x.shape
    nmix = 1 if vector else m.shape[0]
    out = torch.empty((B, T, C) if vector else (nmix, B, T, C), dtype=x.dtype, device=x.device)
    with torch.cuda.device(x.device):
        check(lib.wkv6_shift_mix_forward(B, T, C, _DT[x.dtype], nmix, 1 if vector else 0, _ptr(x), _ptr(m), _ptr(out),
                                         _stream(x.device)))
    return out


def _shift_mix_bwd(x, m, gout, vector: bool):
    B, T, C = x.shape
    nmix = 1 if vector else m.shape[0]
    gx = torch.empty_like(x)
    gm = torch.empty((C,), dtype=torch.float32, device=x.device) if vector else torch.empty_like(m)
    nbytes = lib.wkv6_shift_mix_workspace_bytes(B, T, C, 1 if vector else 0)
    ws = torch.empty((nbytes,), dtype=torch.uint8, device=x.device) if nbytes else None
    with torch.cuda.device(x.device):
        check(lib.wkv6_shift_mix_backward(B, T, C, _DT[x.dtype], nmix, 1 if vector else 0, _ptr(x), _ptr(m), _ptr(gout),
                                          _ptr(gx), _ptr(gm), _ptr(ws), nbytes, _stream(x.device)))
    return gx, gm


class _ShiftMixVec(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, mu):
        _check_cuda(x, mu)
        x = x.contiguous()
        mu32 = mu.detach().to(torch.float32).contiguous()
        ctx.save_for_backward(x, mu32)
        ctx.mu_dtype = mu.dtype
        return _shift_mix_fwd(x, mu32, True)

    @staticmethod
    def backward(ctx, gout):
        x, mu32 = ctx.saved_tensors
        gx, gmu = _shift_mix_bwd(x, mu32, gout.to(x.dtype).contiguous(), True)
        return gx, gmu.to(ctx.mu_dtype)


class _ShiftMixTensors(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, m):
        _check_cuda(x, m)
        x, m = x.contiguous(), m.contiguous()
        assert m.dtype == x.dtype and m.shape[1:] == x.shape and m.shape[0] in (1, 5)
        ctx.save_for_backward(x, m)
        return _shift_mix_fwd(x, m, False)

    @staticmethod
    def backward(ctx, gout):
        x, m = ctx.saved_tensors
        return _shift_mix_bwd(x, m, gout.to(x.dtype).contiguous(), False)


class _ShiftMixPair(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, mu0, mu1, separate_gx):
        _check_cuda(x, mu0, mu1)
        x = x.contiguous()
        mu = [m.detach().to(torch.float32).contiguous() for m in (mu0, mu1)]
        ctx.save_for_backward(x, *mu)
        ctx.mu_dtypes, ctx.separate_gx = (mu0.dtype, mu1.dtype), separate_gx
        B, T, C = x.shape
        out = [torch.empty_like(x) for _ in range(2)]
        with torch.cuda.device(x.device):
            check(lib.wkv6_shift_mix_pair_forward(B, T, C, _DT[x.dtype], _ptr(x), _ptr(mu[0]), _ptr(mu[1]), _ptr(out[0]), _ptr(out[1]),
                                                  _stream(x.device)))
        return tuple(out)

    @staticmethod
    def backward(ctx, g0, g1):
        x, mu0, mu1 = ctx.saved_tensors
        B, T, C = x.shape
        g0, g1 = g0.to(x.dtype).contiguous(), g1.to(x.dtype).contiguous()
        if ctx.separate_gx:
            (gx, gmu0), (gx1, gmu1) = _shift_mix_bwd(x, mu0, g0, True), _shift_mix_bwd(x, mu1, g1, True)
            return gx.add_(gx1), gmu0.to(ctx.mu_dtypes[0]), gmu1.to(ctx.mu_dtypes[1]), None
        gx = torch.empty_like(x)
        gmu = [torch.empty((C,), dtype=torch.float32, device=x.device) for _ in range(2)]
        nbytes = lib.wkv6_shift_mix_workspace_bytes(B, T, C, 2)
        ws = torch.empty((nbytes,), dtype=torch.uint8, device=x.device) if nbytes else None
        with torch.cuda.device(x.device):
            check(lib.wkv6_shift_mix_pair_backward(B, T, C, _DT[x.dtype], _ptr(x), _ptr(mu0), _ptr(mu1), _ptr(g0), _ptr(g1), _ptr(gx),
                                                   _ptr(gmu[0]), _ptr(gmu[1]), _ptr(ws), nbytes, _stream(x.device)))
        return gx, gmu[0].to(ctx.mu_dtypes[0]), gmu[1].to(ctx.mu_dtypes[1]), None


def _pointers(ts):
    return (ctypes.c_void_p * len(ts))(*[t.data_ptr() for t in ts])


def _lora_mix_fwd(x, h, wb, bias, out):
    B, T, C = x.shape
    with torch.cuda.device(x.device):
        check(lib.wkv6_lora_mix_forward(B, T, C, _ptr(x), _ptr(h), _ptr(wb), _ptr(bias), _pointers(out), _stream(x.device)))


class _LoraMix(torch.autograd.Function):
    """The five x + (shift(x) - x) * (bias_j + h_j wb_j) for x [B,T,C], h [B*T, 160], wb [5, 32, C], bias [5, 1, C], all bf16:
    five tensors, or one [5, B, T, C] (``stacked``)."""

    @staticmethod
    def forward(ctx, x, h, wb, bias, stacked):
        x, h, wb, bias = (t.contiguous() for t in (x, h, wb, bias))
        ctx.save_for_backward(x, h, wb, bias)
        ctx.stacked = stacked
        out = torch.empty((5, *x.shape), dtype=x.dtype, device=x.device) if stacked else [torch.empty_like(x) for _ in range(5)]
        _lora_mix_fwd(x, h, wb, bias, out)
        return out if stacked else tuple(out)

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, *gout):
        x, h, wb, bias = ctx.saved_tensors
        B, T, C = x.shape
        gout = [_dense16(g) for g in (gout[0] if ctx.stacked else gout)]
        gx = torch.empty_like(x)
        gl = torch.empty((5, B * T, C), dtype=x.dtype, device=x.device)
        with torch.cuda.device(x.device):
            check(lib.wkv6_lora_mix_backward(B, T, C, _ptr(x), _ptr(h), _ptr(wb), _ptr(bias), _pointers(gout), _ptr(gx), _ptr(gl),
                                             _stream(x.device)))
        h5 = h.view(B * T, 5, -1).permute(1, 2, 0)                                              # [5, 32, B*T]
        gh = torch.bmm(gl, wb.transpose(1, 2)).transpose(0, 1).reshape(h.shape)
        return gx, gh, torch.bmm(h5, gl), gl.sum(1, keepdim=True), None


def _lora_fits(x, h, wb, bias):
    return (x.is_cuda and x.dim() == 3 and x.numel() > 0 and x.shape[-1] % 8 == 0 and wb.shape == (5, 32, x.shape[-1])
            and all(t.dtype == torch.bfloat16 and t.device == x.device for t in (x, h, wb, bias))
            and all(t.data_ptr() % 16 == 0 for t in (x, h, wb, bias)))


def shift_mix_pair(x, mu0, mu1, separate_gx: bool = False):
    """(x + (shift(x) - x) * mu0, the same with mu1) for x [B,T,C] and two mixing vectors [C]: x is read once and gets one gradient.
    ``separate_gx``: that gradient with the bits of two ``shift_mix_vector`` calls, whose gradients are rounded before they are added
    (one pass more, backward)."""
    return _ShiftMixPair.apply(x, mu0, mu1, separate_gx)


def shift_mix_vector(x, mu):
    """x + (shift(x) - x) * mu for x [B,T,C] and one mixing vector mu [C]."""
    return _ShiftMixVec.apply(x, mu)


def shift_mix_tensors(x, m):
    """x + (shift(x) - x) * m[j] for x [B,T,C] and m [nmix,B,T,C] (nmix = 1 or 5); returns [nmix,B,T,C]."""
    return _ShiftMixTensors.apply(x, m)


class TimeMixInputs(torch.nn.Module):
    """The five mixed inputs (xr, xk, xv, xw, xg) of the reference's TimeMix from the block input."""

    ORDER = ("r", "k", "v", "w", "g")

    def __init__(self, hidden_size: int, decomposer_size: int = 32):
        super().__init__()
        D, R = hidden_size, decomposer_size
        self.hidden_size, self.decomposer_size = D, R
        self.time_mix_x = torch.nn.Parameter(torch.zeros(D))
        self.dense_a = torch.nn.Parameter(torch.randn(D, 5 * R) * D ** -0.5)   # dense_a of the five DecomposerDense, side by side
        self.dense_b = torch.nn.Parameter(torch.randn(5, R, D) * R ** -0.5)    # dense_b kernels
        self.bias_b = torch.nn.Parameter(torch.zeros(5, 1, D))                 # dense_b biases (use_bias=True)

    def forward(self, x):
        """[5, B, T, D]: xr, xk, xv, xw, xg stacked."""
        return self._mixes(x, True)

    def split(self, x):
        """The same as five tensors (their gradients need not be stacked again on the way back)."""
        return self._mixes(x, False)

    def _mixes(self, x, stacked):
        B, T, D = x.shape
        x_mix = shift_mix_vector(x, self.time_mix_x)
        h = torch.tanh(x_mix.reshape(B * T, D) @ self.dense_a.to(x.dtype))                      # [B*T, 5R]
        wb, bias = self.dense_b.to(x.dtype), self.bias_b.to(x.dtype)
        if _lora_fits(x, h, wb, bias):
            return _LoraMix.apply(x, h, wb, bias, stacked)
        h = h.reshape(B * T, 5, self.decomposer_size).transpose(0, 1)                            # [5, B*T, R]
        l = torch.baddbmm(bias, h, wb)                                                           # [5, B*T, D]
        return shift_mix_tensors(x, l.reshape(5, B, T, D))                                       # xr, xk, xv, xw, xg
