"""LayerNorm over the channels, with the residual addition in front of it folded in (the two norms of a block,
RWKV_Block in rwkv6_model.py:197-215): one kernel forward and one (plus the small parameter reduction) backward on the C ABI
(``wkv6_layer_norm_forward / _backward``), for bf16 activations and parameters.
"""
from __future__ import annotations

import torch
from torch import nn

from ._lib import check, lib
from .ops import _ptr, _stream

MAX_CHANNELS = 8192


def _raw(x, o, gamma, beta, eps, want_stat):
    D = x.shape[-1]
    rows = x.numel() // D
    s = torch.empty_like(x) if o is not None else x
    y = torch.empty_like(x)
    stat = torch.empty((rows, 2), dtype=torch.float32, device=x.device) if want_stat else None
    with torch.cuda.device(x.device):
        check(lib.wkv6_layer_norm_forward(rows, D, eps, _ptr(x), _ptr(o), _ptr(gamma), _ptr(beta), _ptr(s) if o is not None else None,
                                          _ptr(y), _ptr(stat), _stream(x.device)))
    return s, y, stat


class _ResidualLayerNorm(torch.autograd.Function):
    """(x, o or None) -> (s, LN(s)) with s = x + o; without o the first result is x itself, so that both of its uses come back
    through this node and the addition of their gradients happens in the kernel."""

    @staticmethod
    def forward(ctx, x, o, gamma, beta, eps):
        x = x.contiguous()
        s, y, stat = _raw(x, None if o is None else o.contiguous(), gamma, beta, eps, True)
        ctx.save_for_backward(s, gamma, stat)
        ctx.has_o = o is not None
        ctx.set_materialize_grads(False)
        return (s if o is not None else x.view_as(x)), y

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, gs, gy):
        s, gamma, stat = ctx.saved_tensors
        if gy is None:
            return gs, (gs if ctx.has_o else None), None, None, None
        D = s.shape[-1]
        rows = s.numel() // D
        gy = _dense16(gy)
        gs = None if gs is None else _dense16(gs)
        gx, gg, gb = torch.empty_like(s), torch.empty_like(gamma), torch.empty_like(gamma)
        nbytes = lib.wkv6_layer_norm_workspace_bytes(rows, D)
        ws = torch.empty((max(nbytes, 16),), dtype=torch.uint8, device=s.device)
        with torch.cuda.device(s.device):
            check(lib.wkv6_layer_norm_backward(rows, D, _ptr(s), _ptr(stat), _ptr(gamma), _ptr(gy), _ptr(gs), _ptr(gx), _ptr(gg), _ptr(gb),
                                               _ptr(ws), nbytes, _stream(s.device)))
        return gx, (gx if ctx.has_o else None), gg, gb, None


def _own_forward(module, cls) -> bool:
    """Whether calling ``module`` does what ``cls`` does and nothing else: no subclass, no hooks on it or on all modules."""
    m = torch.nn.modules.module
    return (type(module) is cls and "forward" not in module.__dict__
            and not (module._forward_hooks or module._forward_pre_hooks or module._backward_hooks or module._backward_pre_hooks)
            and not (m._global_forward_hooks or m._global_forward_pre_hooks or m._global_backward_hooks or m._global_backward_pre_hooks))


def _fits(x, ln):
    """Whether the kernel covers ln(x): otherwise the framework's operations run (and raise, where they do)."""
    if not _own_forward(ln, nn.LayerNorm) or not x.is_cuda or x.dtype != torch.bfloat16 or x.numel() == 0:
        return False
    D = x.shape[-1]
    return (D % 8 == 0 and D <= MAX_CHANNELS and tuple(ln.normalized_shape) == (D,)
            and all(p is not None and p.dtype == torch.bfloat16 and p.device == x.device and p.is_contiguous() and p.data_ptr() % 16 == 0
                    for p in (ln.weight, ln.bias))
            and not torch.compiler.is_compiling() and not torch.is_autocast_enabled("cuda"))


def _dense16(t):
    """t dense and at a 16-byte boundary (a copy where it is not)."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def residual_layer_norm(x, o, ln: nn.LayerNorm):
    """(s, ln(s)) with s = x + o (o None: s = x), differentiable.  bf16 tensors and parameters go through the kernel above,
    everything else through the framework's operations."""
    ts = (x,) if o is None else (x, o)
    if not all(_fits(t, ln) and t.data_ptr() % 16 == 0 for t in ts) or (o is not None and (o.shape != x.shape or o.device != x.device)):
        s = x if o is None else x + o
        return s, ln(s)
    if torch.is_grad_enabled() and any(t.requires_grad for t in (*ts, ln.weight, ln.bias)):
        return _ResidualLayerNorm.apply(x, o, ln.weight, ln.bias, float(ln.eps))
    s, y, _ = _raw(x.contiguous(), None if o is None else o.contiguous(), ln.weight, ln.bias, float(ln.eps), False)
    return s, y


def layer_norm(x, ln: nn.LayerNorm):
    """ln(x), differentiable; see ``residual_layer_norm``."""
    return residual_layer_norm(x, None, ln)[1]
