"""Chunked variant cut along T (wkv6_split_segments > 1) against the oracle and the uncut calls: equal segments (up to one
sequence per SM) and two unequal ones (up to two per SM), ragged last chunks, segments of one chunk, chunks beyond the
single-reference limit on either side of a cut, carried states and row strides that are not dense."""
import ctypes

import numpy as np
import pytest
import torch

from helpers import TOL_BF16, np_, oracle_all, rounded, scaled_err
from oracle import wkv6_oracle as O

pytestmark = pytest.mark.gpu
N = 64


def _segments(r, u):
    from star_rwkv6_b200 import _lib as L, ops
    return L.lib.wkv6_split_segments(ctypes.byref(ops.make_problem(r, u, N, r.dtype, L.VARIANT_CHUNK)))


@pytest.mark.parametrize("B,T,H", [(1, 256, 1), (2, 193, 3), (1, 1003, 12), (3, 1040, 2), (1, 2048, 148), (1, 1100, 149), (2, 2070, 128)])
def test_split_training_call(B, T, H):
    from star_rwkv6_b200 import _lib as L, ops
    d = O.make_inputs(B, T, H, N, seed=T)
    d["w"][:, T // 2: T // 2 + 40, ::2] = 2.0      # beyond the single-reference limit: the general kernel redoes these segments
    d["w"][:, T // 3] = -1e9
    t = {n: torch.tensor(d[n]).bfloat16().cuda().requires_grad_(True) for n in "rkvw"}
    u = torch.tensor(d["u"]).cuda().requires_grad_(True)
    assert _segments(t["r"], u) > 1
    y = ops._native.wkv6(t["r"], t["k"], t["v"], t["w"], u, N, L.VARIANT_CHUNK)
    g = torch.autograd.grad(y, (*t.values(), u), torch.tensor(d["gy"]).bfloat16().cuda())
    ref = oracle_all(rounded(d, torch.bfloat16), N)
    for n, a in zip(("y", "gr", "gk", "gv", "gw", "gu"), (y, *g)):
        assert np.isfinite(np_(a)).all(), n
        assert scaled_err(np_(a), ref[n]) <= TOL_BF16, n


@pytest.mark.parametrize("B,T,H", [(2, 333, 3), (1, 1003, 149)])
@pytest.mark.parametrize("kinds,state_dtype", [(0, torch.float32), (1, torch.float32), (2, torch.bfloat16)])
def test_split_states(B, T, H, kinds, state_dtype):
    from star_rwkv6_b200 import _lib as L, ops
    kinds = min(kinds, B)
    d = O.make_inputs(B, T, H, N, seed=21)
    s0 = None if kinds == 0 else torch.randn(kinds, H, N, N, generator=torch.Generator().manual_seed(3)).to(state_dtype).cuda()
    u = torch.tensor(d["u"]).cuda()
    wide = torch.stack([torch.tensor(d[n]).bfloat16() for n in "rkvw"], 2).cuda()     # rows of 4 C elements
    t = list(wide.unbind(2))
    assert _segments(t[0], u) > 1 and not t[0].is_contiguous()
    y, s = ops._native.with_state(*t, u, s0, N, L.VARIANT_CHUNK)
    y1, s1, _ = ops.forward_raw(*t, u, N, s_in=s0, want_state=True, variant=L.VARIANT_CHUNK)   # one piece
    # the entering states differ by the roundings of one bf16 operand per chunk: 2^-8 of the result at most
    assert s.dtype == s1.dtype and scaled_err(np_(y), np_(y1)) <= 2 ** -7
    assert scaled_err(np_(s), np_(s1)) <= 2 ** -7
