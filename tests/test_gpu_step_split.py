"""Sequential variant at head size 64 cut along T (wkv6_split_segments > 1) against the oracle, forward with states and
all gradients, at the smallest split length, lengths that leave a ragged last segment or tile, and strong decays."""
import ctypes

import numpy as np
import pytest
import torch

from helpers import TOL_BF16, TOL_F32, np_, oracle_all, rounded, scaled_err
from oracle import wkv6_oracle as O

pytestmark = pytest.mark.gpu
N = 64


@pytest.mark.parametrize("B,T,H,dtype,tol", [
    (1, 96, 1, torch.float32, TOL_F32), (2, 129, 2, torch.float32, TOL_F32), (3, 1003, 2, torch.float32, TOL_F32),
    (1, 2000, 5, torch.float32, TOL_F32), (2, 300, 3, torch.float16, 2e-3), (2, 300, 3, torch.bfloat16, TOL_BF16)])
def test_split_training_call(B, T, H, dtype, tol):
    from star_rwkv6_b200 import _lib as L, ops
    d = O.make_inputs(B, T, H, N, seed=T)
    d["w"][:, T // 2] = 3.0          # a step that forgets everything, and a masked one
    d["w"][:, T // 3] = -1e9
    t = {n: torch.tensor(d[n]).to(dtype).cuda().requires_grad_(True) for n in "rkvw"}
    u = torch.tensor(d["u"]).cuda().requires_grad_(True)
    p = ops.make_problem(t["r"], u, N, ops.out_dtype(dtype), L.VARIANT_SEQ)
    G = L.lib.wkv6_split_segments(ctypes.byref(p))
    assert G > 1
    y = ops._native.wkv6(t["r"], t["k"], t["v"], t["w"], u, N, L.VARIANT_SEQ)
    g = torch.autograd.grad(y, (*t.values(), u), torch.tensor(d["gy"]).to(y.dtype).cuda())
    dr = rounded(d, dtype, names=("r", "k", "v", "w") + (("gy",) if dtype == torch.bfloat16 else ()))
    ref = oracle_all(dr, N)
    for n, a in zip(("y", "gr", "gk", "gv", "gw", "gu"), (y, *g)):
        assert np.isfinite(np_(a)).all(), n
        assert scaled_err(np_(a), ref[n]) <= tol, n


@pytest.mark.parametrize("kinds,state_dtype", [(0, torch.float32), (1, torch.float32), (2, torch.float32), (2, torch.bfloat16)])
def test_split_states(kinds, state_dtype):
    from star_rwkv6_b200 import _lib as L, ops
    B, T, H = 2, 203, 2
    d = O.make_inputs(B, T, H, N, seed=21)
    s0 = None if kinds == 0 else torch.randn(kinds, H, N, N, generator=torch.Generator().manual_seed(3)).to(state_dtype).cuda()
    t = [torch.tensor(d[n]).cuda() for n in ("r", "k", "v", "w", "u")]
    y, s = ops._native.with_state(*t, s0, N, L.VARIANT_SEQ)
    y1, s1, _ = ops.forward_raw(*t, N, s_in=s0, want_state=True, variant=L.VARIANT_SEQ)   # one piece
    assert s.dtype == s1.dtype and scaled_err(np_(y), np_(y1)) <= 1e-5
    assert scaled_err(np_(s), np_(s1)) <= (1e-5 if state_dtype == torch.float32 else 2 ** -8)
