"""States and bonus that are views at odd offsets of larger buffers (a packed pool): results have the bits of aligned copies.  The
wide accesses are taken at aligned addresses only; every case here runs the element-wise ones."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _at(t, offset):
    """A copy of t that starts ``offset`` elements into its allocation."""
    buf = torch.empty(t.numel() + offset, dtype=t.dtype, device=t.device)
    return buf[offset:].view(t.shape).copy_(t)


@pytest.mark.parametrize("offset", [1, 2, 3])
@pytest.mark.parametrize("dtype,B,T,H", [(torch.float32, 2, 2, 3), (torch.float32, 1, 300, 2), (torch.float16, 2, 70, 2),
                                         (torch.bfloat16, 1, 70, 2), (torch.bfloat16, 1, 300, 2)])
def test_state_and_bonus_at_odd_offsets(dtype, B, T, H, offset):
    from star_rwkv6_b200 import ops
    from star_rwkv6_b200._lib import check, lib
    from star_rwkv6_b200.rwkv_kernel.torch_rwkv_kernel import RWKVKernelOperator
    g = torch.Generator(device="cuda").manual_seed(T)
    r, k, v, w = (torch.randn(B, T, H * 64, generator=g, device="cuda").mul(0.1).to(dtype) for _ in range(4))
    u, s0 = torch.randn(H, 64, generator=g, device="cuda") * 0.1, torch.randn(B, H, 64, 64, generator=g, device="cuda")
    for segments in (1, "whole"):
        op = RWKVKernelOperator(64, T, segments=segments)
        y, s = op(r, k, v, w, u, return_state=True, init_state=s0)
        y1, s1 = op(r, k, v, w, _at(u, offset), return_state=True, init_state=_at(s0, offset))
        assert torch.equal(y, y1) and torch.equal(s, s1)
    y, s, _ = ops.forward_raw(r, k, v, w, u, 64, s_in=s0, want_state=True)
    p = ops.make_problem(r, u, 64, ops.out_dtype(dtype), 0)
    state, y1 = _at(s0, offset), torch.empty_like(y)      # final state over the initial one
    check(lib.wkv6_forward(ctypes.byref(p), *(ops._ptr(t) for t in (r, k, v, w, u, y1, state)), None, B, ops._ptr(state), None,
                           ops._stream(r.device)))
    assert torch.equal(y, y1) and torch.equal(s, state)


@pytest.mark.parametrize("reverse", [0, 1])
def test_state_scan_at_odd_offsets(reverse):
    from star_rwkv6_b200 import ops
    from star_rwkv6_b200._lib import check, lib
    B, H, G = 2, 3, 11
    g = torch.Generator(device="cuda").manual_seed(G)
    dec, b = -torch.rand(B * G, H, 64, generator=g, device="cuda"), torch.randn(B * G, H, 64, 64, generator=g, device="cuda")
    out = []
    for offset in (0, 1, 2):
        bs, o = _at(b, offset), _at(torch.zeros_like(b), offset)
        check(lib.wkv6_state_scan(B, H, 64, G, ops._ptr(dec), ops._ptr(bs), None, ops._ptr(o), None, reverse, ops._stream(b.device)))
        out.append(o)
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])
