"""The native call path of the torch operator (csrc/wkv6_torch.cpp) against the registered custom ops on the same inputs:
both end in the same kernels, so results are equal bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(B, T, H, N, dtype, seed, strided=False):
    g = torch.Generator(device="cuda").manual_seed(seed)
    wide = 2 * H * N if strided else H * N
    mk = lambda s: (torch.randn(B, T, wide, generator=g, device="cuda") * s).to(dtype)[..., :H * N]
    x = [mk(N ** -0.5) for _ in range(3)] + [(torch.rand(B, T, wide, generator=g, device="cuda") * 7 - 6).to(dtype)[..., :H * N]]
    return x, torch.randn(H, N, generator=g, device="cuda") * 0.1, torch.randn(B, T, H * N, generator=g, device="cuda")


@pytest.mark.parametrize("B,T,H,N,dtype,strided", [
    (1, 1, 1, 64, torch.bfloat16, False), (3, 65, 2, 64, torch.bfloat16, False), (2, 33, 3, 64, torch.float16, False),
    (2, 40, 2, 32, torch.float32, False), (2, 130, 2, 64, torch.bfloat16, True)])
def test_training_call_equals_the_custom_ops(B, T, H, N, dtype, strided):
    from star_rwkv6_b200 import ops
    x, u, gy = _inputs(B, T, H, N, dtype, 5, strided)
    gy = gy.to(ops.out_dtype(dtype))
    leaves = [t.detach().requires_grad_(True) for t in (*x, u)]
    y = ops._native.wkv6(*leaves, N, 0)
    assert y is not None
    got = (y, *torch.autograd.grad(y, leaves, gy))
    leaves = [t.detach().requires_grad_(True) for t in (*x, u)]
    y, _ = torch.ops.wkv6_b200.forward(*leaves, N, True, 0)
    want = (y, *torch.autograd.grad(y, leaves, gy))
    for name, a, b in zip(("y", "gr", "gk", "gv", "gw"), got, want):
        assert a.dtype == b.dtype and torch.equal(a, b), name
    # gu: B rows of the same fp32 values added up in row order here, in the framework's order there
    assert (got[5] - want[5]).abs().max() <= B * 2 ** -24 * want[5].abs().max() + 1e-12


def test_calls_it_leaves_to_python():
    from star_rwkv6_b200 import ops
    x, u, _ = _inputs(1, 8, 1, 64, torch.bfloat16, 6)
    assert ops._native.wkv6(*(t.cpu() for t in x), u.cpu(), 64, 0) is None
    assert ops._native.wkv6(*x[:3], x[3][:, :7], u, 64, 0) is None                  # shapes differ
    assert ops._native.with_state(*x, u, torch.zeros(2, 1, 64, 64, device="cuda"), 64, 0) is None   # more states than rows
    assert ops._native.with_state(*x, u, torch.zeros(1, 1, 64, 64), 64, 0) is None  # state on the host
    with pytest.raises(ops._lib.WKV6Error):                                         # head size without a kernel
        ops.wkv6(*x, u, 4)


def test_second_derivative_is_refused():
    from star_rwkv6_b200 import ops
    x, u, gy = _inputs(1, 8, 1, 64, torch.float32, 7)
    leaves = [t.requires_grad_(True) for t in (*x, u)]
    (gr,) = torch.autograd.grad(ops.wkv6(*leaves, 64), leaves[:1], gy, create_graph=True)
    with pytest.raises(RuntimeError, match="not differentiable"):
        gr.sum().backward()
