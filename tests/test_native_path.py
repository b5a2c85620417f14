"""The native call path of the torch operator (csrc/wkv6_torch.cpp) against the registered custom ops on the same inputs: where
sequences are walked in one piece both end in the same kernels, so results are equal bit for bit.  Where the library cuts them (the
custom ops never do) results agree to rounding."""
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


def _gradients(call, x, u, gy):
    leaves = [t.detach().requires_grad_(True) for t in (*x, u)]
    y = call(*leaves)
    return (y.detach(), *torch.autograd.grad(y, leaves, gy))


@pytest.mark.parametrize("B,T,H,dtype,tol", [(1, 1003, 12, torch.bfloat16, 2e-2), (2, 300, 3, torch.float32, 2e-5)])
def test_cut_and_whole_sequences(B, T, H, dtype, tol):
    """A shape that the library cuts: in one piece on request, with the custom ops' bits; cut, with theirs to rounding (bf16: states
    at the segments' ends from bf16 products; fp32: another order of a few hundred sums)."""
    from star_rwkv6_b200 import _lib, ops
    from star_rwkv6_b200.rwkv_kernel.torch_rwkv_kernel import RWKVKernelOperator
    x, u, gy = _inputs(B, T, H, 64, dtype, 8)
    gy = gy.to(dtype)
    assert _lib.lib.wkv6_split_segments(ops.make_problem(x[0], u, 64, dtype, 0)) > 1
    want = _gradients(lambda *a: torch.ops.wkv6_b200.forward(*a, 64, True, 0)[0], x, u, gy)
    whole = _gradients(lambda *a: RWKVKernelOperator(64, T, segments="whole")(*a)[0], x, u, gy)
    cut = _gradients(lambda *a: RWKVKernelOperator(64, T)(*a)[0], x, u, gy)
    for name, a, b, c in zip(("y", "gr", "gk", "gv", "gw"), whole, cut, want):
        assert torch.equal(a, c), name
        assert float((b.double() - c.double()).norm() / c.double().norm()) <= tol, name
    assert float((whole[5] - want[5]).abs().max()) <= B * 2 ** -24 * float(want[5].abs().max()) + 1e-12
    s0 = torch.randn(B, H, 64, 64, device="cuda") * 0.1
    y0, st0, _ = ops.forward_raw(*x, u, 64, s_in=s0, want_state=True)
    y1, st1 = RWKVKernelOperator(64, T, segments="whole")(*x, u, return_state=True, init_state=s0)
    assert torch.equal(y0, y1) and torch.equal(st0, st1)


@pytest.mark.parametrize("B,T,H,dtype", [(2, 70, 2, torch.bfloat16), (1, 300, 2, torch.bfloat16), (2, 33, 2, torch.float32), (1, 130, 2, torch.float32),
                                         (1, 40, 1, torch.float16)])
def test_incoming_gradients_that_are_not_plain(B, T, H, dtype):
    """Batched gradients and a lazily negated one give what plain ones give (to rounding: the custom op is never cut)."""
    from star_rwkv6_b200 import ops
    x, u, _ = _inputs(B, T, H, 64, dtype, 9)
    leaves = [t.requires_grad_(True) for t in (*x, u)]
    gys = torch.randn(3, B, T, H * 64, device="cuda").to(ops.out_dtype(dtype))
    y = ops.wkv6(*leaves, 64)
    want = [torch.autograd.grad(y, leaves, g, retain_graph=True) for g in gys]
    got = torch.autograd.grad(y, leaves, gys, is_grads_batched=True, retain_graph=True)
    neg = torch.autograd.grad(y, leaves, torch._neg_view(-gys[0]), retain_graph=True)
    tol = 2e-2 if dtype == torch.bfloat16 else 2e-3 if dtype == torch.float16 else 2e-5
    for i, name in enumerate(("gr", "gk", "gv", "gw", "gu")):
        for a, b in [(got[i][j], want[j][i]) for j in range(3)] + [(neg[i], want[0][i])]:
            assert a.shape == b.shape and a.dtype == b.dtype
            assert float((a.double() - b.double()).norm()) <= tol * float(b.double().norm()), name


def test_cut_call_captured_on_a_side_stream():
    """A shape that the library cuts, forward and backward in a CUDA graph: replays on new inputs have the bits of eager calls."""
    from star_rwkv6_b200 import ops
    x, u, gy = _inputs(1, 1003, 2, 64, torch.bfloat16, 10)
    gy = gy.to(torch.bfloat16)
    leaves = [t.requires_grad_(True) for t in (*x, u)]
    call = lambda: _gradients(lambda *a: ops.wkv6(*a, 64), leaves[:4], leaves[4], gy)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        eager = call()                  # also the call outside the capture
    torch.cuda.current_stream().wait_stream(side)
    assert all(torch.equal(a, b) for a, b in zip(eager, call()))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call()
    for seed in (11, 12):
        fresh, v, _ = _inputs(1, 1003, 2, 64, torch.bfloat16, seed)
        with torch.no_grad():
            for a, b in zip(leaves, (*fresh, v)):
                a.copy_(b)
        graph.replay()
        assert all(torch.equal(a, b) for a, b in zip(out, call()))
