"""Inputs whose rows share memory (broadcast over the batch or over the tokens, windows of one buffer): the kernels use one stride set
for inputs and outputs and take a stride of 0 for "dense", so such inputs are copied first."""
import pytest
import torch


def _views(C):
    base = torch.arange(40 * C, dtype=torch.float32) / (40 * C)
    return {
        "dense": base[:30 * C].view(3, 10, C),
        "transposed": base[:30 * C].view(10, 3, C).transpose(0, 1),
        "slice": base[:40 * C].view(4, 10, C)[1:, 2:7],
        "wide": base[:40 * C].view(2, 10, 2 * C)[..., :C],
        "batch broadcast": base[:10 * C].view(1, 10, C).expand(3, 10, C),
        "token broadcast": base[:3 * C].view(3, 1, C).expand(3, 10, C),
        "windows": base.as_strided((3, 10, C), (2 * C, C, 1)),
        "one row": base[:C].view(1, 1, C).expand(1, 1, C),
        "one token, batch broadcast": base[:C].view(1, 1, C).expand(5, 1, C),
    }


OVERLAPPING = ("batch broadcast", "token broadcast", "windows", "one token, batch broadcast")


@pytest.mark.parametrize("name", list(_views(8)))
def test_which_layouts_overlap(name):
    from star_rwkv6_b200 import ops
    t = _views(64)[name]
    assert ops._rows_apart(t) == (name not in OVERLAPPING)
    (c,) = ops._apart(t)
    assert (c is t) == (name not in OVERLAPPING) and ops._rows_apart(c) and torch.equal(c, t)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("name", list(_views(8)))
def test_calls_equal_those_of_dense_copies(name, dtype):
    from star_rwkv6_b200 import ops
    from star_rwkv6_b200.rwkv_kernel.torch_rwkv_kernel import RWKVKernelOperator
    base = _views(128)[name]
    B, T, C = base.shape
    lay = (base.shape, base.stride())
    span = sum((n - 1) * s for n, s in zip(*lay)) + 1
    g = torch.Generator(device="cuda").manual_seed(3)
    x = [torch.randn(span, generator=g, device="cuda").mul(0.2).to(dtype).as_strided(*lay).requires_grad_(True) for _ in range(4)]
    u = (torch.randn(2, 64, generator=g, device="cuda") * 0.1).requires_grad_(True)
    gy, s0 = torch.randn(B, T, C, generator=g, device="cuda").to(dtype), torch.randn(B, 2, 64, 64, generator=g, device="cuda")
    op = RWKVKernelOperator(64, T)
    dense = [t.detach().clone(memory_format=torch.contiguous_format).requires_grad_(True) for t in x]
    outs = []
    for ts in (x, dense):
        y, _ = op(*ts, u)
        outs.append((y, *torch.autograd.grad(y, (*ts, u), gy), *op(*[t.detach() for t in ts], u.detach(), return_state=True, init_state=s0),
                     *ops.forward_raw(*[t.detach() for t in ts], u.detach(), 64, want_state=True)[:2]))
    for i, (a, b) in enumerate(zip(*outs)):
        if i == 5:      # gu: B rows of the same fp32 values, summed in row order by the native path, in the framework's by the other
            assert float((a - b).abs().max()) <= B * 2 ** -24 * float(b.abs().max())
        elif T == 1 and i in (6, 7):      # dense: the decode kernel; not dense: the chunked or stepping one (bf16 operands, another order)
            tol = 64 * 2 ** -24 if dtype == torch.float32 else 2 ** -8
            assert float((a - b).abs().max()) <= tol * float(b.abs().max())
        else:
            assert torch.equal(a, b)
    if T == 1:
        k = dense[1].detach()[:1].expand(B, 1, C)
        a, b = (op(dense[0].detach(), t, k, k, u.detach(), return_state=True, init_state=s0) for t in (k, k.contiguous()))
        assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
