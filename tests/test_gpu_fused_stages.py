"""Fused stages of the model's blocks against float64 evaluations of the same expressions: the pair of vector mixes, the five
data-dependent mixes with their low-rank products, and the layer norm with the residual addition, forward and backward, at
sizes around their tiles (channel groups of 32 / 128 / 256, tiles of 16 rows, runs of 4 rows and 8 tokens, batch boundaries)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
# results are rounded to bf16 once (2^-9 of the largest element); sums over rows of rounded terms stay below twice that
TOL = 2 ** -8


def _err(got, ref):
    ref = ref.detach().double()
    return float((got.detach().double() - ref).abs().max() / ref.abs().max().clamp_min(1e-30))


def _randn(g, *shape, scale=1.0):
    return (torch.randn(*shape, generator=g, device="cuda") * scale).bfloat16()


def _shift(x):
    return torch.cat([torch.zeros_like(x[:, :1]), x[:, :-1]], 1) - x


@pytest.mark.parametrize("B,T,C", [(1, 1, 8), (2, 31, 264), (3, 33, 64), (1, 65, 2048)])
def test_pair_of_vector_mixes(B, T, C):
    from star_rwkv6_b200.time_mix_inputs import shift_mix_pair
    g = torch.Generator(device="cuda").manual_seed(T)
    x, go = _randn(g, B, T, C), [_randn(g, B, T, C) for _ in range(2)]
    mu = [torch.rand(C, generator=g, device="cuda") for _ in range(2)]
    args = [t.clone().requires_grad_(True) for t in (x, *mu)]
    out = shift_mix_pair(*args)
    got = torch.autograd.grad(out, args, go)
    args64 = [t.double().requires_grad_(True) for t in (x, *mu)]
    out64 = [args64[0] + _shift(args64[0]) * m for m in args64[1:]]
    ref = torch.autograd.grad(out64, args64, [t.double() for t in go])
    for a, b in zip((*out, *got), (*out64, *ref)):
        assert _err(a, b) <= TOL


@pytest.mark.parametrize("B,T,C,stacked", [(1, 1, 8, False), (2, 17, 136, True), (3, 33, 264, False), (2, 1000, 96, False), (1, 130, 2048, True)])
def test_low_rank_mixes(B, T, C, stacked):
    from star_rwkv6_b200.time_mix_inputs import _LoraMix, _lora_fits
    g = torch.Generator(device="cuda").manual_seed(T)
    x, go = _randn(g, B, T, C), _randn(g, 5, B, T, C)
    h, wb, bias = torch.tanh(_randn(g, B * T, 160)), _randn(g, 5, 32, C, scale=32 ** -0.5), _randn(g, 5, 1, C, scale=0.3)
    assert _lora_fits(x, h, wb, bias)
    args = [t.clone().requires_grad_(True) for t in (x, h, wb, bias)]
    out = _LoraMix.apply(*args, stacked)
    got = torch.autograd.grad(out, args, go if stacked else list(go))
    a64 = [t.double().requires_grad_(True) for t in (x, h, wb, bias)]
    l = a64[3] + torch.bmm(a64[1].view(B * T, 5, 32).transpose(0, 1), a64[2])
    out64 = a64[0] + _shift(a64[0]) * l.view(5, B, T, C)
    ref = torch.autograd.grad(out64, a64, go.double())
    for a, b in zip((out if stacked else torch.stack(out), *got), (out64, *ref)):
        assert _err(a, b) <= 2 * TOL          # gl is rounded to bf16 before the products that make gh, gwb and gbias


@pytest.mark.parametrize("rows,D", [(1, 8), (5, 768), (33, 1032), (9, 2056), (700, 2048), (6, 4104), (3, 8192)])
@pytest.mark.parametrize("add,use_sum", [(False, False), (True, True), (True, False), (False, True)])
def test_layer_norm(rows, D, add, use_sum):
    from star_rwkv6_b200.layer_norm import _fits, residual_layer_norm
    g = torch.Generator(device="cuda").manual_seed(D)
    ln = torch.nn.LayerNorm(D, eps=1e-5).cuda().bfloat16()
    with torch.no_grad():
        ln.weight.copy_(_randn(g, D) + 1); ln.bias.copy_(_randn(g, D))
    x = (_randn(g, rows, D) + 3).requires_grad_(True)       # a mean well away from zero
    o = _randn(g, rows, D).requires_grad_(True) if add else None
    assert _fits(x, ln)
    gy, gs = _randn(g, rows, D), _randn(g, rows, D)
    s, y = residual_layer_norm(x, o, ln)
    ins = [x] + ([o] if add else []) + [ln.weight, ln.bias]
    got = torch.autograd.grad([y] + ([s] if use_sum else []), ins, [gy] + ([gs] if use_sum else []))
    i64 = [t.detach().double().requires_grad_(True) for t in ins]
    total = i64[0] + i64[1] if add else i64[0]
    if add:
        total = total + (s.detach().double() - total.detach())       # the sum as it is stored, rounded
    y64 = torch.nn.functional.layer_norm(total, (D,), i64[-2], i64[-1], 1e-5)
    ref = torch.autograd.grad([y64] + ([total] if use_sum else []), i64, [gy.double()] + ([gs.double()] if use_sum else []))
    assert _err(y, y64) <= TOL and _err(s, total) <= TOL
    for a, b in zip(got, ref):
        assert _err(a, b) <= TOL
    with torch.no_grad():
        s1, y1 = residual_layer_norm(x, o, ln)
    assert torch.equal(y1, y) and torch.equal(s1, s)
