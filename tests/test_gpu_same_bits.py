"""Fused stages that leave the bits of the general path: a training step's gradients follow single rounding steps of bf16 (behind a
token whose WKV output is nearly zero the per-head norm magnifies them), so a stage with another order of the same sums moves
them by percents.  Sizes around the kernels' tiles, runs and batch boundaries."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _randn(g, *shape, scale=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(dtype)


def _leaves(ts):
    return [t.clone().requires_grad_(True) for t in ts]


@pytest.mark.parametrize("stacked", [False, True])
@pytest.mark.parametrize("B,T,C", [(1, 1, 8), (2, 17, 136), (3, 33, 264), (2, 1000, 96), (3, 1003, 768), (1, 130, 2048)])
def test_low_rank_mixes(B, T, C, stacked):
    from star_rwkv6_b200.time_mix_inputs import _LoraMix, shift_mix_tensors
    g = torch.Generator(device="cuda").manual_seed(T + C)
    ins = [_randn(g, B, T, C), torch.tanh(_randn(g, B * T, 160)), _randn(g, 5, 32, C, scale=32 ** -0.5), _randn(g, 5, 1, C, scale=0.3)]
    go = _randn(g, 5, B, T, C)
    a, b = _leaves(ins), _leaves(ins)
    out = _LoraMix.apply(*a, stacked)
    got = torch.autograd.grad(out, a, go if stacked else list(go))
    l = torch.baddbmm(b[3], b[1].reshape(B * T, 5, 32).transpose(0, 1), b[2])
    want = shift_mix_tensors(b[0], l.reshape(5, B, T, C))
    ref = torch.autograd.grad(want, b, go)
    for x, y in zip((out if stacked else torch.stack(out), *got), (want, *ref)):
        assert torch.equal(x, y)
