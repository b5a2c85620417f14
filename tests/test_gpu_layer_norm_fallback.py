"""Norms that the fused layer norm does not cover take the framework's operations, and gradients that do not lie at a 16-byte
boundary are copied: results as of the framework's composition."""
import pytest
import torch
from torch import nn

pytestmark = pytest.mark.gpu
D = 256


def _x(seed=0, rows=5):
    return torch.randn(rows, D, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda").bfloat16()


class _Doubled(nn.LayerNorm):
    def forward(self, x):
        return 2 * super().forward(x)


def _offset_parameters():
    ln = nn.LayerNorm(D).cuda().bfloat16()
    flat = torch.randn(2 * D + 3, device="cuda").bfloat16()
    ln.weight.data, ln.bias.data = flat[1:1 + D], flat[D + 2:2 * D + 2]     # slices of a flat buffer, 2 and 4 bytes off a boundary
    return ln


@pytest.mark.parametrize("make", [lambda: nn.RMSNorm(D).cuda().bfloat16(), lambda: _Doubled(D).cuda().bfloat16(), _offset_parameters,
                                  lambda: nn.LayerNorm(D, bias=False).cuda().bfloat16(), lambda: nn.LayerNorm(D, elementwise_affine=False)])
def test_other_norms(make):
    from star_rwkv6_b200.layer_norm import residual_layer_norm
    ln, x, o = make(), _x(), _x(1)
    with torch.no_grad():
        s, y = residual_layer_norm(x, o, ln)
        assert torch.equal(s, x + o) and torch.equal(y, ln(x + o))
        assert torch.equal(residual_layer_norm(x, None, ln)[1], ln(x))


def test_hooks_fire():
    from star_rwkv6_b200.layer_norm import layer_norm
    ln, x, seen = nn.LayerNorm(D).cuda().bfloat16(), _x(), []
    for register in (ln.register_forward_hook, nn.modules.module.register_module_forward_hook):
        handle = register(lambda m, a, out: seen.append(m is ln))
        with torch.no_grad():
            layer_norm(x, ln)
        handle.remove()
    assert seen == [True, True]


def test_parameters_elsewhere_are_refused():
    from star_rwkv6_b200.layer_norm import _fits, layer_norm
    ln = nn.LayerNorm(D).bfloat16()
    assert not _fits(_x(), ln)
    with pytest.raises(RuntimeError):
        layer_norm(_x(), ln)


def test_gradient_at_an_odd_offset():
    from star_rwkv6_b200.layer_norm import residual_layer_norm
    ln, x = nn.LayerNorm(D).cuda().bfloat16(), _x().requires_grad_(True)
    gy = torch.randn(5 * D + 1, device="cuda").bfloat16()[1:].view(5, D)
    got = torch.autograd.grad(residual_layer_norm(x, None, ln), (x, ln.weight, ln.bias), (gy, gy))
    want = torch.autograd.grad(residual_layer_norm(x, None, ln), (x, ln.weight, ln.bias), (gy.clone(), gy.clone()))
    for a, b in zip(got, want):
        assert torch.equal(a, b)
