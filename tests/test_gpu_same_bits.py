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


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("B,T,C", [(1, 1, 8), (2, 31, 264), (3, 33, 64), (2, 1003, 768), (1, 65, 2048)])
def test_pair_of_vector_mixes(B, T, C, dtype):
    from star_rwkv6_b200.time_mix_inputs import shift_mix_pair, shift_mix_vector     # as ChannelMix calls it
    g = torch.Generator(device="cuda").manual_seed(T + C)
    x, go = _randn(g, B, T, C, dtype=dtype), [_randn(g, B, T, C, dtype=dtype) for _ in range(2)]
    mu = [torch.rand(C, generator=g, device="cuda") for _ in range(2)]
    a, b = _leaves([x, *mu]), _leaves([x, *mu])
    out = shift_mix_pair(*a, separate_gx=True)
    got = torch.autograd.grad(out, a, go)
    want = [shift_mix_vector(b[0], m) for m in b[1:]]
    ref = torch.autograd.grad(want, b, go)
    for p, q in zip((*out, *got), (*want, *ref)):
        assert torch.equal(p, q)


def test_channel_mix_gradients():
    """The channel-mix block against the same block with the two mixes as separate calls."""
    from star_rwkv6_b200 import model
    from star_rwkv6_b200.time_mix_inputs import shift_mix_vector
    torch.manual_seed(0)
    cm = model.ChannelMix(768, 1024).cuda()
    for n, p in cm.named_parameters():
        if p.dim() == 2:
            p.data = p.data.bfloat16()
    g = torch.Generator(device="cuda").manual_seed(1)
    x, go = _randn(g, 2, 203, 768), _randn(g, 2, 203, 768)
    a, b = _leaves([x]), _leaves([x])
    got = torch.autograd.grad(cm(a[0]), a + list(cm.parameters()), go)
    pair, model.shift_mix_pair = model.shift_mix_pair, lambda x, m0, m1, **kw: (shift_mix_vector(x, m0), shift_mix_vector(x, m1))
    try:
        want = torch.autograd.grad(cm(b[0]), b + list(cm.parameters()), go)
    finally:
        model.shift_mix_pair = pair
    for p, q in zip(got, want):
        assert torch.equal(p, q)


@pytest.mark.parametrize("V", [8, 4104, 65536])
def test_loss_of_logits_at_the_end_of_the_range(V):
    """exp(z - max) is formed from the difference: no term overflows where the scaled logit would (|z| > 2.36e38), and the
    probabilities of a row that is one value throughout are equal and sum to one."""
    from star_rwkv6_b200.loss import lm_loss
    logits = torch.zeros(3, V, device="cuda", dtype=torch.bfloat16)
    logits[0, 3], logits[0, 5] = 3.2e38, -3.2e38
    logits[1] = 3.2e38
    logits[2] = -2.5e38
    targets = torch.tensor([3, 1, 2], device="cuda")
    z = logits.clone().requires_grad_(True)
    lm_loss(z * 1, targets).backward()
    p = torch.softmax(logits.double(), 1)
    p[torch.arange(3), targets] -= 1
    assert float((z.grad.double() - p / 3).abs().max()) <= 2 ** -8 / 3


def test_time_mix_walks_sequences_in_one_piece():
    """A shape whose sequences the operator would cut: the block's gradients have the bits of the uncut call."""
    from star_rwkv6_b200 import model
    torch.manual_seed(0)
    tm = model.TimeMix(128).cuda()
    for n, p in tm.named_parameters():
        if not n.endswith(("time_faaaa", "scale", "offset", "time_mix_x")):
            p.data = p.data.bfloat16()
    g = torch.Generator(device="cuda").manual_seed(1)
    x, go = _randn(g, 1, 300, 128), _randn(g, 1, 300, 128)
    a, b = _leaves([x]), _leaves([x])
    got = torch.autograd.grad(tm(a[0]), a + list(tm.parameters()), go)
    wkv6, model.wkv6 = model.wkv6, lambda *t, **kw: torch.ops.wkv6_b200.forward(*t, True, 0)[0]
    try:
        want = torch.autograd.grad(tm(b[0]), b + list(tm.parameters()), go)
    finally:
        model.wkv6 = wkv6
    for p, q in zip(got, want):
        assert torch.equal(p, q)


def test_model_step():
    """Loss and gradients of the whole model against the same modules composed of the general operations: framework norms and
    additions, uncut recurrence, batched low-rank product, one vector mix at a time."""
    from star_rwkv6_b200 import model, time_mix_inputs as tmi
    from star_rwkv6_b200.loss import lm_loss
    torch.manual_seed(0)
    with torch.device("cuda"):
        m = model.RWKV6(2, 512, 256, decomposer_size=32, expand_size=512, decay_rank=32).to_bf16_()
        with torch.no_grad():
            for blk in m.blocks:
                blk.time_mix.mix_inputs.bias_b.normal_(0.0, 0.3)
    tok = torch.randint(0, 512, (1, 334), device="cuda")
    params = dict(m.named_parameters())

    def step(logits):
        loss = lm_loss(logits, tok[:, 1:])
        return (loss, *torch.autograd.grad(loss, list(params.values())))

    def general(tokens):
        x = m.embedding_ln(m.embedding(tokens))
        for blk in m.blocks:
            tm, cm = blk.time_mix, blk.channel_mix
            h = blk.layer_norm_att(x)
            mi, (B, T, D) = tm.mix_inputs, h.shape
            low = torch.tanh(tmi.shift_mix_vector(h, mi.time_mix_x).reshape(B * T, D) @ mi.dense_a).reshape(B * T, 5, -1).transpose(0, 1)
            l = torch.baddbmm(mi.bias_b, low, mi.dense_b)
            xr, xk, xv, xw, xg = tmi.shift_mix_tensors(h, l.reshape(5, B, T, D))
            w = tm.w_b(torch.tanh(tm.w_a(xw)))
            y, _ = torch.ops.wkv6_b200.forward(tm.dense_r(xr), tm.dense_k(xk), tm.dense_v(xv), w, tm.time_faaaa, 64, True, 0)
            x = x + tm.dense_o(tm.group_norm(y, tm.dense_g(xg), gate_is_raw=True))
            h = blk.layer_norm_ffn(x)
            k = model.relu_sq(cm.dense_key(tmi.shift_mix_vector(h, cm.time_mix_k)))
            x = x + model.sigmoid_mul(cm.dense_receptance(tmi.shift_mix_vector(h, cm.time_mix_r)), cm.dense_value(k))
        return m.output_layer(m.output_ln(x))

    got, want = step(m(tok[:, :-1])), step(general(tok[:, :-1]))
    for name, p, q in zip(("loss", *params), got, want):
        assert torch.equal(p, q), name


@pytest.mark.parametrize("how", ["hook", "subclass", "replaced"])
def test_module_of_the_mixed_inputs_is_called(how):
    """Hooks on the module, a forward of a subclass and a module in its place take part in the block's passes."""
    from star_rwkv6_b200 import model
    torch.manual_seed(0)
    tm, seen = model.TimeMix(128).cuda(), []
    x = torch.randn(2, 9, 128, device="cuda")
    with torch.no_grad():
        want, (want_prefill, _) = tm(x), tm.prefill(x)
        mi = tm.mix_inputs
        if how == "hook":
            mi.register_forward_hook(lambda m, args, out: seen.append(out.shape))
        elif how == "subclass":
            mi.__class__ = type("Logged", (type(mi),), {"forward": lambda self, x: (seen.append(x.shape), type(self).__mro__[1].forward(self, x))[1]})
        else:
            tm.mix_inputs = torch.nn.Identity()
            tm.mix_inputs.forward = lambda x: (seen.append(x.shape), mi(x))[1]
        assert torch.equal(tm(x), want) and torch.equal(tm.prefill(x)[0], want_prefill)
    assert len(seen) == 2
