"""Performance cases: the work that users of this package have it do, through its public entry points.

Three kinds of call cover the package's use:

* ``operator``: ``RWKVKernelOperator`` on its own, the drop-in behind an existing RWKV-6 layer - one decode step with a
  carried state, a prompt that returns its state, and a training step's forward and backward;
* ``train``: forward, fused loss and gradients of the whole model (``model.RWKV6``, ``loss.lm_loss``);
* ``serve``: the model's prompt pass (``prefill``) and its token step (``decode``) replayed from a CUDA graph.

Operator inputs have the benchmark's distributions (r, k, v ~ N(0, 1/N), u ~ N(0, 0.1), gy ~ N(0, 1)); the log-log decay w
is U(-6, 1) as in the benchmark ("uniform") or a per-channel spectrum from slow to fast channels with a little noise per
token, as trained models have it ("spectrum").  Models are random-init, with the layer shapes of the package's 1.6B-shape
training step and 7B-shape inference workloads and fewer layers.
"""
import torch

from star_rwkv6_b200.loss import lm_loss
from star_rwkv6_b200.model import RWKV6
from star_rwkv6_b200.rwkv_kernel.torch_rwkv_kernel import RWKVKernelOperator

N = 64                      # head size of every RWKV-6 model
VOCAB = 65536
DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}


def _operator(name, do, B, T, H, dtype="bf16", decay="uniform", segments="1"):
    c = {"kind": "operator", "do": do, "B": B, "T": T, "H": H, "dtype": dtype, "decay": decay, "segments": segments}
    return dict(c, name=name) if name else c


def _model(name, do, B, T, D, layers):
    c = {"kind": "train" if do == "step" else "serve", "do": do, "B": B, "T": T, "D": D, "layers": layers}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one user's chat: a token step of one layer; pure latency
        _operator("decode B1 H32", "decode", 1, 1, 32),
        # a serving batch: 67 MB of states read and written per layer and token
        _operator("decode B64 H64", "decode", 64, 1, 64),
        # one short prompt, its state kept for decoding: few sequences, a short chain
        _operator("prompt B1 T512 H32", "prompt", 1, 512, 32, decay="spectrum"),
        # the 7B-shape prompt batch of the inference workload, one layer of it
        _operator("prompt B16 T4096 H64", "prompt", 16, 4096, 64),
        # the parity configuration, fp32: the smallest training call, launches and host work
        _operator("train B2 T64 H2 f32", "train", 2, 64, 2, dtype="f32"),
        # a small model on odd-length text (768 wide, T not a multiple of anything)
        _operator("train B3 T1003 H12", "train", 3, 1003, 12, decay="spectrum"),
        # the headline configuration
        _operator("train B8 T4096 H32", "train", 8, 4096, 32),
        # the long-sequence configuration, cut into segments by the operator
        _operator("train B1 T131072 H32 auto", "train", 1, 131072, 32, segments="auto"),
        # fp32 training and parity work at an ordinary size
        _operator("train B2 T1024 H32 f32", "train", 2, 1024, 32, dtype="f32"),
        # training step of the 1.6B shape (2048 wide), two layers of it
        _model("model step D2048 B4 T1024", "step", 4, 1024, 2048, 2),
        # prompts of the 7B shape (4096 wide), odd length, two layers
        _model("model prompt D4096 B4 T1001", "prompt", 4, 1001, 4096, 2),
        # token step of the 7B shape at the inference workload's batch, four layers
        _model("model decode D4096 B16", "decode", 16, 1, 4096, 4),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    what = rng.choice(("decode", "prompt", "train", "train", "train", "step", "model prompt", "model decode"))
    H = rng.choice((2, 4, 8, 12, 16, 20, 32, 40, 64))
    decay = rng.choice(("uniform", "spectrum"))
    if what == "decode":
        return _operator(None, "decode", _log(rng, 1, 128), 1, H, rng.choice(("bf16", "bf16", "f16", "f32")), decay)
    if what == "prompt":
        dtype = rng.choice(("bf16", "bf16", "bf16", "f32"))
        return _operator(None, "prompt", _log(rng, 1, 16), _log(rng, 16, 4096 if dtype == "bf16" else 2048), H, dtype, decay)
    if what == "train":
        dtype = rng.choice(("bf16", "bf16", "bf16", "bf16", "f16", "f32"))
        if dtype == "bf16" and rng.random() < 0.25:      # long sequences, left to the operator to cut
            T = 64 * _log(rng, 128, 2048)
            return _operator(None, "train", 1, T, min(H, 32), "bf16", decay, "auto")
        return _operator(None, "train", _log(rng, 1, 8), _log(rng, 16, 4096 if dtype == "bf16" else 2048), min(H, 32), dtype, decay)
    D = rng.choice((768, 1024, 2048))
    if what == "step":
        return _model(None, "step", rng.randint(1, 4), _log(rng, 64, 1024), D, rng.randint(1, 2))
    D = rng.choice((1024, 2048, 2560, 4096))
    if what == "model prompt":
        return _model(None, "prompt", rng.randint(1, 4), _log(rng, 16, 1000), D, 2)
    return _model(None, "decode", _log(rng, 1, 64), 1, D, rng.randint(2, 4))


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _decays(g, B, T, H, decay):
    if decay == "uniform":
        return torch.rand(B, T, H * N, generator=g, device="cuda") * 7.0 - 6.0
    spectrum = torch.linspace(-6.0, 0.5, N, device="cuda").repeat(H)
    return spectrum + 0.3 * torch.randn(B, T, H * N, generator=g, device="cuda")


def _prepare_operator(c, seed):
    g = _generator(seed)
    B, T, H, dt = c["B"], c["T"], c["H"], DTYPES[c["dtype"]]

    def normal(scale, *shape):
        return torch.randn(*shape, generator=g, device="cuda") * scale

    s = dict(c, x=[normal(N ** -0.5, B, T, H * N).to(dt) for _ in range(3)] + [_decays(g, B, T, H, c["decay"]).to(dt)],
             u=normal(0.1, H, N))
    segments = c["segments"] if c["segments"] == "auto" else int(c["segments"])
    s["op"] = RWKVKernelOperator(N, T, segments=segments)
    if c["do"] == "train":   # what autograd hands an operator in the middle of a network: tensors that need gradients, and gy
        s["x"] = [t.requires_grad_(True) for t in s["x"]]
        s["u"].requires_grad_(True)
        s["gy"] = normal(1.0, B, T, H * N).to(torch.float32 if dt == torch.float16 else dt)
    else:                    # a carried state per sequence
        s["state"] = normal(0.1, B, H, N, N)
    return s


def _prepare_model(c, seed):
    D, layers = c["D"], c["layers"]
    torch.manual_seed(seed)
    with torch.device("cuda"):
        model = RWKV6(layers, VOCAB, D, head_size=N, decomposer_size=32, expand_size=D * 7 // 2, decay_rank=64)
    model = model.to_bf16_()
    g = _generator(seed)
    s = dict(c, model=model)
    if c["do"] == "step":
        s["tokens"] = torch.randint(0, VOCAB, (c["B"], c["T"] + 1), generator=g, device="cuda")
        s["parameters"] = list(model.parameters())
        return s
    model.eval()
    if c["do"] == "prompt":
        s["tokens"] = torch.randint(0, VOCAB, (c["B"], c["T"]), generator=g, device="cuda")
        return s
    # a decoding program holds the states a prompt left, the next token of each sequence, and a graph of one step
    prompt = torch.randint(0, VOCAB, (c["B"], 33), generator=g, device="cuda")
    _, states = model.prefill(prompt[:, :32])
    s["token"] = prompt[:, 32:].contiguous()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):        # one step outside the capture, as CUDA graphs of library calls need
        model.decode(s["token"], states)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        logits = model.decode(s["token"], states)
    s["graph"], s["logits"], s["states"] = graph, logits, states
    return s


def prepare(case, seed):
    return _prepare_operator(case, seed) if case["kind"] == "operator" else _prepare_model(case, seed)


def run(s):
    if s["kind"] == "operator":
        r, k, v, w = s["x"]
        if s["do"] == "train":
            y, _ = s["op"](r, k, v, w, s["u"])
            return (y, *torch.autograd.grad(y, (r, k, v, w, s["u"]), s["gy"]))
        return s["op"](r, k, v, w, s["u"], return_state=True, init_state=s["state"])
    if s["do"] == "step":
        tokens = s["tokens"]
        loss = lm_loss(s["model"](tokens[:, :-1]), tokens[:, 1:])
        return (loss, *torch.autograd.grad(loss, s["parameters"]))
    if s["do"] == "prompt":
        return s["model"].prefill(s["tokens"])
    s["graph"].replay()
    return s["logits"], s["states"]


def _layer_weights(D):
    """Parameters of one layer's matrix products: r, k, v, g, o and the receptance, key and value, the two low-rank pairs."""
    return 6 * D * D + 2 * D * (D * 7 // 2) + 2 * 64 * D + 2 * 5 * 32 * D


def work(case):
    B, T = case["B"], case["T"]
    if case["kind"] == "operator":
        H, e = case["H"], DTYPES[case["dtype"]].itemsize
        o = 2 if case["dtype"] == "bf16" else 4                    # fp16 inputs give fp32 results
        rows, pairs, state = B * T * H, B * T * H * N, 4 * B * H * N * N
        if case["do"] == "train":  # r, k, v, w, gy in once for each direction; y and four gradients out
            return {"bytes": pairs * (8 * e + o + 5 * o), "flops": rows * N * N * (4 + 10)}
        return {"bytes": pairs * (4 * e + o) + 2 * state, "flops": rows * N * N * 4}
    D, layers = case["D"], case["layers"]
    H, tokens, P = D // N, B * T, layers * _layer_weights(case["D"])
    wkv = layers * tokens * H * N * N
    if case["do"] == "step":   # weights in, their gradients out; the embedding's gradient is written whole, its rows read by token
        return {"bytes": 2 * (2 * P + 3 * VOCAB * D) + 2 * tokens * D, "flops": 6 * tokens * (P + VOCAB * D) + wkv * 14}
    state = 4 * layers * B * H * N * N
    rows = B                   # positions whose logits are wanted
    moved = 2 * (P + VOCAB * D) + 2 * tokens * D + 2 * rows * VOCAB + state * (2 if case["do"] == "decode" else 1)
    return {"bytes": moved, "flops": 2 * tokens * P + 2 * rows * VOCAB * D + wkv * 4}


def tolerance(case):
    if case["kind"] != "operator":
        # bf16 activations and weights through a few layers; the gradients of small parameters are sums of bf16 terms
        return {"rel": 3e-2 if case["do"] == "step" else 2e-2}
    if case["dtype"] == "bf16":
        # bf16 results; the decay's gradient is a difference of bf16 products
        return {"rel": 2e-2 if case["do"] == "train" else 1e-2}
    return {"rel": 2e-5}       # fp32 sums over up to a few thousand steps (fp16 inputs are exact in fp32)
