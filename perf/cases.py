"""What a user of this framework has it do: the MoE feed-forward block of a Qwen3-30B-A3B-shaped model
(hidden 2048, 128 experts, 8 per token, expert FFN 768; Q4_K gate/up, Q6_K or Q4_K down) from one
decoded token to a full prompt batch of 4096, on device and on host buffers, and the dense
projections beside it.

All cases share one loaded model, as a user's process does: one context, its weights uploaded once
per process.  What differs from case to case and from seed to seed are the activations.
"""
import math

import numpy as np
import torch

from tie_b200 import moe, synth

HIDDEN, EXPERTS, TOP_K, FFN = 2048, 128, 8, 768
MAX_TOKENS = 4096  # the largest prompt batch of the reference
LAYERS = 16  # kept loaded: about 6 GB, so that a step through them never finds its weights in L2
DOWN_KINDS = ("q6_k", "q4_k")  # layers alternate, as files of the Q4_K_M mix have both

# (in, out) of the dense projections of this model: q, k/v, attention output
PROJECTIONS = ((2048, 4096), (2048, 512), (4096, 2048))


def listed():
    return [
        # one token through consecutive blocks, the residual stream on the device, one call per token
        {"name": "stack_decode_1", "call": "stack", "tokens": 1, "layers": 16},
        # one token through the drop-in call of the reference's layer function: pageable host buffers, one
        # synchronous call per layer
        {"name": "host_decode_1", "call": "host", "tokens": 1, "layers": 8, "route": "plain"},
        # a few sequences decoded together, one call per layer as between attention halves
        {"name": "blocks_decode_4", "call": "blocks", "tokens": 4, "layers": 8},
        # a small serving batch of an odd size
        {"name": "blocks_decode_13", "call": "blocks", "tokens": 13, "layers": 4},
        # batched decode under load imbalance: about 30 % of the rows on four hot experts
        {"name": "batch_64_skewed", "call": "ffn", "tokens": 64, "route": "skewed"},
        # a larger decode batch with the LFM2 form of the routing
        {"name": "batch_100_lfm2", "call": "ffn", "tokens": 100, "route": "lfm2"},
        # a short prompt on host buffers, odd length, through the drop-in call
        {"name": "host_prompt_333", "call": "host", "tokens": 333, "layers": 1, "route": "plain"},
        # the prompt batch the headline number is quoted on
        {"name": "prompt_512", "call": "ffn", "tokens": 512, "route": "plain"},
        # a longer, ragged prompt
        {"name": "prompt_1000", "call": "ffn", "tokens": 1000, "route": "plain"},
        # the largest prompt batch
        {"name": "prompt_4096", "call": "ffn", "tokens": 4096, "route": "plain"},
        # attention output projection of a prompt batch
        {"name": "projection_q4k_512", "call": "mat_mat", "tokens": 512, "in": 4096, "out": 2048, "type": "q4_k"},
        # k/v projection of a short ragged batch, the weight kind Q4_K_M files use for v
        {"name": "projection_q6k_37", "call": "mat_mat", "tokens": 37, "in": 2048, "out": 512, "type": "q6_k"},
    ]


def _spread(rng, lo, hi):
    """A whole number from lo to hi, spread evenly over the logarithm."""
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    call = rng.choice(("stack", "host", "blocks", "ffn", "ffn", "ffn", "mat_mat"))
    if call == "stack":
        return {"call": call, "tokens": 1, "layers": rng.randint(4, LAYERS)}
    if call == "blocks":
        return {"call": call, "tokens": _spread(rng, 1, 16), "layers": rng.randint(2, 4)}
    if call == "mat_mat":
        k, n = rng.choice(PROJECTIONS)
        return {"call": call, "tokens": _spread(rng, 16, 2048), "in": k, "out": n, "type": rng.choice(("q4_k", "q6_k"))}
    c = {"call": call, "tokens": _spread(rng, 5, MAX_TOKENS) if call == "ffn" else _spread(rng, 1, 512)}
    if call == "host":
        c["layers"] = 4 if c["tokens"] <= 16 else 1
    c["route"] = rng.choice(("plain", "plain", "skewed", "lfm2")) if call == "ffn" else "plain"
    return c


# ---- the loaded model ----

_loaded = {}


def _block_bytes(kind):
    return synth.Q4K_BYTES if kind == "q4_k" else synth.Q6K_BYTES


def _ggml_type(kind):
    return synth.GGML_Q4_K if kind == "q4_k" else synth.GGML_Q6_K


def _random_blocks(gen, n, kind):
    """n valid super-blocks of the kind, uniform quants and scales, d ~ U(1e-3, 4e-3), dmin ~ U(0, 2e-3)."""
    b = torch.randint(0, 256, (n, _block_bytes(kind)), dtype=torch.uint8, device="cuda", generator=gen)

    def half(lo, hi):
        return (lo + (hi - lo) * torch.rand(n, 1, device="cuda", generator=gen)).half().view(torch.uint8)

    if kind == "q4_k":  # d, dmin, 12 bytes of 6-bit scales and mins, 128 bytes of nibbles
        b[:, 0:2] = half(1e-3, 4e-3)
        b[:, 2:4] = half(0.0, 2e-3)
    else:  # 192 bytes of quants, 16 signed scales, d
        b[:, 192:208] = torch.randint(-32, 32, (n, 16), dtype=torch.int8, device="cuda", generator=gen).view(torch.uint8)
        b[:, 208:210] = half(1e-3, 4e-3)
    return b.reshape(-1).cpu().numpy()


def _model():
    if _loaded:
        return _loaded
    gen = torch.Generator(device="cuda").manual_seed(20)
    gu, dn = FFN * HIDDEN // 256, HIDDEN * FFN // 256  # super-blocks per expert
    # neighbouring layers take overlapping windows of one pool of experts: distinct layers, quickly made
    pool = EXPERTS + LAYERS
    gate, up = _random_blocks(gen, pool * gu, "q4_k"), _random_blocks(gen, pool * gu, "q4_k")
    down = {kind: _random_blocks(gen, pool * dn, kind) for kind in DOWN_KINDS}
    be = moe.MoeBackend(HIDDEN, EXPERTS, TOP_K, FFN, n_layers=LAYERS, max_tokens=MAX_TOKENS)
    stream = torch.cuda.Stream()
    be.set_stream(stream.cuda_stream)
    norm = np.ones(HIDDEN, dtype=np.float32)
    for layer in range(LAYERS):
        router = (0.02 * torch.randn(EXPERTS, HIDDEN, device="cuda", generator=gen)).cpu().numpy()
        kind = DOWN_KINDS[layer % 2]
        g, d = gu * synth.Q4K_BYTES, dn * _block_bytes(kind)
        experts = synth.MoeLayer(synth.MoeShape(), router, gate[layer * g:(layer + EXPERTS) * g], up[layer * g:(layer + EXPERTS) * g],
                                 down[kind][layer * d:(layer + EXPERTS) * d], down_type=_ggml_type(kind))
        be.upload_layer(layer, experts, norm)
    # the selection bias of the skewed load: alpha * ln(p * E) of a Zipf(1.1) popularity
    logp, _ = synth.zipf_logp(EXPERTS, 0)
    bias = torch.from_numpy((0.5536 * logp).astype(np.float32)).cuda()
    _loaded.update(be=be, stream=stream, bias=bias, projections={})
    return _loaded


def _projection(m, case):
    """The registered dense tensor of the case: host address, for the library to find its device copy by."""
    key = (case["in"], case["out"], case["type"])
    if key not in m["projections"]:
        gen = torch.Generator(device="cuda").manual_seed(sum(key[:2]))
        w = _random_blocks(gen, case["in"] * case["out"] // 256, case["type"])
        m["be"].register_tensor(w, _ggml_type(case["type"]), case["in"])
        m["projections"][key] = w
    return m["projections"][key]


# ---- the cases ----

def prepare(case, seed):
    m = _model()
    gen = torch.Generator(device="cuda").manual_seed(seed)
    t, call = case["tokens"], case["call"]

    def normal(*shape):
        return torch.randn(*shape, device="cuda", generator=gen)

    s = {"case": case, "be": m["be"], "stream": m["stream"], "bias": m["bias"]}
    if call == "mat_mat":
        s.update(w=_projection(m, case), x=normal(t, case["in"]), out=torch.empty(t, case["out"], device="cuda"))
    elif call == "stack":
        s.update(x=normal(t, HIDDEN), hidden=torch.empty(t, HIDDEN, device="cuda"))
    elif call == "blocks":  # every layer's own residual rows, as the attention halves would leave them
        s.update(x=normal(case["layers"], t, HIDDEN), hidden=torch.empty(case["layers"], t, HIDDEN, device="cuda"))
    elif call == "host":
        s.update(x=list(normal(case["layers"], t, HIDDEN).cpu().numpy()),
                 out=[np.empty((t, HIDDEN), dtype=np.float32) for _ in range(case["layers"])])
    else:
        s.update(x=normal(t, HIDDEN), out=torch.empty(t, HIDDEN, device="cuda"))
    return s


def run(s):
    case, be = s["case"], s["be"]
    t, call = case["tokens"], case["call"]
    flags = moe.DEVICE | moe.NO_SYNC | moe.GRAPH
    if call == "stack":
        with torch.cuda.stream(s["stream"]):
            s["hidden"].copy_(s["x"])
        be.moe_stack_inplace_ptr(0, case["layers"], s["hidden"], t, flags)
        return s["hidden"]
    if call == "blocks":
        with torch.cuda.stream(s["stream"]):
            s["hidden"].copy_(s["x"])
        for layer in range(case["layers"]):
            be.moe_block_inplace_ptr(layer, s["hidden"][layer], t, flags)
        return s["hidden"]
    if call == "mat_mat":
        return be.mat_mat(s["w"], s["x"], s["out"], t, case["in"], case["out"], moe.DEVICE | moe.NO_SYNC)
    if call == "host":
        for layer in range(case["layers"]):
            be.moe_ffn_ptr(layer, s["x"][layer], s["out"][layer], t, moe.HOST | moe.GRAPH)
        return s["out"]
    if case["route"] == "lfm2":
        flags |= moe.ROUTE_LFM2
    be.moe_ffn_ptr(0, s["x"], s["out"], t, flags, s["bias"] if case["route"] == "skewed" else None)
    return s["out"]


def work(case):
    t = case["tokens"]
    if case["call"] == "mat_mat":
        k, n = case["in"], case["out"]
        return {"bytes": k * n // 256 * _block_bytes(case["type"]) + 4 * t * (k + n), "flops": 2 * t * k * n}
    # the router, the weights of every expert that is expected to get a token, the activations in and out
    layers = case.get("layers", 1)
    active = EXPERTS * (1.0 - (1.0 - TOP_K / EXPERTS) ** t)
    if case.get("route") == "skewed":  # fewer of them: counted on random scores under the bias
        logp, _ = synth.zipf_logp(EXPERTS, 0)
        scores = 0.9 * np.random.RandomState(0).randn(t, EXPERTS) + 0.5536 * logp
        active = len(np.unique(np.argpartition(-scores, TOP_K, axis=1)[:, :TOP_K]))
    weights = 0.0
    for layer in range(layers):
        weights += 4 * EXPERTS * HIDDEN
        weights += active * HIDDEN * FFN // 256 * (2 * synth.Q4K_BYTES + _block_bytes(DOWN_KINDS[layer % 2]))
    rows = layers * t if case["call"] != "stack" else t  # the stack's rows stay on the chip between layers
    return {"bytes": weights + 8 * rows * HIDDEN,
            "flops": layers * t * (2 * EXPERTS * HIDDEN + TOP_K * 6 * HIDDEN * FFN)}


def tolerance(case):
    # fp32 sums over exact integer weights times activations of 22 bits or more, the largest Q6_K products
    # rounded to 11 bits; the stack feeds each block's error to the next one
    if case["call"] == "stack":
        return {"rel": 1e-4, "max": 2e-3}
    return {"rel": 3e-5, "max": 5e-4}
