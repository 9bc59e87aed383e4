"""The work that is timed: whole decode steps of GPT-2 and single layers of the other designs, through the calls that a
program makes that holds a model, a cache manager and a step runner.

A case names its ``kind`` and its sizes:

``decode``   one step of the engine's decode path: every request brings one token, the step is packed, uploaded and replayed
             from its CUDA graph, and returns logits (``DecodeGraphs.run``);
``block``    one GPT-2 layer (norm, attention, norm, feed-forward) over a mixed step: prompt portions beside single tokens;
``latent``   a latent attention (one cached latent of 512 and a rotated key part of 64 per token, shared by all heads);
``rotary``   a grouped rotary attention (four query heads to a key/value head, head norms, learned sinks, optional chunks);
``moe``      a routed feed-forward: 16 experts of which 2 run per token, beside a shared one;
``mlstm``    a matrix memory per head with exponential gates.

A layer's step of single tokens is captured once into a CUDA graph and replayed, as a serving loop does; every other
layer is called as ``Model.forward`` calls it.  Weights have the distributions of the random-weights mode, rows are
normed activations, and cached keys and values lie in pages that earlier steps filled."""

from __future__ import annotations

import math

import numpy as np
import torch

from ayaka_py_b200.cache.manager import CacheManager
from ayaka_py_b200.engine.graphs import DecodeGraphs
from ayaka_py_b200.engine.step import StepEntry, StepRunner
from ayaka_py_b200.models.model import Model
from ayaka_py_b200.registry import architecture_for
from ayaka_py_b200.weights.loader import DictStore, load_weights
from ayaka_py_b200 import models, parts  # noqa: F401  (register the architectures and the part kinds)

DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
PAGE = 16
EPS = 1e-6
RANK, ROT, HEAD = 512, 64, 128         # latent, its rotated part, size of a head in the designs other than GPT-2
EXPERTS, TOP = 16, 2
GATE_CAP = 15.0
VOCAB = 256                            # of the one-layer models, whose embedding and head are not run
GPT2_SHAPES = {768: (12, 12), 1024: (16, 24), 1280: (20, 36), 1600: (25, 48)}      # width: heads, layers


# ------------------------------------------------------------------- cases --

def listed():
    return [
        # one user of the small model: the least work a step can have, where launches and latency are all there is
        {"name": "gpt2-small-decode-1", "kind": "decode", "width": 768, "layers": 12, "vocab": 50257, "requests": 1, "context": 96},
        # the headline workload: decode steps of the XL shape at 8 requests
        {"name": "gpt2-xl-decode-8", "kind": "decode", "width": 1600, "layers": 48, "vocab": 50257, "requests": 8, "context": 590},
        # a layer of the XL shape while two whole prompts are read
        {"name": "gpt2-xl-prefill-2x1024", "kind": "block", "dtype": "bfloat16", "width": 1600, "prompts": 2, "rows": 1024, "ragged": 0,
         "start": 0, "decodes": 0, "context": 0},
        # continuous batching of the large shape: 64 requests decode beside a 512-token portion of a long prompt
        {"name": "gpt2-large-mixed-64+512", "kind": "block", "dtype": "bfloat16", "width": 1280, "prompts": 1, "rows": 512, "ragged": 0,
         "start": 256, "decodes": 64, "context": 600},
        # the true 32-bit engine on short ragged prompts and a few decoding requests
        {"name": "gpt2-small-float32-ragged", "kind": "block", "dtype": "float32", "width": 768, "prompts": 3, "rows": 161, "ragged": 37,
         "start": 0, "decodes": 5, "context": 200},
        # latent attention while two prompts of unequal length are read
        {"name": "latent-prefill-1024+777", "kind": "latent", "width": 2048, "window": 0, "requests": 2, "rows": 1024, "ragged": 247,
         "context": 0},
        # the same layer while 8 requests decode
        {"name": "latent-decode-8", "kind": "latent", "width": 2048, "window": 0, "requests": 8, "rows": 1, "ragged": 0, "context": 576},
        # grouped attention inside chunks while two whole prompts are read
        {"name": "rotary-prefill-2x1024", "kind": "rotary", "width": 2048, "chunk": 512, "requests": 2, "rows": 1024, "ragged": 0,
         "context": 0},
        # grouped attention over long contexts while 32 requests decode
        {"name": "rotary-decode-32", "kind": "rotary", "width": 2048, "chunk": 0, "requests": 32, "rows": 1, "ragged": 0, "context": 1900},
        # routed experts while prompts are read: every expert has many rows
        {"name": "moe-prefill-2048", "kind": "moe", "width": 2048, "rows": 2048},
        # routed experts while 8 requests decode: every pair streams its expert
        {"name": "moe-decode-8", "kind": "moe", "width": 2048, "rows": 8},
        # the matrix memory while two prompts of unequal length are read
        {"name": "mlstm-prefill-1024+777", "kind": "mlstm", "width": 2048, "requests": 2, "rows": 1024, "ragged": 247},
    ]


def _spread(rng, low, high):
    """A whole number between low and high, even over its logarithm."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["decode", "block", "block", "latent", "latent", "latent", "rotary", "rotary", "moe", "moe", "mlstm"])
    if kind == "decode":
        width = rng.choice([768, 1024, 1280, 1600])
        return {"kind": kind, "width": width, "layers": rng.randint(2, 12), "vocab": 50257, "requests": _spread(rng, 1, 64),
                "context": _spread(rng, 8, 900)}
    if kind == "block":
        dtype = rng.choice(["bfloat16", "bfloat16", "bfloat16", "float32"])
        width = rng.choice([768, 1024, 1280, 1600]) if dtype == "bfloat16" else 768
        prompts = rng.randint(1, 3)
        rows = _spread(rng, 2, (1024 if prompts <= 2 else 600) if dtype == "bfloat16" else 200)
        return {"kind": kind, "dtype": dtype, "width": width, "prompts": prompts, "rows": rows, "ragged": rng.randint(0, rows // 4),
                "start": 0 if rows > 500 else rng.choice([0, rng.randint(1, 500)]),
                "decodes": rng.choice([0, _spread(rng, 1, 64 if dtype == "bfloat16" else 8)]), "context": _spread(rng, 8, 900)}
    width = rng.choice([1024, 2048]) if kind != "moe" else rng.choice([512, 1024, 2048])
    if kind == "moe":
        return {"kind": kind, "width": width, "rows": _spread(rng, 1, 2048)}
    requests = rng.randint(1, 2)
    rows = _spread(rng, 2, 1024)
    if kind == "mlstm":
        return {"kind": kind, "width": width, "requests": requests, "rows": rows, "ragged": rng.randint(0, rows // 4)}
    reach = "window" if kind == "latent" else "chunk"
    if rng.random() < 0.4:                                 # a decode step
        return {"kind": kind, "width": width, reach: rng.choice([0, 0, 512]), "requests": _spread(rng, 1, 32), "rows": 1, "ragged": 0,
                "context": _spread(rng, 8, 1500 if kind == "latent" else 1900)}
    return {"kind": kind, "width": width, reach: rng.choice([0, 512]), "requests": requests, "rows": rows,
            "ragged": rng.randint(0, rows // 4), "context": 0 if rows > 500 else rng.choice([0, rng.randint(1, 500)])}


def _entries(case):
    """(tokens cached before, tokens brought) of every request, in the order in which the step packs them."""
    kind = case["kind"]
    if kind == "moe":
        return [(0, case["rows"])]
    if kind == "decode":
        return [(max(1, case["context"] - 7 * i), 1) for i in range(case["requests"])]
    if kind == "block":
        single = [(max(1, case["context"] - 5 * i), 1) for i in range(case["decodes"])]
        prompts = [(case["start"], max(2, case["rows"] - i * case["ragged"])) for i in range(case["prompts"])]
        return single + prompts
    start = case.get("context", 0)
    least = 1 if case["rows"] == 1 else 2
    return [(max(1, start - 13 * i) if start else 0, max(least, case["rows"] - i * case["ragged"])) for i in range(case["requests"])]


def _dtype(case):
    return DTYPES[case.get("dtype", "bfloat16")]


def _graphed(case):
    """Does a serving loop replay this layer's step from a graph?  Steps of single tokens only."""
    return case["kind"] in ("latent", "rotary") and case["rows"] == 1 or case["kind"] == "moe" and case["rows"] <= 64


# ------------------------------------------------------ weights and inputs --

def _document(case):
    d, kind = case["width"], case["kind"]
    heads = d // HEAD
    if kind in ("decode", "block"):
        return {"architectures": ["GPT2LMHeadModel"], "model_type": "gpt2", "vocab_size": case.get("vocab", VOCAB), "n_positions": 2048 if kind == "block" else 1024,
                "n_embd": d, "n_layer": case.get("layers", 1), "n_head": GPT2_SHAPES[d][0], "n_inner": 4 * d,
                "layer_norm_epsilon": 1e-5, "activation_function": "gelu_new"}
    if kind == "mlstm":
        layer = {"type": "mlstm", "mixer": {"heads": heads, "dim": HEAD, "vdim": HEAD, "gate_cap": GATE_CAP}, "mlp": None}
        return {"architecture": "Tesozen", "vocab": VOCAB, "width": d, "norm": {"eps": EPS}, "embedding": {"scale": 1.0}, "layers": [layer]}
    if kind == "latent":
        mixer = {"heads": heads, "dim": HEAD, "rot_dim": ROT, "vdim": HEAD, "kv_rank": RANK, "scale": (HEAD + ROT) ** -0.5,
                 "rot": {"base": 500000.0, "dims": ROT}}
        if case["window"]:
            mixer["mask"] = {"size": case["window"]}
        layer = {"type": "latent_attention", "mixer": mixer, "mlp": None}
    else:
        mixer = {"heads": heads, "kv_heads": max(1, heads // 4), "dim": HEAD, "vdim": HEAD, "scale": HEAD ** -0.5,
                 "rot": {"base": 50000.0, "dims": 64}}
        if kind == "moe":
            mixer.update(heads=1, kv_heads=1)
        if case.get("chunk"):
            mixer["mask"] = {"size": case["chunk"]}
        layer = {"type": "attention", "mixer": mixer, "mlp": None}
        if kind == "moe":
            layer["mlp"] = {"kind": "moe", "router": {"experts": EXPERTS, "top": TOP}, "expert": {"ff": d}, "shared": {"ff": d * 3 // 4}}
    return {"architecture": "Tomodra", "vocab": VOCAB, "width": d, "norm": {"eps": EPS}, "postln_alpha": 1.5, "layers": [layer]}


class _Source:
    """Seeded numbers on the GPU, in the order in which they are asked for."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)

    def normal(self, shape, std=1.0, mean=0.0, dtype=torch.float32):
        return torch.randn(shape, generator=self.gen, dtype=torch.float32, device="cuda").mul_(std).add_(mean).to(dtype)


def _weights(case, seed):
    """Checkpoint name -> tensor, with the spreads that the architectures give their random weights."""
    src, dtype, d, kind = _Source(seed), _dtype(case), case["width"], case["kind"]
    heads, out = d // HEAD, {}

    def matrix(name, rows, cols, std=None, gain=1.0):
        out[name] = src.normal((rows, cols), gain / math.sqrt(cols) if std is None else std, dtype=dtype)

    def vector(name, n, std, mean=0.0):
        out[name] = src.normal((n,), std, mean)

    if kind in ("decode", "block"):
        layers = case.get("layers", 1)
        matrix("transformer.wte.weight", case.get("vocab", VOCAB), d, 0.02)
        matrix("transformer.wpe.weight", 2048 if kind == "block" else 1024, d, 0.02)
        for i in range(layers):
            p = f"transformer.h.{i}."
            small = 0.02 / math.sqrt(2.0 * GPT2_SHAPES[d][1])
            for norm in ("ln_1", "ln_2"):
                vector(p + norm + ".weight", d, 0.05, 1.0)
                vector(p + norm + ".bias", d, 0.02)
            for name, rows, cols, std in (("attn.c_attn", d, 3 * d, 0.02), ("attn.c_proj", d, d, small),
                                          ("mlp.c_fc", d, 4 * d, 0.02), ("mlp.c_proj", 4 * d, d, small)):
                matrix(p + name + ".weight", rows, cols, std)
                vector(p + name + ".bias", cols, 0.01)
        vector("transformer.ln_f.weight", d, 0.05, 1.0)
        vector("transformer.ln_f.bias", d, 0.02)
        return out
    matrix("embed", VOCAB, d, 1.0)
    m, f = "l0.mix.", "l0.mlp."
    if kind == "mlstm":
        for name, rows in (("q", d), ("k", d), ("v", d), ("i", heads), ("f", heads), ("g", d), ("o", d)):
            matrix(m + name, rows, d)
        vector(m + "i.b", heads, 0.5)
        vector(m + "f.b", heads, 1.0, 2.0)
        vector(m + "norm", d, 0.1, 1.0)
        for name in ("l0.norm1", "l0.norm1b", "final.norm"):
            vector(name, d, 0.1, 1.0)
            vector(name + ".b", d, 0.1)
        return out
    matrix("head", VOCAB, d)
    vector("final.norm", d, 0.1, 1.0)
    vector("l0.norm1", d, 0.1, 1.0)
    if kind == "latent":
        matrix(m + "q", heads * (HEAD + ROT), d)
        matrix(m + "dkv", RANK + ROT, d)
        vector(m + "dkv.norm", RANK, 0.1, 1.0)
        matrix(m + "uk", d, RANK)
        matrix(m + "uv", d, RANK)
        matrix(m + "o", d, d)
        return out
    h, g = (1, 1) if kind == "moe" else (heads, max(1, heads // 4))
    for name, rows in (("q", h * HEAD), ("k", g * HEAD), ("v", g * HEAD)):
        matrix(m + name, rows, d)
    matrix(m + "o", d, h * HEAD)
    vector(m + "q.norm", HEAD, 0.1, 1.0)
    vector(m + "k.norm", HEAD, 0.1, 1.0)
    vector(m + "sink", h, 0.5)
    if kind == "moe":
        inner, shared = d, d * 3 // 4
        vector("l0.norm2", d, 0.1, 1.0)
        matrix(f + "router", EXPERTS, d, gain=2.0)
        matrix(f + "shared.gate", shared, d)
        matrix(f + "shared.up", shared, d)
        matrix(f + "shared.down", d, shared)
        matrix(f + "shared.sg", 1, d)
        for e in range(EXPERTS):
            matrix(f"{f}e{e}.gate", inner, d)
            matrix(f"{f}e{e}.up", inner, d)
            matrix(f"{f}e{e}.down", d, inner)
    return out


def _tokens(case, seed):
    entries, rs = _entries(case), np.random.RandomState(seed % (1 << 31))
    return [rs.randint(0, case.get("vocab", VOCAB), n).tolist() for _, n in entries]


def _rows(case, seed):
    """What a layer is given: normed rows in the compute dtype, for a GPT-2 layer the 32-bit stream itself."""
    total = sum(n for _, n in _entries(case))
    src = _Source(seed + 101)
    return src.normal((total, case["width"]), 0.1) if case["kind"] == "block" else src.normal((total, case["width"]), dtype=_dtype(case))


def _cached(case, seed, layer):
    """Keys and values that earlier steps cached for every request: [(keys [n, heads, size], values [n, heads, size])]."""
    src, d, kind = _Source(seed + 1009 * (layer + 1)), case["width"], case["kind"]
    dtype = _dtype(case)
    key, value = {"latent": ((1, ROT), (1, RANK)), "rotary": ((max(1, d // HEAD // 4), HEAD),) * 2}.get(kind) or (
        (GPT2_SHAPES[d][0], 64),) * 2
    std = 0.02 * math.sqrt(d) if kind in ("decode", "block") else 1.0
    return [(src.normal((start, *key), std, dtype=dtype), src.normal((start, *value), std, dtype=dtype)) for start, _ in _entries(case)]


# ------------------------------------------------------------ prepare, run --

def prepare(case, seed):
    document, kind, dtype = _document(case), case["kind"], _dtype(case)
    arch = architecture_for(document)
    config = arch.config_class.from_dict(document)
    model = Model(arch.build_spec(config), dtype, "cuda")
    load_weights(model, DictStore(_weights(case, seed)), arch.normalize_name, config)

    entries = _entries(case)
    longest = max(a + n for a, n in entries)
    max_len = 1024 if kind == "decode" else max(1024, -(-longest // 512) * 512)
    pages = sum(-(-(a + n) // PAGE) for a, n in entries) + 2
    total = sum(n for _, n in entries)
    cache = CacheManager(model.groups, kv_pages=pages, page_size=PAGE, max_requests=max(len(entries), 2), max_len=max_len,
                         dtype=dtype, device="cuda")
    runner = StepRunner(model, cache, max_tokens=max(total, 64), max_requests=max(len(entries), 2))
    slots = [cache.open(f"r{i}") for i in range(len(entries))]
    for sl, (start, _) in zip(slots, entries):
        if start:
            cache.commit(cache.reserve([(sl, 0, start)]))
    for layer in range(case.get("layers", 1) if kind in ("decode", "block", "latent", "rotary") else 0):
        keys, values = cache.kv_layer(0, layer)
        table = cache.table_rows(0, slots)
        for row, (start, _), (k, v) in zip(table, entries, _cached(case, seed, layer)):
            if start:
                at = np.flatnonzero(row[np.arange(start) // PAGE])       # pages that a window has passed are given back
                k, v = k[torch.from_numpy(at).cuda()], v[torch.from_numpy(at).cuda()]
                cells = torch.from_numpy(row[at // PAGE].astype(np.int64) * PAGE + at % PAGE).cuda()
                keys.view(-1, *keys.shape[2:])[cells] = k
                values.view(-1, *values.shape[2:])[cells] = v
    tokens = _tokens(case, seed)
    step = [StepEntry(sl, start, toks, [len(toks) - 1]) for sl, (start, _), toks in zip(slots, entries, tokens)]
    reserved = [(sl, start, n) for sl, (start, n) in zip(slots, entries)]
    state = {"kind": kind, "model": model, "cache": cache, "step": step, "reserved": reserved}
    if kind == "decode":
        state["graphs"] = DecodeGraphs(runner, model, len(entries))
        cache.rollback(_run_decode(state)[1])              # captures the step's graph
        torch.cuda.synchronize()
        return state

    cache.reserve(reserved)
    state["ctx"] = ctx = runner.prepare(step)
    state["rows"] = rows = _rows(case, seed)
    block = model.blocks[0]
    binding = model.bindings[0].get("mixer")
    if kind == "block":
        stream = torch.empty_like(rows)

        def layer():
            stream.copy_(rows)
            return block.forward(stream, ctx, model.bindings[0])
    elif kind == "moe":
        def layer():
            return block.ffn.forward(rows, None, ctx)
    elif kind == "mlstm":
        memory = cache.state_layer(binding.group, binding.layer)

        def layer():
            memory.zero_()                                  # requests that start here
            return block.mixer.forward(rows, None, ctx, binding)
    else:
        def layer():
            return block.mixer.forward(rows, None, ctx, binding)
    state["layer"] = layer
    if kind in ("block", "latent", "rotary"):
        state["kept"] = cache.kv[0]
    elif kind == "mlstm":
        state["kept"] = (cache.state[binding.group],)
    else:
        state["kept"] = ()
    if _graphed(case):
        layer()
        torch.cuda.synchronize()
        state["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(state["graph"]):
            state["out"] = layer()
    torch.cuda.synchronize()
    return state


def _run_decode(state):
    reservation = state["cache"].reserve(state["reserved"])
    return state["graphs"].run(state["step"]), reservation


def run(state):
    if state["kind"] == "decode":
        logits, reservation = _run_decode(state)
        state["cache"].rollback(reservation)               # the next pass brings the same tokens again
        return {"logits": logits, "keys": state["cache"].kv[0][0], "values": state["cache"].kv[0][1]}
    if "graph" in state:
        state["graph"].replay()
        out = state["out"]
    else:
        out = state["layer"]()
    return {"out": out, "kept": list(state["kept"])}


# ----------------------------------------------------------- floor of work --

def _seen(case):
    """Sum over the step's rows of the keys that a row sees, and the cached tokens that some row reads."""
    reach = case.get("window") or case.get("chunk") or 0
    pairs = read = 0
    for start, n in _entries(case):
        first = start
        for i in range(start, start + n):
            low = 0
            if reach:
                low = max(0, i - reach + 1) if case["kind"] == "latent" else i // reach * reach
            pairs += i - low + 1
            first = min(first, low)
        read += start - first
    return pairs, read


def work(case):
    d, kind, item = case["width"], case["kind"], _dtype(case).itemsize
    T = sum(n for _, n in _entries(case))
    heads = d // HEAD
    if kind == "moe":
        chosen = min(EXPERTS, EXPERTS * (1.0 - (1.0 - TOP / EXPERTS) ** T))       # experts that some row is expected to choose
        expert, shared = 3 * d * d, 3 * d * (d * 3 // 4)
        return {"bytes": int(item * (chosen * expert + shared + (EXPERTS + 1) * d) + T * d * (item + 4)),
                "flops": 2 * T * (TOP * expert + shared + (EXPERTS + 1) * d)}
    if kind == "mlstm":
        weights = 5 * d * d + 2 * heads * d
        state = heads * (HEAD * HEAD + HEAD + 4) * 4 * case["requests"]
        return {"bytes": item * weights + T * d * (item + 4) + state, "flops": 2 * T * weights + T * heads * 4 * HEAD * (HEAD + 1)}
    pairs, read = _seen(case)
    if kind == "latent":
        weights = d * (heads * (HEAD + ROT) + RANK + ROT) + 2 * d * RANK + d * d
        per_pair = 2 * heads * (RANK + ROT + RANK)
        cached = RANK + ROT
    elif kind == "rotary":
        g = max(1, heads // 4)
        weights = d * (heads + 2 * g) * HEAD + d * d
        per_pair = 4 * d
        cached = 2 * g * HEAD
    else:
        weights = 12 * d * d
        per_pair = 4 * d
        cached = 2 * d
    layer_bytes = item * (weights + cached * (read + T))
    layer_flops = 2 * T * weights + per_pair * pairs
    if kind == "decode":
        head = case["vocab"] * d
        return {"bytes": case["layers"] * layer_bytes + item * head + T * (case["vocab"] * 4 + 2 * d * item),
                "flops": case["layers"] * layer_flops + 2 * T * head}
    return {"bytes": layer_bytes + T * d * ((8 if kind == "block" else item + 4)), "flops": layer_flops}


# --------------------------------------------------------------- tolerance --

def tolerance(case):
    """About four times the difference between the path and the same in 64 bits: in bfloat16 the operands of every product
    are rounded to 16 bits (measured 1.5e-3 for a GPT-2 layer's stream, 1.6e-3 to 3.4e-3 for the other layers, 5e-3 for the
    logits behind all layers), in float32 the sums alone differ (7e-7)."""
    if case.get("dtype") == "float32":
        return {"rel": 4e-6}
    return {"rel": {"decode": 2e-2, "block": 6e-3}.get(case["kind"], 1.2e-2)}


# ------------------------------------------------------- the same in 64 bits --

def _wide(t):
    return t.to(torch.float64)


def _mul(x, w):
    return x @ _wide(w).T


def _rms(x, weight=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)
    return y if weight is None else y * _wide(weight)


def _layernorm(x, weight, bias):
    c = x - x.mean(-1, keepdim=True)
    return c / torch.sqrt((c * c).mean(-1, keepdim=True) + 1e-5) * _wide(weight) + _wide(bias)


def _turn(x, start, base, dims, neighbours):
    """x [n, heads, size]: the first ``dims`` numbers of every head turn by the row's position."""
    freq = base ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device=x.device) / dims)
    angle = (torch.arange(x.shape[0], dtype=torch.float64, device=x.device) + start)[:, None] * freq
    c, s = torch.cos(angle)[:, None], torch.sin(angle)[:, None]
    out = x.clone()
    if neighbours:
        u, v = x[..., 0:dims:2], x[..., 1:dims:2]
        out[..., 0:dims:2], out[..., 1:dims:2] = u * c - v * s, v * c + u * s
    else:
        u, v = x[..., :dims // 2], x[..., dims // 2:dims]
        out[..., :dims // 2], out[..., dims // 2:dims] = u * c - v * s, v * c + u * s
    return out


def _attend(q, k, v, start, scale, window=0, chunk=0, sink=None):
    """Rows q [n, H, D] from position ``start`` on over keys k [m, G, D] and values v [m, G, E] from position 0 on."""
    n, H, _ = q.shape
    i = torch.arange(n, device=q.device)[:, None] + start
    j = torch.arange(k.shape[0], device=q.device)[None]
    seen = j <= i
    if window:
        seen &= i - j < window
    if chunk:
        seen &= i // chunk == j // chunk
    out = []
    for h in range(H):
        g = h // (H // k.shape[1])
        s = (q[:, h] @ k[:, g].T * scale).masked_fill(~seen, -math.inf)
        if sink is not None:
            s = torch.cat([s, _wide(sink[h]).expand(n, 1)], dim=1)
        p = torch.softmax(s, dim=1)[:, :k.shape[0]]
        out.append(p @ v[:, g])
    return torch.stack(out, dim=1)


def _gpt2_layer(x, w, p, case, seed, layer):
    d, entries = case["width"], _entries(case)
    heads, at, mixed = GPT2_SHAPES[d][0], 0, []
    h = _layernorm(x, w[p + "ln_1.weight"], w[p + "ln_1.bias"])
    qkv = h @ _wide(w[p + "attn.c_attn.weight"]) + _wide(w[p + "attn.c_attn.bias"])
    for (start, n), (ck, cv) in zip(entries, _cached(case, seed, layer)):
        q, k, v = (t.reshape(n, heads, 64) for t in qkv[at:at + n].split(d, dim=1))
        o = _attend(q, torch.cat([_wide(ck), k]), torch.cat([_wide(cv), v]), start, 64 ** -0.5)
        mixed.append(o.reshape(n, d))
        at += n
    x = x + torch.cat(mixed) @ _wide(w[p + "attn.c_proj.weight"]) + _wide(w[p + "attn.c_proj.bias"])
    h = _layernorm(x, w[p + "ln_2.weight"], w[p + "ln_2.bias"])
    u = h @ _wide(w[p + "mlp.c_fc.weight"]) + _wide(w[p + "mlp.c_fc.bias"])
    u = 0.5 * u * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (u + 0.044715 * u ** 3)))
    return x + u @ _wide(w[p + "mlp.c_proj.weight"]) + _wide(w[p + "mlp.c_proj.bias"])


def _exact_decode(case, seed, w):
    tokens = torch.tensor([t[0] for t in _tokens(case, seed)], device="cuda")
    places = torch.tensor([start for start, _ in _entries(case)], device="cuda")
    x = _wide(w["transformer.wte.weight"][tokens]) + _wide(w["transformer.wpe.weight"][places])
    for layer in range(case["layers"]):
        x = _gpt2_layer(x, w, f"transformer.h.{layer}.", case, seed, layer)
    h = _layernorm(x, w["transformer.ln_f.weight"], w["transformer.ln_f.bias"])
    return {"logits": _mul(h, w["transformer.wte.weight"]), "keys": None, "values": None}


def _exact_latent(case, seed, w, h):
    H, m, at, out = case["width"] // HEAD, "l0.mix.", 0, []
    for (start, n), (ck, cv) in zip(_entries(case), _cached(case, seed, 0)):
        x = h[at:at + n]
        at += n
        q = _mul(x, w[m + "q"]).reshape(n, H, HEAD + ROT)
        down = _mul(x, w[m + "dkv"])
        c = torch.cat([_wide(cv)[:, 0], _rms(down[:, :RANK], w[m + "dkv.norm"])])
        kr = torch.cat([_wide(ck), _turn(down[:, None, RANK:], start, 500000.0, ROT, False)])
        uk, uv = _wide(w[m + "uk"]).reshape(H, HEAD, RANK), _wide(w[m + "uv"]).reshape(H, HEAD, RANK)
        both = torch.cat([torch.einsum("nhd,hdr->nhr", q[..., :HEAD], uk), _turn(q[..., HEAD:], start, 500000.0, ROT, False)], dim=2)
        o = _attend(both, torch.cat([c[:, None], kr], dim=2), c[:, None], start, (HEAD + ROT) ** -0.5, window=case["window"])
        out.append(_mul(torch.einsum("nhr,hdr->nhd", o, uv).reshape(n, H * HEAD), w[m + "o"]))
    return torch.cat(out)


def _exact_rotary(case, seed, w, h):
    H, m, at, out = case["width"] // HEAD, "l0.mix.", 0, []
    G = max(1, H // 4)
    for (start, n), (ck, cv) in zip(_entries(case), _cached(case, seed, 0)):
        x = h[at:at + n]
        at += n
        q = _turn(_rms(_mul(x, w[m + "q"]).reshape(n, H, HEAD), w[m + "q.norm"]), start, 50000.0, 64, True)
        k = _turn(_rms(_mul(x, w[m + "k"]).reshape(n, G, HEAD), w[m + "k.norm"]), start, 50000.0, 64, True)
        v = _mul(x, w[m + "v"]).reshape(n, G, HEAD)
        o = _attend(q, torch.cat([_wide(ck), k]), torch.cat([_wide(cv), v]), start, HEAD ** -0.5, chunk=case["chunk"], sink=w[m + "sink"])
        out.append(_mul(o.reshape(n, H * HEAD), w[m + "o"]))
    return torch.cat(out)


def _exact_moe(case, w, h):
    f = "l0.mlp."

    def expert(x, p):
        g = _mul(x, w[p + "gate"])
        return _mul(g * torch.sigmoid(g) * _mul(x, w[p + "up"]), w[p + "down"])

    best, chosen = torch.topk(_mul(h, w[f + "router"]), TOP, dim=1)
    out = torch.sigmoid(_mul(h, w[f + "shared.sg"])) * expert(h, f + "shared.")
    for e in range(EXPERTS):
        rows, place = torch.nonzero(chosen == e, as_tuple=True)
        if rows.numel():
            out.index_add_(0, rows, expert(torch.sigmoid(best[rows, place])[:, None] * h[rows], f"{f}e{e}."))
    return out


def _exact_mlstm(case, w, h):
    H, m, at, out = case["width"] // HEAD, "l0.mix.", 0, []
    for _, n in _entries(case):
        x = h[at:at + n]
        at += n
        q = _mul(x, w[m + "q"]).reshape(n, H, HEAD) * HEAD ** -0.5
        k = _mul(x, w[m + "k"]).reshape(n, H, HEAD)
        v = _mul(x, w[m + "v"]).reshape(n, H, HEAD)
        i = GATE_CAP * torch.tanh((_mul(x, w[m + "i"]) + _wide(w[m + "i.b"])) / GATE_CAP)
        f = torch.nn.functional.logsigmoid(GATE_CAP * torch.tanh((_mul(x, w[m + "f"]) + _wide(w[m + "f.b"])) / GATE_CAP))
        # the recurrence unrolled: with b the running sums of f, the maximum is b_t + max(0, max_(s<=t) (i_s - b_s))
        b = f.cumsum(0)
        a = i - b
        top = torch.clamp(torch.cummax(a, dim=0).values, min=0.0)
        rows = []
        for head in range(H):
            reach = torch.exp(a[None, :, head] - top[:, None, head]).tril()
            s = q[:, head] @ k[:, head].T * reach
            rows.append((s @ v[:, head]) / (torch.clamp(s.sum(1).abs(), min=torch.exp(-(b + top)[:, head])) + 1e-6)[:, None])
        o = _rms(torch.stack(rows, dim=1)).reshape(n, H * HEAD)
        out.append(_mul(o * _wide(w[m + "norm"]) * torch.sigmoid(_mul(x, w[m + "g"])), w[m + "o"]))
    return torch.cat(out)


def exact(case, seed):
    w, kind = _weights(case, seed), case["kind"]
    if kind == "decode":
        return _exact_decode(case, seed, w)
    h = _wide(_rows(case, seed))
    if kind == "block":
        return {"out": _gpt2_layer(h, w, "transformer.h.0.", case, seed, 0), "kept": [None, None]}
    if kind == "latent":
        return {"out": _exact_latent(case, seed, w, h), "kept": [None, None]}
    if kind == "rotary":
        return {"out": _exact_rotary(case, seed, w, h), "kept": [None, None]}
    if kind == "moe":
        return {"out": _exact_moe(case, w, h), "kept": []}
    return {"out": _exact_mlstm(case, w, h), "kept": [None]}
