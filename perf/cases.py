"""Performance cases: the work a user of this package has it do, through its public entry points.

Four paths, each over the range of sizes, codebooks and options it is used with:

  linear       one EPTQLinear module call: decode rows, with bias, group scales, ragged sizes
  block        the seven linears of a LLaMA-style decoder layer, q/k/v and gate/up grouped where a
               decode step groups them, as plain module calls in a prefill
  dequantize   bit-exact reconstruction of a layer's fp16 weight
  decode       prompt prefill and greedy token loop of a whole decoder stack in the decode engine

``listed()`` gives the named cases, ``draw(rng)`` one more of the same ranges.  ``prepare`` makes what a
program holds before the call, ``run`` makes the call, ``work`` states the bytes and operations the call
cannot do without, ``tolerance`` how far another correct implementation may be off.
"""
from __future__ import annotations

import math

import torch

from eptq_b200.engine import DecoderLayerWeights, LlamaDecodeEngine
from eptq_b200.kernels.linear import EPTQLinear, forward_group
from eptq_b200.quantizers import E8D4Quantizer, E8LatticeQuantizer
from eptq_b200.synthetic import make_activations, make_layer

DEVICE = "cuda"
CRITICAL_FRACTION = 0.002            # share of 8-weight blocks kept as fp16 critical blocks
GROUP_MAX_TOKENS = 16                # rows a grouped launch takes; longer inputs are module calls
DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
_tables: dict = {}


def listed() -> list:
    return [
        # The smallest call: one fc1 projection of a 125M-parameter OPT at one token, all latency.
        {"name": "opt125m_fc1_e8_1tok", "path": "linear", "codebook": "e8_lattice", "out": 3072, "in": 768,
         "tokens": 1, "bias": False, "qb_size": 0, "dtype": "fp16"},
        # One attention projection of a 7B model called on its own, as an unmodified model's forward does.
        {"name": "linear_4096_d4_1tok", "path": "linear", "codebook": "e8_d4", "out": 4096, "in": 4096,
         "tokens": 1, "bias": False, "qb_size": 0, "dtype": "fp16"},
        # A layer whose sizes fit no tile, with a bias, for a handful of sequences.
        {"name": "linear_ragged_d4_5tok", "path": "linear", "codebook": "e8_d4", "out": 2056, "in": 1411,
         "tokens": 5, "bias": True, "qb_size": 0, "dtype": "fp16"},
        # Group scales at decode: the gate projection of an 8B model quantized in blocks of 128 rows.
        {"name": "linear_group_scales_d4_1tok", "path": "linear", "codebook": "e8_d4", "out": 14336, "in": 4096,
         "tokens": 1, "bias": False, "qb_size": 128, "dtype": "fp16"},
        # One decoder layer of a 7B model per decoded token: the step every single-user session repeats.
        {"name": "block_7b_d4_1tok", "path": "block", "codebook": "e8_d4", "hidden": 4096, "intermediate": 11008,
         "kv": 4096, "tokens": 1, "qb_size": 0, "dtype": "fp16"},
        # The same layer with the E8 codebook for a few sequences decoded together.
        {"name": "block_7b_e8_4tok", "path": "block", "codebook": "e8_lattice", "hidden": 4096, "intermediate": 11008,
         "kv": 4096, "tokens": 4, "qb_size": 0, "dtype": "fp16"},
        # A full decode batch of a small server.
        {"name": "block_7b_d4_16tok", "path": "block", "codebook": "e8_d4", "hidden": 4096, "intermediate": 11008,
         "kv": 4096, "tokens": 16, "qb_size": 0, "dtype": "fp16"},
        # A short chat prompt in a model that runs in bf16 (the module casts in and out).
        {"name": "block_7b_d4_100tok_bf16", "path": "block", "codebook": "e8_d4", "hidden": 4096,
         "intermediate": 11008, "kv": 4096, "tokens": 100, "qb_size": 0, "dtype": "bf16"},
        # A long prompt through an 8B model's layer with grouped-query heads and group scales.
        {"name": "block_8b_d4_2048tok_groups", "path": "block", "codebook": "e8_d4", "hidden": 4096,
         "intermediate": 14336, "kv": 1024, "tokens": 2048, "qb_size": 128, "dtype": "fp16"},
        # Reconstructing a weight for export, comparison or fine-tuning.
        {"name": "dequantize_11008x4096_e8", "path": "dequantize", "codebook": "e8_lattice", "out": 11008,
         "in": 4096, "qb_size": 0},
        # A whole 7B model: 512-token prompt, 128 greedy tokens, one sequence.
        {"name": "decode_7b_d4", "path": "decode", "codebook": "e8_d4", "hidden": 4096, "intermediate": 11008,
         "layers": 32, "heads": 32, "kv_heads": 32, "vocab": 32000, "batch": 1, "prompt": 512, "new_tokens": 128},
        # Eight sequences with a long context through layers of a 70B model (a pipeline stage of it).
        {"name": "decode_70b_layers_e8_8seq", "path": "decode", "codebook": "e8_lattice", "hidden": 8192,
         "intermediate": 28672, "layers": 4, "heads": 64, "kv_heads": 8, "vocab": 32000, "batch": 8,
         "prompt": 1024, "new_tokens": 24},
    ]


def _log_int(rng, lo: int, hi: int, step: int = 1) -> int:
    """A multiple of ``step`` in [lo, hi], uniform in the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(max(round(v / step) * step, lo), hi))


def _draw_linear(rng) -> dict:
    ragged = rng.random() < 0.4
    qb = 0 if ragged else rng.choice([0, 0, 128])
    out = _log_int(rng, 768, 14336, 8 if ragged else 128)
    inn = _log_int(rng, 768, 14336, 1 if ragged else 64)
    return {"path": "linear", "codebook": rng.choice(["e8_d4", "e8_lattice"]), "out": out, "in": inn,
            "tokens": rng.choice([1, 1, _log_int(rng, 2, 16)]), "bias": rng.random() < 0.3, "qb_size": qb,
            "dtype": rng.choice(["fp16", "fp16", "bf16"])}


def _draw_block(rng, prefill: bool) -> dict:
    hidden = _log_int(rng, 1024, 5120, 256)
    inter = _log_int(rng, 2 * hidden, 7 * hidden // 2, 128)
    tokens = _log_int(rng, 17, 4096) if prefill else rng.choice([1, _log_int(rng, 2, 16)])
    return {"path": "block", "codebook": rng.choice(["e8_d4", "e8_lattice"]), "hidden": hidden, "intermediate": inter,
            "kv": hidden // rng.choice([1, 2]), "tokens": tokens, "qb_size": rng.choice([0, 0, 128]) if prefill else 0,
            "dtype": rng.choice(["fp16", "fp16", "bf16"])}


def _draw_dequantize(rng) -> dict:
    return {"path": "dequantize", "codebook": rng.choice(["e8_d4", "e8_lattice"]), "out": _log_int(rng, 768, 14336, 128),
            "in": _log_int(rng, 768, 14336, rng.choice([1, 64])), "qb_size": rng.choice([0, 0, 128])}


def _draw_decode(rng) -> dict:
    heads = rng.choice([8, 16, 24, 32])
    hidden = 128 * heads
    return {"path": "decode", "codebook": rng.choice(["e8_d4", "e8_lattice"]), "hidden": hidden,
            "intermediate": _log_int(rng, 2 * hidden, 7 * hidden // 2, 128), "layers": rng.randint(2, 8), "heads": heads,
            "kv_heads": heads // rng.choice([1, 4]), "vocab": 32000, "batch": rng.choice([1, 1, 1, _log_int(rng, 2, 12)]),
            "prompt": _log_int(rng, 16, 1024), "new_tokens": rng.randint(16, 64)}


def draw(rng) -> dict:
    kind = rng.random()
    if kind < 0.30:
        return _draw_linear(rng)
    if kind < 0.52:
        return _draw_block(rng, prefill=False)
    if kind < 0.74:
        return _draw_block(rng, prefill=True)
    if kind < 0.82:
        return _draw_dequantize(rng)
    return _draw_decode(rng)


# ---- inputs ------------------------------------------------------------------------------------

def _codebook(kind: str) -> torch.Tensor:
    """The fp32 table on the GPU, made once per process: every layer of every model shares it."""
    if kind not in _tables:
        if kind == "e8_d4":
            table = E8D4Quantizer(radius=1.75).codes
        else:
            q = E8LatticeQuantizer(radius=1.6)
            q.remove_last()
            table = q.points
        _tables[kind] = table.to(DEVICE)
    return _tables[kind]


def _module(kind: str, out: int, inn: int, seed: int, bias: bool = False, qb_size: int = 0) -> EPTQLinear:
    qd = make_layer(out, inn, seed=seed, outlier_frac=CRITICAL_FRACTION, bias=bias, qb_size=qb_size or None, device=DEVICE)
    # row scales such that a unit-variance input gives outputs of order one, as trained layers do
    qd.g = (qd.g.float() / math.sqrt(inn)).to(torch.float16)
    return EPTQLinear.from_quantized_data(qd, _codebook(kind), kind)


def _block_shapes(case: dict) -> list:
    h, i, kv = case["hidden"], case["intermediate"], case["kv"]
    return [("q", h, h), ("k", kv, h), ("v", kv, h), ("o", h, h), ("gate", i, h), ("up", i, h), ("down", h, i)]


def _decode_shapes(case: dict) -> list:
    return _block_shapes(dict(case, kv=case["kv_heads"] * (case["hidden"] // case["heads"])))


def _engine(case: dict, seed: int) -> LlamaDecodeEngine:
    """A decoder stack with random weights.  The embedding carries through the residual stream and lm_head
    is a permutation of it, so that the picked token stands out from the others as in a trained model."""
    hidden, heads, vocab = case["hidden"], case["heads"], case["vocab"]
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    layers = []
    for n in range(case["layers"]):
        m = {name: _module(case["codebook"], out, inn, seed=seed + 101 * n + k)
             for k, (name, out, inn) in enumerate(_decode_shapes(case))}
        for name in ("o", "down"):
            m[name].g.mul_(0.25)
        norms = [(1 + 0.1 * torch.randn(hidden, generator=gen, device=DEVICE)).half() for _ in range(2)]
        layers.append(DecoderLayerWeights(m["q"], m["k"], m["v"], m["o"], m["gate"], m["up"], m["down"], *norms))
    embed = torch.randn((vocab, hidden), generator=gen, device=DEVICE)
    head = torch.empty_like(embed, dtype=torch.float16)
    head[torch.randperm(vocab, generator=gen, device=DEVICE)] = (0.02 * embed).half()
    head_dim = hidden // heads
    inv_freq = 1.0 / (10000.0 ** (torch.arange(0, head_dim, 2, device=DEVICE).float() / head_dim))
    return LlamaDecodeEngine(layers, embed.half(), torch.ones(hidden, dtype=torch.float16, device=DEVICE), head, inv_freq,
                             1e-5, head_dim, heads, case["kv_heads"], max_len=case["prompt"] + case["new_tokens"],
                             batch=case["batch"])


def prepare(case: dict, seed: int) -> dict:
    state = dict(case)
    if case["path"] == "decode":
        engine = _engine(case, seed)
        gen = torch.Generator(device=DEVICE).manual_seed(seed + 7)
        ids = torch.randint(0, case["vocab"], (case["batch"], case["prompt"]), generator=gen, device=DEVICE)
        engine.prefill(ids)                              # a server starts up warm: kernels loaded, token step captured
        engine.capture()
        state.update(engine=engine, ids=ids)
        return state
    if case["path"] == "block":
        state["layers"] = {name: _module(case["codebook"], out, inn, seed=seed + k, qb_size=case["qb_size"])
                           for k, (name, out, inn) in enumerate(_block_shapes(case))}
        dt = DTYPES[case["dtype"]]
        for k, (name, width) in enumerate((("x", case["hidden"]), ("att", case["hidden"]), ("act", case["intermediate"]))):
            state[name] = make_activations(case["tokens"], width, seed=seed + 50 + k, device=DEVICE).to(dt)
        return state
    state["layer"] = _module(case["codebook"], case["out"], case["in"], seed, case.get("bias", False), case["qb_size"])
    if case["path"] == "linear":
        state["x"] = make_activations(case["tokens"], case["in"], seed=seed + 50, device=DEVICE).to(DTYPES[case["dtype"]])
    return state


# ---- the call ----------------------------------------------------------------------------------

@torch.no_grad()
def run(state: dict):
    path = state["path"]
    if path == "linear":
        return state["layer"](state["x"])
    if path == "dequantize":
        return state["layer"].dequantize()
    if path == "decode":
        engine = state["engine"]
        tokens, _ = engine.decode(state["ids"], state["new_tokens"])
        return {"tokens": tokens, "keys": engine.k_cache, "values": engine.v_cache}
    m, x = state["layers"], state["x"]
    if state["tokens"] <= GROUP_MAX_TOKENS and not state["qb_size"]:
        q, k, v = forward_group([m["q"], m["k"], m["v"]], [x, x, x])
        o = m["o"](state["att"])
        gate, up = forward_group([m["gate"], m["up"]], [x, x])
        down = m["down"](state["act"])
    else:
        q, k, v, o = m["q"](x), m["k"](x), m["v"](x), m["o"](state["att"])
        gate, up, down = m["gate"](x), m["up"](x), m["down"](state["act"])
    return [q, k, v, o, gate, up, down]


# ---- what a pass cannot do without -------------------------------------------------------------

def _weight_bytes(out: int, inn: int, qb_size: int = 0, bias: bool = False) -> float:
    blocks = out // 8 * inn
    return 2 * blocks + 16 * CRITICAL_FRACTION * blocks + 2 * out + 2 * inn + (2 * out if bias else 0) \
        + (2 * (out // qb_size) * inn if qb_size else 0)


def _linear_work(out: int, inn: int, tokens: int, qb_size: int = 0, bias: bool = False):
    return _weight_bytes(out, inn, qb_size, bias) + 2 * tokens * (inn + out), 2.0 * tokens * out * inn


def _table_bytes(kind: str) -> int:
    return 2 * 2048 if kind == "e8_d4" else 2 * 8 * 65535


def work(case: dict) -> dict:
    nbytes, flops = float(_table_bytes(case["codebook"])), 0.0
    if case["path"] == "linear":
        b, f = _linear_work(case["out"], case["in"], case["tokens"], case["qb_size"], case["bias"])
        return {"bytes": nbytes + b, "flops": f}
    if case["path"] == "dequantize":
        return {"bytes": nbytes + _weight_bytes(case["out"], case["in"], case["qb_size"]) + 2 * case["out"] * case["in"],
                "flops": 3.0 * case["out"] * case["in"]}
    if case["path"] == "block":
        for _, out, inn in _block_shapes(case):
            b, f = _linear_work(out, inn, case["tokens"], case["qb_size"])
            nbytes, flops = nbytes + b, flops + f
        return {"bytes": nbytes, "flops": flops}
    B, T, steps, L = case["batch"], case["prompt"], case["new_tokens"] - 1, case["layers"]
    kv = case["kv_heads"] * (case["hidden"] // case["heads"])
    head_bytes, head_flops = 2.0 * case["vocab"] * case["hidden"], 2.0 * B * case["vocab"] * case["hidden"]
    for _, out, inn in _decode_shapes(case):
        b, f = _linear_work(out, inn, B * T)
        nbytes, flops = nbytes + L * b, flops + L * f
        b, f = _linear_work(out, inn, B)
        nbytes, flops = nbytes + steps * L * b, flops + steps * L * f
    flops += L * B * 2.0 * T * T * case["hidden"]                         # causal attention over the prompt
    nbytes += L * B * 4.0 * T * kv
    for s in range(steps):
        nbytes += L * B * 4.0 * (T + s + 1) * kv
        flops += L * B * 4.0 * (T + s + 1) * case["hidden"]
    return {"bytes": nbytes + (steps + 1) * head_bytes, "flops": flops + (steps + 1) * head_flops}


def tolerance(case: dict):
    if case["path"] == "dequantize":
        return "exact"
    if case["path"] == "decode":
        # fp16 roundings that add up along the residual stream of the stack
        return {"rel": 1e-2, "max": 0.2, "differ": 0.01}
    if case["dtype"] == "bf16":
        return {"rel": 1e-2, "max": 2e-2}
    return {"rel": 1e-3, "max": 1e-2}                                       # fp16 weights, inputs and outputs
