"""The work this framework is used for, as cases that can be timed and compared.

A case is a dict of plain values; `prepare` makes what a user's program holds before the call, `run` is one
pass through the public entry points, `work` is what that pass cannot do without.  The kinds:

  projection  one INT4 projection (q / k / v / o, an output head): mlx_affine_qmv or mlx_affine_residual_qmv
  mlp         the fused INT4 MLP with the residual, through an executor bound to its weights
  dense       the bf16 small-batch projection or SwiGLU whose rows do not depend on the batch
  norm        residual add + RMSNorm
  attention   one decode query per sequence and head over an in-place KV cache
  prefill     a prompt through a patched model into its KV caches
  decode      tokens of a batch through a patched model, one replayed CUDA graph per token

Widths come from the shapes the tests and the benchmark use (hidden 512 to 5120, MLP 2.5 to 6 times as wide,
an output head of 128256) and are multiples of the quantisation group, 64; row counts run from one decode row
to a prompt of two thousand.
"""

from __future__ import annotations

import math

import torch

from metile_b200 import backends
from metile_b200.integrations import blocks
from metile_b200.integrations.graphed import GraphedDecoder
from metile_b200.integrations.torch_lm import apply_metile_to_torch_lm

GROUP = 64
BYTES_PER_WEIGHT = 0.5 + 2 * 2 / GROUP  # a nibble, and a bf16 scale and bias per group
EPS = 1e-6
ROPE_THETA = 1e6
DECODE_STEPS = 8

# No drawn case costs more than the largest listed one.
MOST_FLOPS = 2.0 * 2000 * 3 * 2048 * 8192
MOST_WEIGHTS = 3 * 5120 * 27648
MOST_KV_BYTES = 512 << 20


def listed():
    return [
        # The smallest call: one decode row through one projection of a small model (up to 8960 wide).
        {"name": "projection_1", "kind": "projection", "rows": 1, "k": 1536, "n": 8960, "residual": False},
        # The output head of a model with a large vocabulary, once per generated token.
        {"name": "projection_head", "kind": "projection", "rows": 1, "k": 2048, "n": 128256, "residual": False},
        # An attention output projection with its residual for an odd number of concurrent sequences.
        {"name": "projection_37", "kind": "projection", "rows": 37, "k": 1536, "n": 1536, "residual": True},
        # Single-stream decoding at the Llama-3.2-1B shape: the latency case.
        {"name": "mlp_1", "kind": "mlp", "rows": 1, "hidden": 2048, "inter": 8192},
        # A handful of concurrent sequences (or a speculative draft) at the same shape.
        {"name": "mlp_8", "kind": "mlp", "rows": 8, "hidden": 2048, "inter": 8192},
        # A full decode batch at the Qwen2.5-32B shape, one GPU: the most weights a call streams.
        {"name": "mlp_128", "kind": "mlp", "rows": 128, "hidden": 5120, "inter": 27648},
        # The MLP of a long prompt (not a whole number of tiles): the largest call.
        {"name": "mlp_prompt", "kind": "mlp", "rows": 2000, "hidden": 2048, "inter": 8192},
        # bf16 weights at a small decode batch.
        {"name": "dense_16", "kind": "dense", "rows": 16, "k": 1536, "n": 8960, "swiglu": False},
        # Residual add + RMSNorm over a prompt.
        {"name": "norm_512", "kind": "norm", "rows": 512, "width": 4096},
        # Decode attention of a Qwen2.5-1.5B block: 16 sequences of 2048 tokens.
        {"name": "attention_16", "kind": "attention", "batch": 16, "kv_heads": 2, "group": 6, "dim": 128,
         "tokens": 2048, "ragged": False},
        # A prompt through four Qwen2.5-1.5B-shaped blocks and a 32768-entry head.
        {"name": "prefill_512", "kind": "prefill", "batch": 1, "prompt": 512, "layers": 4, "hidden": 1536,
         "inter": 8960, "kv_heads": 2, "group": 6, "dim": 128, "vocab": 32768},
        # Eight tokens of sixteen sequences at a KV length of 2048 through the same model.
        {"name": "decode_16", "kind": "decode", "batch": 16, "prompt": 2040, "layers": 4, "hidden": 1536,
         "inter": 8960, "kv_heads": 2, "group": 6, "dim": 128, "vocab": 32768},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _width(rng, low, high, step=GROUP):
    return max(low, min(high, _log_int(rng, low, high) // step * step))


def draw(rng):
    kind = rng.choice(("projection", "projection", "projection", "mlp", "mlp", "mlp", "mlp", "dense", "norm",
                       "attention", "prefill", "decode"))
    if kind == "projection":
        k = _width(rng, 512, 8192)
        n = _log_int(rng, 128, 131072)
        rows = 1 if rng.random() < 0.4 else _log_int(rng, 2, 2000)  # single-stream decoding is the common call
        return {"kind": kind, "rows": max(1, min(rows, int(MOST_FLOPS / (2.0 * k * n)))), "k": k, "n": n,
                "residual": rng.random() < 0.5}
    if kind == "mlp":
        hidden = _width(rng, 512, 5120)
        inter = min(int(hidden * rng.uniform(2.5, 6.0)), MOST_WEIGHTS // (3 * hidden)) // GROUP * GROUP
        rows = 1 if rng.random() < 0.2 else _log_int(rng, 2, 2000)
        return {"kind": kind, "rows": max(1, min(rows, int(MOST_FLOPS / (6.0 * hidden * inter)))), "hidden": hidden,
                "inter": inter}
    if kind == "dense":
        return {"kind": kind, "rows": _log_int(rng, 1, 128), "k": _width(rng, 512, 4096, 128),
                "n": _log_int(rng, 256, 12000), "swiglu": rng.random() < 0.5}
    if kind == "norm":
        return {"kind": kind, "rows": _log_int(rng, 1, 4096), "width": _width(rng, 512, 8192)}
    kv_heads, group, dim = rng.choice((1, 2, 4, 8)), rng.randint(1, 8), rng.choice((64, 128))
    if kind == "attention":
        batch, tokens = _log_int(rng, 1, 64), _log_int(rng, 64, 8192)
        return {"kind": kind, "batch": batch, "kv_heads": kv_heads, "group": group, "dim": dim,
                "tokens": max(64, min(tokens, MOST_KV_BYTES // (batch * kv_heads * dim * 4))),
                "ragged": rng.random() < 0.5}
    kv_heads = rng.choice((1, 2, 4))
    group = max(1, min(8, 2048 // (kv_heads * dim)))
    hidden = _width(rng, 512, 2048)
    model = {"layers": rng.randint(1, 4), "hidden": hidden, "inter": int(hidden * rng.uniform(2.5, 5.0)) // GROUP * GROUP,
             "kv_heads": kv_heads, "group": group, "dim": dim, "vocab": _log_int(rng, 4096, 32768)}
    if kind == "prefill":
        return {"kind": kind, "batch": 1, "prompt": _log_int(rng, 32, 1024), **model}
    return {"kind": kind, "batch": _log_int(rng, 1, 16), "prompt": _log_int(rng, 64, 2040), **model}


# ---- inputs ----------------------------------------------------------------------------------------------


class _Maker:
    """Seeded tensors on the GPU with the distributions the benchmark names."""

    def __init__(self, seed):
        self.device = torch.device("cuda")
        self.generator = torch.Generator(device=self.device).manual_seed(int(seed))

    def normal(self, *shape, std=1.0, mean=0.0):
        values = torch.randn(shape, generator=self.generator, device=self.device, dtype=torch.float32)
        return (values * std + mean).to(torch.bfloat16)

    def affine(self, n, k):
        """q uniform 0..15; scale ~ U(0.002, 0.02); bias = -8 scale + N(0, 1e-3)."""
        words = torch.randint(-2**31, 2**31, (n, k // 8), generator=self.generator, device=self.device, dtype=torch.int32)
        uniform = torch.rand((n, k // GROUP), generator=self.generator, device=self.device)
        scales = (uniform * 0.018 + 0.002).to(torch.bfloat16)
        noise = torch.randn((n, k // GROUP), generator=self.generator, device=self.device) * 1e-3
        return words.view(torch.uint32), scales, (-8.0 * scales.float() + noise).to(torch.bfloat16)

    def tokens(self, vocab, *shape):
        return torch.randint(0, vocab, shape, generator=self.generator, device=self.device)

    def model(self, case):
        """A random-init decoder-only model with 4-bit projections, patched with every feature."""
        hidden, inter, dim = case["hidden"], case["inter"], case["dim"]
        kv_heads, heads = case["kv_heads"], case["kv_heads"] * case["group"]

        def linear(fan_in, fan_out):
            return blocks.QuantizedLinear(*self.affine(fan_out, fan_in))

        def norm():
            return blocks.RMSNorm(self.normal(hidden, std=0.02, mean=1.0), EPS)

        layers = []
        for _ in range(case["layers"]):
            attention = blocks.Attention(linear(hidden, heads * dim), linear(hidden, kv_heads * dim),
                                         linear(hidden, kv_heads * dim), linear(heads * dim, hidden), heads, kv_heads,
                                         dim, ROPE_THETA)
            mlp = blocks.GatedMLP(linear(hidden, inter), linear(hidden, inter), linear(inter, hidden))
            layers.append(blocks.DecoderBlock(norm(), attention, norm(), mlp))
        embedding = torch.nn.Embedding.from_pretrained(self.normal(case["vocab"], hidden), freeze=True)
        model = blocks.TinyCausalLM(embedding, layers, norm(), linear(hidden, case["vocab"]), case["vocab"])
        return model, apply_metile_to_torch_lm(model, attention=True)


def _lengths(case):
    """Tokens in use per sequence of an attention case: all of them, or a spread from an eighth up."""
    batch, tokens = case["batch"], case["tokens"]
    if not case["ragged"]:
        return [tokens] * batch
    low = max(1, tokens // 8)
    return [low + (tokens - low) * (b * 5 % batch) // max(1, batch - 1) for b in range(batch)]


def prepare(case, seed):
    make, kind = _Maker(seed), case["kind"]
    if kind == "projection":
        return {"kind": kind, "x": make.normal(case["rows"], case["k"]), "weight": make.affine(case["n"], case["k"]),
                "residual": make.normal(case["rows"], case["n"]) if case["residual"] else None}
    if kind == "mlp":
        hidden, inter = case["hidden"], case["inter"]
        x, residual = make.normal(case["rows"], hidden), make.normal(case["rows"], hidden)
        gate, up, down = make.affine(inter, hidden), make.affine(inter, hidden), make.affine(hidden, inter)
        return {"kind": kind, "x": x, "residual": residual,
                "execute": backends.mlx_affine_mlp_executor(x, *gate, *up, *down, residual)}
    if kind == "dense":
        weights = [make.normal(case["n"], case["k"], std=0.02) for _ in range(2 if case["swiglu"] else 1)]
        return {"kind": kind, "x": make.normal(case["rows"], case["k"]), "weights": weights,
                "residual": None if case["swiglu"] else make.normal(case["rows"], case["n"])}
    if kind == "norm":
        return {"kind": kind, "x": make.normal(case["rows"], case["width"]),
                "residual": make.normal(case["rows"], case["width"]),
                "weight": make.normal(case["width"], std=0.02, mean=1.0)}
    if kind == "attention":
        batch, kv_heads, dim, tokens = case["batch"], case["kv_heads"], case["dim"], case["tokens"]
        lengths = torch.tensor(_lengths(case), dtype=torch.int32, device=make.device) if case["ragged"] else None
        return {"kind": kind, "query": make.normal(batch, kv_heads * case["group"], 1, dim),
                "keys": make.normal(batch, kv_heads, tokens, dim), "values": make.normal(batch, kv_heads, tokens, dim),
                "lengths": lengths, "scale": dim ** -0.5}
    # A patched model with its caches.  For decode the prompt has been read and the step's graph captured.
    model, patch = make.model(case)
    prompt = make.tokens(case["vocab"], case["batch"], case["prompt"])
    decoder = GraphedDecoder(model, batch=case["batch"], capacity=case["prompt"] + DECODE_STEPS)
    state = {"kind": kind, "decoder": decoder, "patch": patch, "prompt": prompt}
    if kind == "decode":
        state["next"] = list(make.tokens(case["vocab"], DECODE_STEPS, case["batch"]))
        state["length"] = case["prompt"]
        decoder.stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(decoder.stream):
            decoder.prefill(prompt)
            decoder.step(state["next"][0])
    return state


# ---- one pass --------------------------------------------------------------------------------------------


def run(state):
    kind = state["kind"]
    if kind == "projection":
        if state["residual"] is None:
            return backends.mlx_affine_qmv(state["x"], *state["weight"])
        return backends.mlx_affine_residual_qmv(state["x"], *state["weight"], state["residual"])
    if kind == "mlp":
        return state["execute"](state["x"], state["residual"])
    if kind == "dense":
        if len(state["weights"]) == 2:
            return backends.mlx_dense_swiglu(state["x"], *state["weights"])
        return backends.mlx_dense_residual_qmv(state["x"], state["weights"][0], state["residual"])
    if kind == "norm":
        return backends.mlx_add_rms_norm(state["x"], state["residual"], state["weight"], EPS)
    if kind == "attention":
        return backends.mlx_attention_decode(state["query"], state["keys"], state["values"], scale=state["scale"],
                                             lengths=state["lengths"])
    decoder = state["decoder"]
    if kind == "prefill":
        logits = decoder.prefill(state["prompt"])
    else:
        # Another continuation of the same prompt, tokens chosen by the caller.  The serving loop stays on the
        # decoder's own stream, so that its resets, token choices and copies are ordered with the replays; the
        # caller's stream hands the tokens over and takes the logits back.
        caller = torch.cuda.current_stream()
        decoder.stream.wait_stream(caller)
        with torch.cuda.stream(decoder.stream):
            for cache in decoder.cache:
                cache.reset(state["length"])
            logits = [decoder.step(token).clone() for token in state["next"]]
        caller.wait_stream(decoder.stream)
    return {"logits": logits, "keys": [cache.keys for cache in decoder.cache],
            "values": [cache.values for cache in decoder.cache]}


# ---- what a pass cannot do without -----------------------------------------------------------------------


def work(case):
    kind = case["kind"]
    if kind == "projection":
        rows, k, n = case["rows"], case["k"], case["n"]
        return {"bytes": n * k * BYTES_PER_WEIGHT + 2 * rows * (k + n * (2 if case["residual"] else 1)),
                "flops": 2.0 * rows * k * n}
    if kind == "mlp":
        rows, hidden, inter = case["rows"], case["hidden"], case["inter"]
        return {"bytes": 3 * hidden * inter * BYTES_PER_WEIGHT + 2 * rows * 3 * hidden,
                "flops": 6.0 * rows * hidden * inter}
    if kind == "dense":
        rows, k, n, streams = case["rows"], case["k"], case["n"], 2 if case["swiglu"] else 1
        return {"bytes": 2 * (streams * n * k + rows * (k + n * (1 if case["swiglu"] else 2))),
                "flops": 2.0 * streams * rows * k * n}
    if kind == "norm":
        values = case["rows"] * case["width"]
        return {"bytes": 2 * (4 * values + case["width"]), "flops": 6.0 * values}
    heads, dim = case["kv_heads"] * case["group"], case["dim"]
    if kind == "attention":
        used = sum(_lengths(case))
        return {"bytes": 2 * (2 * used * case["kv_heads"] * dim + 2 * case["batch"] * heads * dim),
                "flops": 4.0 * used * heads * dim}
    # The model: every weight once per pass (prefill) or per token (decode), the caches as attention reads them.
    hidden, layers, batch, prompt = case["hidden"], case["layers"], case["batch"], case["prompt"]
    per_layer = hidden * (2 * heads + 2 * case["kv_heads"]) * dim + 3 * hidden * case["inter"]
    weights = layers * per_layer + hidden * case["vocab"]
    kv_row = 2 * 2 * layers * case["kv_heads"] * dim  # bytes of one token's keys and values
    if kind == "prefill":
        tokens = batch * prompt
        # Of the head's rows only the last position's logits are returned.
        return {"bytes": weights * BYTES_PER_WEIGHT + tokens * (kv_row + 2 * hidden) + 4 * batch * case["vocab"],
                "flops": 2.0 * (tokens * layers * per_layer + batch * hidden * case["vocab"])
                + 2.0 * layers * batch * heads * dim * prompt * prompt}
    read = sum(prompt + 1 + step for step in range(DECODE_STEPS)) * batch
    return {"bytes": DECODE_STEPS * (weights * BYTES_PER_WEIGHT + 4 * batch * case["vocab"]) + read * kv_row,
            "flops": 2.0 * DECODE_STEPS * batch * weights + 4.0 * read * layers * heads * dim}


def tolerance(case):
    # bf16 results of fp32 sums.  The dense rows keep one fp32 order; whole models compose some thirty bf16
    # roundings per layer pair.
    if case["kind"] == "dense":
        return {"rel": 5e-3, "max": 0.05}
    if case["kind"] in ("prefill", "decode"):
        return {"rel": 2e-2, "max": 0.3}
    return {"rel": 1e-2, "max": 0.1}
