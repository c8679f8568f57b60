"""The work this package is used for, as cases that can be timed: the quantized linear layers a
loaded model calls (one token, a few, a chunk of a prompt, a whole prompt; int4 and int8, bf16 and
f16), the quantizers that make their weights, and whole decode steps of the Llama-shaped decoder.

`listed()` are fixed cases, `draw(rng)` gives others of the same ranges.  `prepare` makes what a
program holds before the call (weights, activations, a decoder with its captured step), `run` is
one pass through the public entry points, `work` what a pass cannot do without.
"""

from __future__ import annotations

import math
import random
from dataclasses import replace

import torch

from linnet_b200 import decoder, int4, kernels, quant, quantized

_DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
_MAX_FLOPS = 2.0 * 2048 * 4096 * 28672  # the fused gate|up projection of a 2048-token prompt


def listed() -> list[dict]:
    return [
        # One token through the attention output projection of an 8B-shaped model: the smallest
        # call there is, what the latency of a call shows in.
        {"name": "int4_1x4096x4096", "op": "int4", "rows": 1, "depth": 4096, "width": 4096, "group": 128, "dtype": "bf16"},
        # Sixteen sequences decoding together through the down projection.
        {"name": "int4_16x14336x4096", "op": "int4", "rows": 16, "depth": 14336, "width": 4096, "group": 128, "dtype": "bf16"},
        # A large decode batch (or the tail of a prompt), not a whole number of tiles, through gate|up.
        {"name": "int4_100x4096x28672", "op": "int4", "rows": 100, "depth": 4096, "width": 28672, "group": 128, "dtype": "bf16"},
        # A 2048-token prompt through gate|up: the largest product.
        {"name": "int4_2048x4096x28672", "op": "int4", "rows": 2048, "depth": 4096, "width": 28672, "group": 128, "dtype": "bf16"},
        # A chunk of a prompt in f16 with groups of 32, as imported GPTQ checkpoints come.
        {"name": "int4_f16_g32_333x4096x4096", "op": "int4", "rows": 333, "depth": 4096, "width": 4096, "group": 32, "dtype": "f16"},
        # int8 weights, one scale a row: one token.
        {"name": "int8_1x4096x14336", "op": "int8", "rows": 1, "depth": 4096, "width": 14336, "group": 0, "rounded": False, "dtype": "bf16"},
        # int8 weights, one scale a row: a chunk of a prompt with 16-bit activations.
        {"name": "int8_200x4096x14336", "op": "int8", "rows": 200, "depth": 4096, "width": 14336, "group": 0, "rounded": False, "dtype": "bf16"},
        # int8 weights and activations (rounded per row on the way in): a 2048-token prompt.
        {"name": "w8a8_2048x4096x14336", "op": "int8", "rows": 2048, "depth": 4096, "width": 14336, "group": 0, "rounded": True, "dtype": "bf16"},
        # Packing a 70B-shaped up projection to 4 bits while a checkpoint is converted.
        {"name": "quantize4_28672x8192", "op": "quantize", "bits": 4, "width": 28672, "depth": 8192, "group": 128, "dtype": "bf16"},
        # One decode step of a stack of 8B-shaped layers with output head, one sequence at full
        # context.  (Four layers: through more of them, bf16 roundings in another order grow to
        # more than results can be compared by.)
        {"name": "decode_1", "op": "decode", "rows": 1, "layers": 4, "hidden": 4096, "vocab": 32000, "context": 2048},
        # The same for small and large serving batches of sequences of different lengths.
        {"name": "decode_8", "op": "decode", "rows": 8, "layers": 4, "hidden": 4096, "vocab": 32000, "context": 2048},
        {"name": "decode_64", "op": "decode", "rows": 64, "layers": 4, "hidden": 4096, "vocab": 32000, "context": 2048},
    ]


def _log(rng: random.Random, low: float, high: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng: random.Random) -> dict:
    op = rng.choice(["int4", "int4", "int4", "int8", "int8", "quantize", "decode"])
    if op == "decode":
        return {"op": op, "rows": _log(rng, 1, 64), "layers": rng.randint(2, 4), "hidden": rng.choice([1024, 2048, 4096]),
                "vocab": 32000, "context": rng.randint(128, 2048)}
    if op == "quantize":
        bits = rng.choice([4, 8])
        depth = 128 * _log(rng, 8, 112)
        group = rng.choice([32, 64, 128, 128, depth if bits == 8 else 128])
        width = min(_log(rng, 512, 28672), 28672 * 8192 // depth)
        return {"op": op, "bits": bits, "width": width, "depth": depth, "group": group, "dtype": rng.choice(["bf16", "bf16", "f32"])}
    rows = 1 if rng.random() < 0.2 else _log(rng, 1, 2048)
    depth = 128 * _log(rng, 8, 112)  # 1024 .. 14336 inputs
    width = _log(rng, 1024, 28672)
    if rng.random() < 0.8:           # most layers' widths are round, some (an added token, a classifier) are not
        width = max(1, width // 64) * 64
    width = min(width, int(_MAX_FLOPS / (2.0 * rows * depth)), 14336 * 8192 // depth)
    if op == "int4":
        return {"op": op, "rows": rows, "depth": depth, "width": width, "group": rng.choice([32, 64, 128, 128, 128]),
                "dtype": rng.choice(["bf16", "bf16", "f16"])}
    group = rng.choice([0, 0, 128])
    return {"op": op, "rows": rows, "depth": depth, "width": width, "group": group,
            "rounded": group == 0 and rng.random() < 0.3, "dtype": rng.choice(["bf16", "bf16", "f16"])}


# ---- what a program holds before the call ---------------------------------------------------


def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(shape: tuple[int, ...], std: float, dtype: torch.dtype, gen: torch.Generator) -> torch.Tensor:
    return torch.empty(shape, device="cuda", dtype=dtype).normal_(0.0, std, generator=gen)


def _config(case: dict) -> decoder.DecoderConfig:
    hidden = case["hidden"]  # the 8B proportions: heads of 128, four to a KV head, an MLP of 3.5 x hidden
    return replace(decoder.DecoderConfig.llama31_8b(), layers=case["layers"], hidden=hidden, heads=hidden // 128,
                   kv_heads=hidden // 512, mlp=hidden * 7 // 2, vocab=case["vocab"])


def _positions(case: dict) -> list[int]:
    """The first sequence at the end of its context, the others spread over its second half."""
    context = case["context"]
    return [context - 1 - (i * 37) % max(1, context // 2) for i in range(case["rows"])]


def _prepare_decode(case: dict, seed: int) -> dict:
    device, cfg, batch = torch.device("cuda"), _config(case), case["rows"]
    gen = _generator(seed)
    model = decoder.build_random(cfg, torch.device("cuda", torch.cuda.current_device()), rank=0, tp=1, seed=seed,
                                 linear=kernels.int4_linear, quantize=quant.quantize_int4_groups)
    model.allocate_cache(batch, gen)
    # the layers' caches as slices of one allocation for K and one for V
    keys, values = torch.stack(model.cache_k), torch.stack(model.cache_v)
    model.cache_k, model.cache_v = list(keys.unbind(0)), list(values.unbind(0))
    tokens = torch.randint(0, cfg.vocab, (batch,), device=device, generator=gen)
    fed = tokens.clone()  # the buffer the captured step reads its token ids from
    positions = torch.tensor(_positions(case), device=device, dtype=torch.long)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        model.step(fed, positions)
    torch.cuda.current_stream().wait_stream(stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        logits = model.step(fed, positions)
    return {"op": "decode", "model": model, "graph": graph, "fed": fed, "tokens": tokens, "positions": positions,
            "out": {"logits": logits, "keys": keys, "values": values}}


def prepare(case: dict, seed: int) -> dict:
    op = case["op"]
    if op == "decode":
        return _prepare_decode(case, seed)
    gen, dtype = _generator(seed), _DTYPES[case["dtype"]]
    if op == "quantize":
        return {"op": op, "bits": case["bits"], "group": case["group"],
                "weight": _normal((case["width"], case["depth"]), 0.015, dtype, gen)}
    weight = _normal((case["width"], case["depth"]), 0.02, torch.bfloat16, gen)
    x = _normal((case["rows"], case["depth"]), 1.0, dtype, gen)
    if op == "int4":
        packed, _, zero, scale = quant.quantize_int4_groups(weight, case["group"], scale_dtype=case["dtype"])
        return {"op": op, "x": x, "raw": packed, "scale": scale, "zero": zero, "packed": int4._int4_pack(packed, scale, zero)}
    group = case["group"]
    q, scale = quant.quantize_int8_groups(weight, group or case["depth"], "f32")
    if group:
        return {"op": "int8_group", "x": x, "operands": quantized.int8_group_operands(q, scale)}
    return {"op": op, "x": x, "operands": quantized.int8_operands(q, scale, int(case["rounded"]))}


# ---- one pass ---------------------------------------------------------------------------------


def run(state: dict):
    op = state["op"]
    if op == "int4":
        return int4._int4_linear(state["x"], state["packed"], None, state["raw"], state["scale"], state["zero"])
    if op == "int8":
        return quantized.int8_linear(state["x"], state["operands"], None)
    if op == "int8_group":
        return quantized.int8_group_linear(state["x"], state["operands"], None)
    if op == "quantize":
        if state["bits"] == 4:
            return quant.quantize_int4_groups(state["weight"], state["group"], scale_dtype="bf16")
        return quant.quantize_int8_groups(state["weight"], state["group"], "f32")
    state["fed"].copy_(state["tokens"])
    state["graph"].replay()
    return state["out"]


# ---- what a pass cannot do without --------------------------------------------------------------


def work(case: dict) -> dict:
    op = case["op"]
    if op == "decode":
        cfg, batch = _config(case), case["rows"]
        keys = sum(p + 1 for p in _positions(case))
        row = cfg.kv_heads * cfg.head_dim * 2 * 2  # bytes of K and V of one position
        weights = cfg.int4_elements()
        return {"bytes": weights * (0.5 + 3.0 / cfg.group) + cfg.layers * row * (keys + batch) + 2.0 * batch * cfg.vocab,
                "flops": 2.0 * batch * weights + 4.0 * cfg.layers * cfg.heads * cfg.head_dim * keys}
    width, depth, group = case["width"], case["depth"], case["group"]
    size = 4 if case["dtype"] == "f32" else 2
    if op == "quantize":
        if case["bits"] == 4:  # packed nibbles; scale in f32 and as stored, zero point
            out = 0.5 + (4 + 2 + 1) / group
        else:
            out = 1.0 + 4 / group
        return {"bytes": width * depth * (size + out), "flops": 0.0}
    rows = case["rows"]
    if op == "int4":
        weights = width * depth * (0.5 + 3.0 / group)
    else:
        weights = width * depth + 4.0 * width * (depth // group if group else 1)
    return {"bytes": weights + 2.0 * rows * (depth + width), "flops": 2.0 * rows * depth * width}


def tolerance(case: dict):
    op = case["op"]
    if op == "quantize":
        return "exact"  # the levels, scales and zero points are defined bit for bit
    if op == "decode":
        # 16-bit roundings that fall elsewhere (library products, unfused glue, weights rounded or
        # not) move the logits by 0.008 to 0.018 through two to four layers: twice that is more
        # than a comparison can use
        return {"rel": 0.03}
    # against the product in f64, with the weights rounded to the activation type (as the CPU route
    # has them) or not: 0.0016 to 0.0023 in bf16, 0.0002 to 0.00028 in f16
    return {"rel": 0.009} if case["dtype"] == "bf16" else {"rel": 0.0012}
