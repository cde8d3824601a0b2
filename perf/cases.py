"""The work that is timed: what a user of this package has it do, through its public entry points.

A quantization run goes through a model block by block.  Every linear layer gets a `GPTQ` handle;
`update` folds each calibration batch into the handle's Hessian, one of the `quantize` calls turns
the layer into 4-bit codes and scales, and the results are dequantized back into the block, measured
against the Hessian and packed into int32 words.  The cases follow these steps, each with the whole
path a user pays for: handles are new in every pass, calibration batches come in several pieces of
uneven length, and what comes back is everything the caller gets (codes, scales, zero points, words
and the Hessian left in the handle).

Weights are 0.02 N(0,1); activations are N(0,1) with one LogNormal(0,1) factor per input channel,
which gives the outlier channels that make the method differ from plain rounding.
"""
import math

import torch
import torch.nn as nn

from moe_quant_b200 import GPTQ, pack_weight, quant_utils
from moe_quant_b200.gptq import quantize_many, quantize_shared

BITS = 4
REL_DAMP = 1e-2
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def listed():
    return [
        # the smallest call there is: the first few tokens a narrow layer sees
        {"name": "calibrate_first_tokens", "kind": "calibrate", "cols": 512, "tokens": 37, "batches": 1, "dtype": "bf16"},
        # a routed expert: of every calibration sequence only some hundred tokens reach it, so its
        # wide Hessian takes many short updates
        {"name": "calibrate_expert", "kind": "calibrate", "cols": 7168, "tokens": 1011, "batches": 8, "dtype": "bf16"},
        # a layer that sees all tokens: whole sequences of 4096
        {"name": "calibrate_shared", "kind": "calibrate", "cols": 7168, "tokens": 8192, "batches": 2, "dtype": "bf16"},
        # a small fp32 layer with narrow groups, sizes that fill no tile
        {"name": "quantize_small_fp32", "kind": "quantize", "rows": 500, "cols": 1056, "group": 32, "tokens": 1500, "batches": 2,
         "dtype": "fp32"},
        # gate_proj of a routed expert, the layer most of a model's layers look like
        {"name": "quantize_gate_proj", "kind": "quantize", "rows": 2048, "cols": 7168, "group": 128, "tokens": 4096, "batches": 4,
         "dtype": "bf16"},
        # down_proj of a routed expert, with its packed words, as a checkpoint writer wants it
        {"name": "quantize_packed_down_proj", "kind": "quantize_packed", "rows": 7168, "cols": 2048, "group": 64, "tokens": 8192,
         "batches": 4, "dtype": "fp16"},
        # the expert loop of a block: gate/up pairs that share a Hessian, and down projections
        {"name": "quantize_experts", "kind": "experts", "experts": 4, "hidden": 7168, "inner": 2048, "group": 128, "tokens": 20480,
         "batches": 4, "tied": True, "dtype": "bf16"},
        # the attention projections of a block, from the narrow latent ones to the widest layer of the model
        {"name": "quantize_attention", "kind": "attention", "hidden": 7168, "q_rank": 1536, "kv_rank": 512, "heads": 128, "group": 128,
         "tokens": 20480, "batches": 5, "dtype": "bf16"},
        # the two options of the command line: columns ordered by activation, scales searched by MSE
        {"name": "quantize_act_order", "kind": "act_order", "rows": 2048, "cols": 7168, "group": 128, "tokens": 8192, "batches": 2,
         "dtype": "bf16"},
        {"name": "quantize_mse_scales", "kind": "mse", "rows": 7168, "cols": 2048, "group": 128, "tokens": 4096, "batches": 2,
         "dtype": "bf16"},
        # the logged error of a quantized layer
        {"name": "error_metric", "kind": "error", "rows": 2048, "cols": 7168, "group": 128, "dtype": "bf16"},
        # what happens to a layer's codes afterwards: back into the block, and packed for the checkpoint
        {"name": "dequantize_and_pack", "kind": "export", "rows": 7168, "cols": 2048, "group": 128, "dtype": "bf16"},
    ]


# ---------------------------------------------------------------- drawn cases
def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cols(rng, lo, hi, step=8):
    """A layer width: mostly whole 128-column tiles, often any multiple of 8."""
    c = _log_int(rng, lo, hi)
    a = 128 if rng.random() < 0.6 else step
    return max(lo, c // a * a)


def _group(rng, cols):
    """A group size that divides the width; 0 is one group per row."""
    fits = [g for g in (32, 64, 128) if cols % g == 0]
    return rng.choice(fits + [0]) if fits else 0


def _draw_once(rng):
    kind = rng.choice(["calibrate", "calibrate", "quantize", "quantize", "quantize_packed", "experts", "attention", "act_order", "mse",
                       "error", "export"])
    dtype = rng.choice(["bf16", "bf16", "fp16", "fp32"])
    case = {"kind": kind}
    if kind == "calibrate":
        cols = _cols(rng, 256, 16384, rng.choice([1, 8]))
        case.update(cols=cols, tokens=_log_int(rng, 1, 16384), dtype=dtype)
    elif kind == "experts":
        hidden, inner = _cols(rng, 512, 7168, 32), _cols(rng, 512, 2048, 32)
        case.update(experts=rng.randint(2, 4), hidden=hidden, inner=inner, group=rng.choice([32, 64, 128]), tied=rng.random() < 0.5,
                    dtype=dtype)
        if hidden % case["group"] or inner % case["group"]:
            case["group"] = 32
        case["tokens"] = case["experts"] * _log_int(rng, 0.7 * hidden, 8000)
    elif kind == "attention":
        case.update(hidden=_cols(rng, 1024, 7168, 128), q_rank=128 * rng.randint(3, 12), kv_rank=128 * rng.randint(2, 4),
                    heads=rng.choice([16, 24, 40, 64, 96, 128]), group=rng.choice([64, 128]), dtype=rng.choice(["bf16", "fp16"]))
        widest = max(case["hidden"], 128 * case["heads"])
        case["tokens"] = _log_int(rng, widest, 1.25 * widest)
    else:
        cols = _cols(rng, 256, 16384 if kind == "quantize" else 7168)
        case.update(rows=_log_int(rng, 1 if kind in ("error", "export") else 64, 32768), cols=cols, group=_group(rng, cols), dtype=dtype)
        if kind not in ("error", "export"):
            # about as many tokens as channels or more: with far fewer the damped Hessian is so ill conditioned
            # that any two 32-bit factorisations part on more codes than a comparison can allow
            case["tokens"] = _log_int(rng, cols, 2 * cols)
    if "tokens" in case:
        case["batches"] = rng.randint(1, min(8, case["tokens"]))
    return case


def draw(rng):
    most = work(next(c for c in listed() if c["kind"] == "attention"))
    while True:
        case = _draw_once(rng)
        w = work(case)
        if case["kind"] == "mse" and case["rows"] * case["cols"] > 1 << 24:
            continue
        if case.get("dtype") == "fp32" and 6 * w["flops"] > most["flops"]:
            continue
        if w["flops"] <= most["flops"] and w["bytes"] <= most["bytes"]:
            return case


# ---------------------------------------------------------------- inputs
def _pieces(total, parts):
    """`total` cut into `parts` uneven pieces, none empty."""
    weights = [3 + (5 * i) % 7 for i in range(parts)]
    out = [max(1, total * w // sum(weights)) for w in weights]
    out[0] += total - sum(out)
    return out


def _layer(rows, cols, dtype, gen):
    layer = nn.Linear(cols, rows, bias=False, device="cuda", dtype=dtype)
    layer.weight.data = (0.02 * torch.randn(rows, cols, generator=gen, device="cuda")).to(dtype)
    return layer


def _batches(tokens, batches, cols, dtype, gen):
    factor = torch.exp(torch.randn(cols, generator=gen, device="cuda"))
    return [(torch.randn(m, cols, generator=gen, device="cuda") * factor).to(dtype) for m in _pieces(tokens, batches)]


def _attention_shapes(case):
    """(rows, columns) of q_a, q_b, kv_a, kv_b and o."""
    h, heads = case["hidden"], case["heads"]
    return [(case["q_rank"], h), (192 * heads, case["q_rank"]), (case["kv_rank"] + 64, h), (256 * heads, case["kv_rank"]), (h, 128 * heads)]


def _expert_tokens(case):
    return _pieces(case["tokens"], case["experts"])


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, dtype = case["kind"], DTYPES[case["dtype"]]
    state = {"case": case}
    if kind == "calibrate":
        # of the layer only its width matters here
        state["layer"] = _layer(8, case["cols"], dtype, gen)
        state["batches"] = _batches(case["tokens"], case["batches"], case["cols"], dtype, gen)
    elif kind == "experts":
        hidden, inner = case["hidden"], case["inner"]
        state["experts"] = [
            {"gate": _layer(inner, hidden, dtype, gen), "up": _layer(inner, hidden, dtype, gen), "down": _layer(hidden, inner, dtype, gen),
             "x": _batches(m, case["batches"], hidden, dtype, gen), "h": _batches(m, case["batches"], inner, dtype, gen)}
            for m in _expert_tokens(case)]
    elif kind == "attention":
        shapes = _attention_shapes(case)
        state["layers"] = [_layer(r, c, dtype, gen) for r, c in shapes]
        state["batches"] = [_batches(case["tokens"], case["batches"], c, dtype, gen) for _, c in shapes]
        state["batches"][2] = state["batches"][0]      # both projections of the hidden state see the same tokens
    elif kind in ("error", "export"):
        rows, cols = case["rows"], case["cols"]
        groups = cols // (case["group"] or cols)
        weight = _layer(rows, cols, dtype, gen).weight.data
        scale = (weight.float().reshape(rows, groups, -1).abs().amax(-1) * (2 / 15)).to(dtype)
        wide = scale.float().repeat_interleave(cols // groups, -1)
        codes = torch.clamp(torch.floor(weight.float() / wide + 8.5), 0, 15).to(torch.uint8)
        state["result"] = (codes, scale, torch.full_like(scale, 8))
        if kind == "error":
            state["weight"] = weight
            handle = GPTQ(nn.Linear(cols, 8, bias=False, device="cuda", dtype=dtype), case["group"] or None, True, REL_DAMP)
            for x in _batches(1024, 1, cols, dtype, gen):
                handle.update(x)
            state["hessian"] = handle.H
    else:
        state["layer"] = _layer(case["rows"], case["cols"], dtype, gen)
        state["batches"] = _batches(case["tokens"], case["batches"], case["cols"], dtype, gen)
    return state


# ---------------------------------------------------------------- one pass
def _handle(layer, case, **options):
    return GPTQ(layer, case.get("group") or None, True, REL_DAMP, **options)


def _calibrated(layer, batches, case, **options):
    handle = _handle(layer, case, **options)
    for x in batches:
        handle.update(x)
    return handle


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "calibrate":
        handle = _calibrated(state["layer"], state["batches"], case)
        return {"hessian": handle.H, "tokens": handle.tokens_collected}
    if kind == "experts":
        handles = []
        for e in state["experts"]:
            gate = _calibrated(e["gate"], e["x"], case)
            up = _handle(e["up"], case, tied_gptq_handle=gate) if case["tied"] else _calibrated(e["up"], e["x"], case)
            handles += [gate, up, _calibrated(e["down"], e["h"], case)]
        results = quantize_many(handles, BITS)
        return {"results": results, "hessians": [h.H for h in handles if h.tied_gptq_handle is None]}
    if kind == "attention":
        handles = [_calibrated(layer, xs, case, is_distributed=True) for layer, xs in zip(state["layers"], state["batches"])]
        results = quantize_shared(handles, BITS)
        return {"results": results, "hessians": [h.H for h in handles]}
    if kind == "error":
        codes, scale, zero = state["result"]
        restored = quant_utils.dequantize_linear_weight(codes, scale, zero)
        error = quant_utils.get_relative_mse_error(restored.float(), state["weight"].float(), state["hessian"])
        return {"restored": restored, "error": error}
    if kind == "export":
        codes, scale, zero = state["result"]
        restored = quant_utils.dequantize_linear_weight(codes, scale, zero)
        packed = pack_weight({"qweight": codes, "scale": scale, "zero": zero}, BITS, True, case["group"] or None)
        return {"restored": restored, "packed": packed}
    options = {"act_order": {"quantization_order": "activation"},
               "mse": {"quantization_scale": quant_utils.QuantizationScale.MSE}}.get(kind, {})
    handle = _calibrated(state["layer"], state["batches"], case, **options)
    result = handle.quantize_packed(BITS) if kind == "quantize_packed" else handle.quantize(BITS)
    return {"result": result, "hessian": handle.H}


# ---------------------------------------------------------------- what a pass cannot do without
def _size(case):
    return 4 if case["dtype"] == "fp32" else 2


def _hessian_work(cols, tokens, size):
    """Every token read once, the Hessian written once; X^T X of a symmetric result."""
    return {"bytes": tokens * cols * size + 4 * cols * cols, "flops": tokens * cols * (cols + 1)}


def _layer_work(rows, cols, group, size, factor=True):
    """Weights in, codes, scales and zero points out; one Cholesky factorisation and the errors' way through the columns behind."""
    groups = cols // (group or cols)
    return {"bytes": rows * cols * (size + 1) + 2 * size * rows * groups,
            "flops": (cols ** 3 / 3 if factor else 0) + rows * cols * (cols - 1)}


def _sum(parts):
    return {k: float(sum(p[k] for p in parts)) for k in ("bytes", "flops")}


def work(case):
    kind, size = case["kind"], _size(case)
    if kind == "calibrate":
        return _sum([_hessian_work(case["cols"], case["tokens"], size)])
    if kind == "experts":
        hidden, inner, g = case["hidden"], case["inner"], case["group"]
        parts = []
        for m in _expert_tokens(case):
            parts += [_hessian_work(hidden, m, size)] * (1 if case["tied"] else 2) + [_hessian_work(inner, m, size)]
            parts += [_layer_work(inner, hidden, g, size), _layer_work(inner, hidden, g, size, factor=not case["tied"]),
                      _layer_work(hidden, inner, g, size)]
        return _sum(parts)
    if kind == "attention":
        parts = []
        for r, c in _attention_shapes(case):
            parts += [_hessian_work(c, case["tokens"], size), _layer_work(r, c, case["group"], size)]
        return _sum(parts)
    rows, cols = case["rows"], case["cols"]
    groups = cols // (case["group"] or cols)
    if kind == "error":
        # two quadratic forms of a symmetric matrix
        return {"bytes": float(rows * cols * (1 + 2 * size) + 4 * cols * cols), "flops": 2.0 * rows * cols * (cols + 1)}
    if kind == "export":
        return {"bytes": float(rows * cols * (1 + size) + rows * cols / 2 + 2 * size * rows * groups), "flops": 2.0 * rows * cols}
    return _sum([_hessian_work(cols, case["tokens"], size), _layer_work(rows, cols, case["group"], size)])


def tolerance(case):
    kind = case["kind"]
    if kind == "export":
        return "exact"
    # Measured between the tensor-core arithmetic and 32-bit sums on the CUDA cores (rel / max): Hessians
    # 1.1e-5 / 1.6e-4 (bf16) and 2.9e-5 / 9e-5 (fp16) after some thousand tokens, error metric 6e-7.
    if kind == "error":
        return {"rel": 3e-6, "max": 3e-6}
    if kind == "calibrate":
        return {"rel": 5e-5, "max": 5e-4}
    # A code on a rounding boundary turns with the last bits of the factor, and takes a share of the codes
    # behind it in its row along: 0.3 % of the codes of a wide layer differ between the two.
    return {"rel": 5e-5, "max": 5e-4, "differ": 0.01}
