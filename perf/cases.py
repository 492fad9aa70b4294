"""The work that a user of this library has it do, as cases that can be timed.

Five kinds of pass, each through the public classes and functions:

  forward    the packed linears of one or more decoder blocks on `tokens` rows of activations: decode (a few
             tokens, usually replayed from a CUDA graph as a serving loop does), small batches, prefill
  train      forward and backward of the packed linears of a block with frozen weights, as adapter fine-tuning
             on a quantized model runs them
  quantize   round-to-nearest quantization of a decoder block (`quantize_block`)
  roundtrip  `quantize_rtn` of one weight matrix and `dequantize_rtn` of the result
  tune       one step of the trainable mode: `WrapperLinear` forward, backward into its range factors

Weights are N(0, 0.02^2) and activations N(0, 1), the distributions of a transformer's linears behind a norm.
The linears of a block get inputs of their own instead of each other's outputs: attention and norms are the
model's, not this library's.
"""
import math

import torch
import torch.nn as nn
import torch.nn.functional as F

from bitween_b200 import QuantizedLinear, dequantize_rtn, quantize_rtn
from bitween_b200.gradual.base_wrapper import quantize_block
from bitween_b200.wrapper import WrapperLinear

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}
SIZES = {"fp16": 2, "bf16": 2, "fp32": 4}
MOST_FLOPS = 3.5e12          # of a drawn case; the largest listed one has 3.57e12
MOST_WEIGHTS = 850e6         # packed weights of a drawn case (four blocks of the 8B shapes have 872e6)


def _forward(name, hidden, kv, ffn, gated, blocks, bits, group, tokens, dtype, bias, graph):
    return {"name": name, "kind": "forward", "hidden": hidden, "kv": kv, "ffn": ffn, "gated": gated, "blocks": blocks,
            "bits": bits, "group": group, "tokens": tokens, "dtype": dtype, "bias": bias, "graph": graph}


def listed():
    return [
        # The smallest calls: one token through a block of OPT-125m at the library's default precision, called
        # layer by layer from Python as generate() does. Launches and host work are what it costs.
        _forward("opt125m_block_1tok_w8", 768, 768, 3072, False, 1, 8, 32, 1, "fp16", True, False),
        # The same way of calling on a block of the Llama-3-8B shapes, two sequences, 8 bits.
        _forward("8b_block_2tok_w8_eager", 4096, 1024, 14336, True, 1, 8, 128, 2, "fp16", False, False),
        # Single-sequence decode of a served model: four blocks (more weights than L2 holds), one CUDA graph.
        _forward("8b_decode_1tok_w4", 4096, 1024, 14336, True, 4, 4, 128, 1, "fp16", False, True),
        # The same with a batch of 16 and bf16 activations, as most checkpoints have them.
        _forward("8b_decode_16tok_w4_bf16", 4096, 1024, 14336, True, 4, 4, 128, 16, "bf16", False, True),
        # Feed-forward width 11008: 86 quantization groups a row, not a whole number of 16-byte scale vectors.
        _forward("7b_decode_5tok_w4_ragged", 4096, 4096, 11008, True, 4, 4, 128, 5, "fp16", False, True),
        # A larger decode batch (or a draft of speculative decoding being checked).
        _forward("8b_decode_48tok_w4", 4096, 1024, 14336, True, 4, 4, 128, 48, "fp16", False, True),
        # A prompt of ordinary, odd length.
        _forward("8b_prefill_509tok_w4", 4096, 1024, 14336, True, 1, 4, 128, 509, "fp16", False, False),
        # The largest: a batch of prompts, bf16 activations.
        _forward("8b_prefill_8192tok_w4_bf16", 4096, 1024, 14336, True, 1, 4, 128, 8192, "bf16", False, False),
        # Fine-tuning an adapter on frozen packed weights: every linear forward and backward.
        {"name": "8b_train_2048tok_w4", "kind": "train", "hidden": 4096, "kv": 1024, "ffn": 14336, "gated": True,
         "bits": 4, "group": 128, "tokens": 2048, "dtype": "fp16"},
        # Quantizing a checkpoint, block by block.
        {"name": "8b_quantize_block_bf16_w4", "kind": "quantize", "hidden": 4096, "kv": 1024, "ffn": 14336, "gated": True,
         "bits": 4, "group": 128, "dtype": "bf16"},
        # Both directions of the wire format on one fp32 matrix at the default precision.
        {"name": "roundtrip_4096_fp32_w8", "kind": "roundtrip", "rows": 4096, "cols": 4096, "bits": 8, "group": 32, "dtype": "fp32"},
        # A training step of the trainable mode on a calibration batch.
        {"name": "tune_4096_bf16_w4", "kind": "tune", "rows": 4096, "cols": 4096, "bits": 4, "group": 128, "tokens": 256, "dtype": "bf16"},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _block_sizes(rng, weights, group):
    """hidden, kv and ffn of a block with at most `weights` weights. Widths are multiples of 128 (of the head size
    and of every group size); the feed-forward width is any multiple of the group size."""
    while True:
        hidden = 128 * round(_log(rng, 4, 64))
        kv = max(128, hidden // rng.choice((1, 4, 8)) // 128 * 128)
        ffn = group * round(hidden * rng.uniform(2.0, 4.0) / group)
        gated = rng.random() < 0.7
        if sum(n * k for _, n, k in _linears(hidden, kv, ffn, gated)) <= weights:
            return hidden, kv, ffn, gated


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode", "prefill", "train", "quantize", "roundtrip", "tune"))
    bits, group = rng.choice((2, 4, 4, 8)), rng.choice((32, 64, 128, 128))
    dtype = rng.choice(("fp16", "fp16", "bf16", "fp32"))
    if kind in ("decode", "prefill", "train"):
        hidden, kv, ffn, gated = _block_sizes(rng, 450e6 if kind == "decode" else 300e6, group)
        weights = sum(n * k for _, n, k in _linears(hidden, kv, ffn, gated))
        most = MOST_FLOPS / weights / (2 if kind != "train" else 4)
        if kind == "train":
            return {"kind": "train", "hidden": hidden, "kv": kv, "ffn": ffn, "gated": gated, "bits": bits, "group": group,
                    "tokens": max(1, round(_log(rng, 16, min(2048, most)))), "dtype": dtype}
        tokens = max(1, round(_log(rng, 1, 64))) if kind == "decode" else max(65, round(_log(rng, 65, min(8192, most))))
        blocks = rng.randint(1, max(1, min(4, int(MOST_WEIGHTS / weights)))) if kind == "decode" else 1
        case = _forward("", hidden, kv, ffn, gated, blocks, bits, group, tokens, dtype, not gated, kind == "decode" and rng.random() < 0.6)
        del case["name"]
        return case
    if kind == "quantize":
        hidden, kv, ffn, gated = _block_sizes(rng, 220e6, group)
        return {"kind": "quantize", "hidden": hidden, "kv": kv, "ffn": ffn, "gated": gated, "bits": bits, "group": group, "dtype": dtype}
    rows, cols = round(_log(rng, 256, 16384)), group * round(_log(rng, 512, 8192) / group)
    if kind == "roundtrip":
        return {"kind": "roundtrip", "rows": rows, "cols": cols, "bits": bits, "group": group, "dtype": dtype}
    return {"kind": "tune", "rows": min(rows, 8192), "cols": cols, "bits": bits, "group": group,
            "tokens": round(_log(rng, 32, 512)), "dtype": dtype}


def _linears(hidden, kv, ffn, gated):
    """(which input, out_features, in_features) of a decoder block's linears."""
    attention = [("hidden", hidden, hidden), ("hidden", kv, hidden), ("hidden", kv, hidden), ("attention", hidden, hidden)]
    up = [("hidden", ffn, hidden)] * (2 if gated else 1)
    return attention + up + [("ffn", hidden, ffn)]


def _layers(case):
    return _linears(case["hidden"], case["kv"], case["ffn"], case["gated"])


def _float_linear(gen, n, k, dtype, bias=False):
    layer = nn.Linear(k, n, bias=bias, device="meta")
    layer.weight = nn.Parameter(torch.randn(n, k, generator=gen, device="cuda", dtype=dtype).mul_(0.02), requires_grad=False)
    if bias:
        layer.bias = nn.Parameter(torch.randn(n, generator=gen, device="cuda", dtype=dtype).mul_(0.1), requires_grad=False)
    return layer


def _packed_block(case, gen, bias=False):
    return [QuantizedLinear.from_float(_float_linear(gen, n, k, torch.float16, bias), case["bits"], case["group"]) for _, n, k in _layers(case)]


def _inputs(case, gen, dtype):
    widths = {"hidden": case["hidden"], "attention": case["hidden"], "ffn": case["ffn"]}
    return {which: torch.randn(case["tokens"], w, generator=gen, device="cuda").to(dtype) for which, w in widths.items()}


class Block(nn.Module):
    """The linears of a decoder block under one module, as a checkpoint's block holds them."""

    def __init__(self, layers):
        super().__init__()
        self.layers = nn.ModuleList(layers)


def _forward_pass(state):
    return [layer(state["x"][which]) for block in state["blocks"] for (which, _, _), layer in zip(state["order"], block)]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, dtype = case["kind"], DTYPES[case["dtype"]]
    state = {"kind": kind}
    if kind == "forward":
        state["order"] = _layers(case)
        state["blocks"] = [_packed_block(case, gen, case["bias"]) for _ in range(case["blocks"])]
        state["x"] = _inputs(case, gen, dtype)
        state["graph"] = None
        if case["graph"]:
            # as a serving loop sets itself up: one warm-up pass on a side stream, then the capture
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.no_grad(), torch.cuda.stream(side):
                _forward_pass(state)
            torch.cuda.current_stream().wait_stream(side)
            state["graph"] = torch.cuda.CUDAGraph()
            with torch.no_grad(), torch.cuda.graph(state["graph"]):
                state["out"] = _forward_pass(state)
    elif kind == "train":
        state["order"] = _layers(case)
        state["layers"] = _packed_block(case, gen)
        x = _inputs(case, gen, dtype)
        # one leaf per linear, so that every gradient comes back by itself
        state["x"] = [x[which].clone().requires_grad_(True) for which, _, _ in state["order"]]
        state["grad"] = [torch.randn(case["tokens"], n, generator=gen, device="cuda").mul_(0.01).half() for _, n, _ in state["order"]]
    elif kind == "quantize":
        state["block"] = Block([_float_linear(gen, n, k, dtype) for _, n, k in _layers(case)])
        state["bits"], state["group"] = case["bits"], case["group"]
    elif kind == "roundtrip":
        state["weight"] = torch.randn(case["rows"], case["cols"], generator=gen, device="cuda").mul_(0.02).to(dtype)
        state["bits"], state["group"] = case["bits"], case["group"]
    else:
        state["layer"] = WrapperLinear(_float_linear(gen, case["rows"], case["cols"], dtype), bits=case["bits"], group_size=case["group"])
        with torch.no_grad():
            state["layer"].value.copy_(torch.rand(case["rows"], case["cols"], generator=gen, device="cuda").sub_(0.5))
        state["x"] = torch.randn(case["tokens"], case["cols"], generator=gen, device="cuda")
        state["target"] = torch.randn(case["tokens"], case["rows"], generator=gen, device="cuda")
    return state


def run(state):
    kind = state["kind"]
    if kind == "forward":
        if state["graph"] is not None:
            state["graph"].replay()
            return state["out"]
        with torch.no_grad():
            return _forward_pass(state)
    if kind == "train":
        out = []
        for layer, x, g in zip(state["layers"], state["x"], state["grad"]):
            y = layer(x)
            out += [y.detach(), *torch.autograd.grad(y, x, g)]
        return out
    if kind == "quantize":
        block = quantize_block(state["block"], state["bits"], state["group"])
        return [t for layer in block.layers for t in (layer.qweight, layer.scale, layer.zero_point)]
    if kind == "roundtrip":
        q, scale, zero_point, group = quantize_rtn(state["weight"], state["bits"], state["group"])
        return [q, scale, zero_point, dequantize_rtn(q, scale, zero_point, group, state["bits"])]
    layer = state["layer"]
    layer.zero_grad(set_to_none=True)
    y = layer(state["x"])
    F.mse_loss(y, state["target"]).backward()
    return [y.detach(), layer.min_scale.grad, layer.max_scale.grad]


def work(case):
    kind, size = case["kind"], SIZES[case["dtype"]]
    if kind in ("forward", "train"):
        layers, m = _layers(case), case["tokens"]
        packed = sum(n * k * case["bits"] / 8 + 4 * n * k / case["group"] for _, n, k in layers)
        flops = sum(2 * m * n * k for _, n, k in layers)
        outs = sum(2 * m * n for _, n, _ in layers)
        if kind == "forward":
            # a block's three inputs are read once and shared by its linears (and by the blocks)
            ins = size * m * (2 * case["hidden"] + case["ffn"])
            return {"bytes": case["blocks"] * (packed + outs) + ins, "flops": case["blocks"] * flops}
        ins = sum(size * m * k for _, _, k in layers)
        return {"bytes": packed + 2 * ins + 2 * outs, "flops": 2 * flops}
    if kind == "quantize":
        weights = sum(n * k for _, n, k in _layers(case))
        return {"bytes": weights * (size + case["bits"] / 8 + 4 / case["group"]), "flops": 0}
    weights = case["rows"] * case["cols"]
    if kind == "roundtrip":
        # weights in, packed words and parameters out; the dequantized fp32 matrix out
        return {"bytes": weights * (size + case["bits"] / 8 + (size + 4) / case["group"] + 4), "flops": 0}
    m = case["tokens"]
    # weight and perturbation in; activations, target and outputs; the range factors and their gradients;
    # one product forward and one (the weight's gradient) backward
    return {"bytes": 2 * size * weights + 4 * m * (case["cols"] + 2 * case["rows"]) + 16 * weights / case["group"],
            "flops": 4 * m * weights}


def tolerance(case):
    kind = case["kind"]
    if kind in ("quantize", "roundtrip"):
        return "exact"           # codes, scales, zero points and dequantized weights are defined to the bit
    if kind == "tune":
        return {"rel": 5e-6, "max": 4e-5}     # fp32 sums in another order: 1.2e-6 and 8.5e-6 from 64-bit sums
    # one rounding of an fp32 sum to fp16, a second one where a bias is added: 2.1e-4 (3.2e-4) and at most
    # 5e-4 (1e-3) from 64-bit sums of the same fp16 weights
    return {"rel": 1.2e-3, "max": 4e-3}
