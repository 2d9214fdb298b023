"""The calls whose speed is followed: what a user of the package has it do, through its public entry points.

`listed()` names twelve of them, `draw(rng)` gives others of the same ranges. Inputs are synthetic: activations N(0, 1)
in which one channel in a hundred is an outlier (x 20), weights N(0, 0.02^2), gradients N(0, 1e-3^2), and for IF4
Student-t(4) activations. Everything is made from the seed on the GPU.
"""

from __future__ import annotations

import math

import torch
from torch import nn

import fouroversix_b200 as fos
from fouroversix_b200.model.experts import FourOverSixExperts

TORCH = {"bf16": torch.bfloat16, "fp16": torch.float16}
OUT = {"bf16": "bfloat16", "fp16": "float16"}
BYTES = {"nvfp4": 0.5 + 1 / 16, "if4": 0.5 + 1 / 16, "mxfp4": 0.5 + 1 / 32}     # of a packed value with its scale

LARGEST_FLOPS = 2.0 * 32768 * 8192 * 28672
LARGEST_VALUES = 1 << 27


def listed():
    return [
        # one decoding step of a batch of 16 sequences through an 8192-wide projection: launches and latency
        {"name": "linear_decode", "do": "linear", "tokens": 16, "k": 8192, "n": 8192, "type": "bf16", "rule": "mse", "bias": False},
        # a short prompt of an odd length through a layer with a bias, in fp16, static scales, sizes off the tile grid
        {"name": "linear_ragged", "do": "linear", "tokens": 333, "k": 2880, "n": 5000, "type": "fp16", "rule": "static_6", "bias": True},
        # an ordinary prompt through the grouped-query projection of an 8192-wide model
        {"name": "linear_prefill", "do": "linear", "tokens": 4096, "k": 8192, "n": 10240, "type": "bf16", "rule": "mse", "bias": False},
        # a full batch of 16 x 2048 tokens through the widest MLP projection
        {"name": "linear_largest", "do": "linear", "tokens": 32768, "k": 8192, "n": 28672, "type": "bf16", "rule": "mse", "bias": False},
        # forward, dgrad and wgrad of one training step: master weights in 16 x 16 blocks, rotated and stochastically
        # rounded gradients (the layer's defaults)
        {"name": "train_step", "do": "train", "tokens": 4096, "k": 4096, "n": 4096, "type": "bf16", "rule": "mse", "round": "stochastic"},
        # packing one activation tensor (also: a weight, a cache entry, a checkpoint)
        {"name": "quantize_act", "do": "quantize", "rows": 8192, "cols": 4096, "type": "bf16", "format": "nvfp4", "rule": "mse",
         "transpose": False, "blocks_2d": False},
        # unpacking a large weight
        {"name": "dequantize_weight", "do": "dequantize", "rows": 16384, "cols": 8192, "type": "bf16", "format": "nvfp4", "rule": "mse"},
        # the product of two packed tensors by itself
        {"name": "matmul_8192", "do": "matmul", "tokens": 8192, "k": 8192, "n": 8192, "type": "bf16", "format": "nvfp4", "rule": "mse",
         "packed": True},
        # an MLP up projection in IF4: plain activation, packed weight
        {"name": "if4_mlp_up", "do": "matmul", "tokens": 4096, "k": 4096, "n": 14336, "type": "bf16", "format": "if4", "rule": "mse",
         "packed": False},
        # an MLP down projection in MXFP4
        {"name": "mxfp4_mlp_down", "do": "matmul", "tokens": 1024, "k": 14336, "n": 4096, "type": "bf16", "format": "mxfp4",
         "rule": "static_6", "packed": False},
        # a mixture-of-experts layer: a decoding step of many sequences, and a prompt
        {"name": "experts_decode", "do": "experts", "tokens": 256, "k": 2880, "inner": 2880, "experts": 32, "top": 4, "type": "bf16"},
        {"name": "experts_prefill", "do": "experts", "tokens": 8192, "k": 2880, "inner": 2880, "experts": 32, "top": 4, "type": "bf16"},
    ]


def _log(rng, low, high, unit=1):
    """A multiple of `unit` between low and high, spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(low), math.log(high)))
    return max(unit, min(high // unit, round(v / unit)) * unit)


def draw(rng):
    do = rng.choice(["linear", "linear", "linear", "train", "quantize", "dequantize", "matmul", "matmul", "experts"])
    rule = rng.choice(["mse", "mse", "mse", "static_6"])
    kind = rng.choice(["bf16", "bf16", "fp16"])
    if do == "linear":
        k, n = _log(rng, 1024, 14336, 16), _log(rng, 1024, 28672, 8)
        tokens = _log(rng, 1, 32768)
        while 2.0 * tokens * k * n > LARGEST_FLOPS:
            tokens //= 2
        return {"do": do, "tokens": tokens, "k": k, "n": n, "type": kind, "rule": rule, "bias": rng.random() < 0.25}
    if do == "train":
        return {"do": do, "tokens": _log(rng, 256, 16384, 16), "k": _log(rng, 1024, 8192, 16), "n": _log(rng, 1024, 8192, 16),
                "type": "bf16", "rule": rule, "round": rng.choice(["stochastic", "nearest"])}
    if do in ("quantize", "dequantize"):
        rows, cols = _log(rng, 16, 16384), _log(rng, 512, 16384, rng.choice([8, 64, 64]))
        while rows * cols > LARGEST_VALUES:
            rows //= 2
        form = rng.choice(["nvfp4", "nvfp4", "if4", "mxfp4"])
        case = {"do": do, "rows": rows, "cols": cols, "type": kind, "format": form, "rule": _rule(form, rule)}
        if do == "quantize":
            case |= {"transpose": rng.random() < 0.3, "blocks_2d": rng.random() < 0.2}
        return case
    if do == "matmul":
        form = rng.choice(["nvfp4", "nvfp4", "if4", "mxfp4"])
        tokens, k, n = _log(rng, 16, 8192), _log(rng, 1024, 14336, 64), _log(rng, 1024, 14336, 8)
        return {"do": do, "tokens": tokens, "k": k, "n": n, "type": kind, "format": form, "rule": _rule(form, rule),
                "packed": rng.random() < 0.5}
    return {"do": do, "tokens": _log(rng, 16, 8192), "k": _log(rng, 1024, 2880, 64), "inner": _log(rng, 1024, 2880, 64),
            "experts": rng.choice([8, 16, 32]), "top": rng.choice([2, 4]), "type": "bf16"}


def _rule(form, rule):
    return {"if4": "mse", "mxfp4": "static_6"}.get(form, rule)


# ---------------------------------------------------------------------------------------------------------- inputs

def _activations(g, rows, cols, case):
    x = torch.randn(rows, cols, generator=g, device="cuda")
    if case.get("format") == "if4":
        # Student-t with four degrees of freedom: a normal over the root of a chi-square / 4
        chi = torch.zeros_like(x)
        for _ in range(4):
            chi += torch.randn(rows, cols, generator=g, device="cuda").square_()
        x = 0.5 * x * (chi / 4).rsqrt_()
    else:
        x[:, torch.randperm(cols, generator=g, device="cuda")[: max(1, cols // 100)]] *= 20
    return x.to(TORCH[case["type"]])


def _weight(g, *shape, case):
    return (torch.randn(*shape, generator=g, device="cuda") * 0.02).to(TORCH[case["type"]])


def _config(case, **more):
    return fos.QuantizationConfig(dtype=case["format"], scale_rule=case["rule"], **more)


def _linear(g, case, config):
    layer = nn.Linear(case["k"], case["n"], bias=case.get("bias", False), device="cuda", dtype=TORCH[case["type"]])
    with torch.no_grad():
        layer.weight.copy_(_weight(g, case["n"], case["k"], case=case))
        if layer.bias is not None:
            layer.bias.copy_(_weight(g, case["n"], case=case))
    return fos.FourOverSixLinear(layer, config)


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    torch.manual_seed(seed)                 # stochastic rounding draws its seeds from torch's CPU generator
    do = case["do"]
    state = {"case": case}
    if do == "linear":
        layer = _linear(g, case, fos.ModuleQuantizationConfig(scale_rule=case["rule"], output_dtype=OUT[case["type"]]))
        state["layer"] = layer.quantize_weight_()
        state["x"] = _activations(g, case["tokens"], case["k"], case)
    elif do == "train":
        state["layer"] = _linear(g, case, fos.ModuleQuantizationConfig(
            keep_master_weights=True, weight_scale_2d=True, scale_rule=case["rule"], gradient_round_style=case["round"]))
        state["x"] = _activations(g, case["tokens"], case["k"], case).requires_grad_()
        state["dy"] = (torch.randn(case["tokens"], case["n"], generator=g, device="cuda") * 1e-3).to(TORCH[case["type"]])
    elif do == "quantize":
        state["config"] = _config(case, transpose=case["transpose"], block_scale_2d=case["blocks_2d"])
        state["x"] = _activations(g, case["rows"], case["cols"], case)
    elif do == "dequantize":
        state["q"] = fos.quantize(_weight(g, case["rows"], case["cols"], case=case), _config(case))
    elif do == "matmul":
        state["config"] = _config(case)
        x = _activations(g, case["tokens"], case["k"], case)
        state["x"] = fos.quantize(x, state["config"]) if case["packed"] else x
        state["w"] = fos.quantize(_weight(g, case["n"], case["k"], case=case), state["config"])
    else:
        e, h, i = case["experts"], case["k"], case["inner"]
        state["layer"] = FourOverSixExperts(_weight(g, e, 2 * i, h, case=case), _weight(g, e, 2 * i, case=case),
                                            _weight(g, e, h, i, case=case), _weight(g, e, h, case=case))
        state["x"] = torch.randn(case["tokens"], h, generator=g, device="cuda").to(TORCH[case["type"]])
        scores, state["indices"] = torch.randn(case["tokens"], e, generator=g, device="cuda").topk(case["top"])
        state["weights"] = scores.softmax(-1).to(TORCH[case["type"]])
    return state


# ------------------------------------------------------------------------------------------------------- one pass

def run(state):
    case = state["case"]
    do = case["do"]
    if do == "linear":
        with torch.no_grad():
            return state["layer"](state["x"])
    if do == "train":
        layer, x = state["layer"], state["x"]
        x.grad = layer.weight.grad = None
        y = layer(x)
        y.backward(state["dy"])
        return {"y": y.detach(), "dx": x.grad, "dw": layer.weight.grad}
    if do == "quantize":
        q = fos.quantize(state["x"], state["config"])
        return {"values": q.values, "scales": q.scale_factors.view(torch.uint8), "amax": q.amax}
    if do == "dequantize":
        return fos.dequantize(state["q"], TORCH[case["type"]])
    if do == "matmul":
        return fos.quantized_matmul(state["x"], state["w"], input_config=state["config"], out_dtype=OUT[case["type"]])
    with torch.no_grad():
        return state["layer"](state["x"], state["indices"], state["weights"])


def work(case):
    do = case["do"]
    if do in ("quantize", "dequantize"):
        return {"bytes": (2 + BYTES[case["format"]]) * case["rows"] * case["cols"], "flops": 0}
    t, k = case["tokens"], case["k"]
    if do == "experts":
        i, pairs = case["inner"], t * case["top"]
        return {"bytes": BYTES["nvfp4"] * 3 * k * i * min(case["experts"], pairs) + 4 * t * k, "flops": 2 * 3 * pairs * k * i}
    n = case["n"]
    if do == "train":
        return {"bytes": 2 * 2 * (t * k + n * k + t * n), "flops": 3 * 2 * t * k * n}
    packed = BYTES[case.get("format", "nvfp4")]
    return {"bytes": (packed if case.get("packed") else 2) * t * k + packed * n * k + 2 * t * n, "flops": 2 * t * k * n}


def tolerance(case):
    if case["do"] in ("quantize", "dequantize"):
        return "exact"                      # every step of the two is one rounding of a stated operation
    if case["do"] == "experts":
        # the hidden product is quantized again: where the order of its sums moves one of its roundings, a code moves
        return {"rel": 1e-2, "max": 1e-1}
    if case["type"] == "fp16" and case.get("format") != "if4":
        # measured against a product of the unpacked operands in 64 bits: 2.9e-4, the output's rounding; one output
        # off by a unit in the last place: 1e-3
        return {"rel": 1.2e-3, "max": 4e-3}
    # the same in bf16: 1.7e-3 and 7.8e-3; IF4 values times their scale rounded to fp16: 1.0e-3 before the output's rounding
    return {"rel": 6e-3, "max": 3e-2}
