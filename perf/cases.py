"""The work that is timed: one pass per case through the public entry points.

Five kinds of pass, over the sizes of this repository's benchmark, tests and model-shaped workloads (hidden sizes
1024 to 5120, MLP widths 12288 to 17408, 1 to 16384 tokens, calibration sets of 16 to 128 sequences):

  linear   `FPQuantLinear.forward` with pre-quantised weights (inference): rotate + quantise, FP4 GEMM
  gated    `FPQuantLinear.forward_silu_mul`: the down-projection of a gated MLP
  train    forward and backward of an `FPQuantLinear` that holds its master weight
  gptq     MR-GPTQ of one linear: rotation, Hessian over the calibration tokens, factor, column loop, error metric
  rtn      round-to-nearest of one weight: rotation, scales, codes, dequantised weight
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "fp-quant_b200"))

from fpq_b200.fp_quant import FPQuantConfig, FPQuantDtype, FPQuantLinear  # noqa: E402
from fpq_b200.quantization.gptq import GPTQ, get_relative_mse_error  # noqa: E402
from fpq_b200.quantization.quant_ops import pack_fp4_to_uint8  # noqa: E402
from fpq_b200.quantization.quantizer import Quantizer  # noqa: E402
from fpq_b200.transforms.transforms import HadamardTransform  # noqa: E402

DEV = "cuda"
DTYPE = {"mxfp4": FPQuantDtype.MXFP4, "nvfp4": FPQuantDtype.NVFP4, "mxfp8": FPQuantDtype.MXFP8, "bf16": FPQuantDtype.BF16}
GROUP = {"mxfp4": 32, "nvfp4": 16}


def _linear(name, m, k, n, fmt, method="abs_max", group=32, bias=False):
    return {"name": name, "kind": "linear", "m": m, "k": k, "n": n, "fmt": fmt, "method": method, "group": group, "bias": bias}


def _gated(name, m, k, n, fmt, group=32):
    return {"name": name, "kind": "gated", "m": m, "k": k, "n": n, "fmt": fmt, "method": "abs_max", "group": group, "bias": False}


def _train(name, m, k, n, fmt, backward, method, bias=False):
    return {"name": name, "kind": "train", "m": m, "k": k, "n": n, "fmt": fmt, "backward": backward, "method": method,
            "group": 16 if fmt == "nvfp4" else 32, "bias": bias}


def _gptq(name, rows, cols, seqs, length, fmt):
    return {"name": name, "kind": "gptq", "rows": rows, "cols": cols, "seqs": seqs, "length": length, "fmt": fmt, "group": 128}


def _rtn(name, rows, cols, fmt, observer="minmax"):
    return {"name": name, "kind": "rtn", "rows": rows, "cols": cols, "fmt": fmt, "observer": observer, "group": 128}


def listed():
    return [
        # one token of one request through an attention projection: the smallest call there is
        _linear("decode_1", 1, 4096, 4096, "mxfp4"),
        # a small decode batch through an up-projection with a bias, NVFP4 with its own rotation size
        _linear("decode_16_nvfp4", 16, 4096, 12288, "nvfp4", group=16, bias=True),
        # a decode batch of 64 through the down-projection of a gated MLP
        _gated("decode_64_gated", 64, 17408, 5120, "mxfp4"),
        # a prompt of odd length, NVFP4 with the 128-wide rotation that MR-GPTQ checkpoints carry
        _linear("prefill_3001_nvfp4", 3001, 5120, 17408, "nvfp4", group=128),
        # a full prefill batch with the default scale rule (QuEST)
        _linear("prefill_8192_quest", 8192, 12288, 4096, "mxfp4", method="quest"),
        # prefill of 8 x 2048 tokens through the down-projection of a gated MLP
        _gated("prefill_16384_gated", 16384, 17408, 5120, "mxfp4"),
        # a fine-tuning step of a layer, the three backward types: MXFP8 on a small batch, ...
        _train("train_2048_mxfp8", 2048, 4096, 4096, "mxfp4", "mxfp8", "abs_max"),
        # ... MXFP4 with QuEST scales and their clip masks (the default configuration) on a large one, ...
        _train("train_8192_mxfp4_quest", 8192, 4096, 12288, "mxfp4", "mxfp4", "quest"),
        # ... and bf16, the one that NVFP4 trains with, on a ragged batch
        _train("train_4000_nvfp4", 4000, 4096, 4096, "nvfp4", "bf16", "abs_max", bias=True),
        # round-to-nearest of a square weight
        _rtn("rtn_4096", 4096, 4096, "nvfp4"),
        # MR-GPTQ of an up-projection over 128 x 2048 calibration tokens
        _gptq("gptq_up", 14336, 4096, 128, 2048, "nvfp4"),
        # MR-GPTQ of a down-projection, whose Hessian is the widest
        _gptq("gptq_down", 4096, 14336, 128, 2048, "mxfp4"),
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of `step` between lo and hi, spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi // step * step, max(-(-lo // step) * step, round(v / step) * step))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "linear", "gated", "gated", "train", "train", "train", "gptq", "gptq", "rtn"])
    if kind in ("linear", "gated"):
        fmt = rng.choice(["mxfp4", "nvfp4"])
        group = rng.choice([32, 32, 64, 128] if fmt == "mxfp4" else [16, 16, 64, 128])
        method = "quest" if kind == "linear" and fmt == "mxfp4" and rng.random() < 0.5 else "abs_max"
        case = {"kind": kind, "m": _log(rng, 1, 16384), "k": _log(rng, 1024, 17408, max(64, group)), "n": _log(rng, 1024, 17408, 16),
                "fmt": fmt, "method": method, "group": group, "bias": kind == "linear" and rng.random() < 0.3}
    elif kind == "train":
        backward = rng.choice(["mxfp8", "mxfp4", "bf16"])
        fmt = rng.choice(["mxfp4", "nvfp4"]) if backward == "bf16" else "mxfp4"
        case = {"kind": kind, "m": _log(rng, 512, 8192), "k": _log(rng, 1024, 12288, 128), "n": _log(rng, 1024, 12288, 128),
                "fmt": fmt, "backward": backward, "method": rng.choice(["abs_max", "quest"]) if fmt == "mxfp4" else "abs_max",
                "group": 16 if fmt == "nvfp4" else 32, "bias": rng.random() < 0.5}
    elif kind == "gptq":
        cols = _log(rng, 1024, 14336, 128)
        length = rng.choice([2048, rng.randrange(1024, 2048)])
        seqs = rng.randrange(max(16, -(-4 * cols // length)), 129)      # at least four tokens per column
        case = {"kind": kind, "rows": min(_log(rng, 1024, 14336, 8), 14336 * 4096 // cols // 8 * 8), "cols": cols, "seqs": seqs,
                "length": length, "fmt": rng.choice(["nvfp4", "mxfp4"]), "group": 128}
    else:
        case = {"kind": kind, "rows": _log(rng, 1024, 14336, 8), "cols": _log(rng, 1024, 14336, 128), "fmt": rng.choice(["nvfp4", "mxfp4"]),
                "observer": rng.choice(["minmax", "mse"]), "group": 128}
    return case


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _activations(g, m, k):
    """Student-t(4) * 0.5 with one channel of a hundred scaled by 20."""
    x = torch.randn(m, k, device=DEV, generator=g)
    chi = torch.zeros_like(x)
    for _ in range(4):
        chi += torch.randn(m, k, device=DEV, generator=g).square_()
    x.mul_(chi.div_(4).rsqrt_()).mul_(0.5)
    x[:, torch.randperm(k, device=DEV, generator=g)[: max(1, k // 100)]] *= 20
    return x.to(torch.bfloat16)


def _weight(g, n, k):
    return (torch.randn(n, k, device=DEV, generator=g) * 0.02).to(torch.bfloat16)


def _calibration(g, seqs, length, d):
    """Correlated activations: a rank-64 mixture plus noise of the same size, so that the Hessian is far from diagonal."""
    mix = torch.randn(64, d, device=DEV, generator=g) / 8
    x = torch.empty(seqs, length, d, device=DEV, dtype=torch.bfloat16)
    for i in range(seqs):
        z = torch.randn(length, 64, device=DEV, generator=g)
        x[i] = z @ mix + torch.randn(length, d, device=DEV, generator=g)
    return x


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind == "gptq":
        shell = torch.nn.Linear(case["cols"], case["rows"], bias=False, device="meta").requires_grad_(False)
        return {"case": case, "weight": _weight(g, case["rows"], case["cols"]), "layer": shell,
                "x": _calibration(g, case["seqs"], case["length"], case["cols"]), "rotate": HadamardTransform(case["group"])}
    if kind == "rtn":
        return {"case": case, "weight": _weight(g, case["rows"], case["cols"]), "rotate": HadamardTransform(case["group"])}
    m, k, n = case["m"], case["k"], case["n"]
    config = FPQuantConfig(forward_dtype=DTYPE[case["fmt"]], forward_method=case["method"],
                           backward_dtype=DTYPE[case.get("backward", "bf16")], store_master_weights=kind == "train",
                           hadamard_group_size=case["group"])
    layer = FPQuantLinear(k, n, config, bias=case["bias"], device=DEV, dtype=torch.bfloat16)
    with torch.no_grad():
        layer.weight.copy_(_weight(g, n, k))
        if case["bias"]:
            layer.bias.copy_((torch.randn(n, device=DEV, generator=g) * 0.1).to(torch.bfloat16))
    layer.pre_forward()
    state = {"case": case, "layer": layer}
    if kind == "gated":
        state["gate"] = torch.randn(m, k, device=DEV, generator=g).to(torch.bfloat16)
        state["up"] = _activations(g, m, k)
    else:
        state["x"] = _activations(g, m, k)
    if kind == "train":
        state["x"].requires_grad_(True)
        state["grad"] = (torch.randn(m, n, device=DEV, generator=g) * 0.01).to(torch.bfloat16)
    return state


# ------------------------------------------------------------------------------------------------ one pass
def _quantizer(case):
    nv = case["fmt"] == "nvfp4"
    return Quantizer(bits=4, symmetric=True, format="nvfp" if nv else "mxfp", granularity="group", group_size=GROUP[case["fmt"]],
                     scale_precision="e4m3" if nv else "e8m0", observer=case.get("observer", "minmax"))


def run(state):
    case = state["case"]
    return {"linear": _run_linear, "gated": _run_gated, "train": _run_train, "gptq": _run_gptq, "rtn": _run_rtn}[case["kind"]](state, case)


def _run_linear(state, case):
    with torch.no_grad():
        return state["layer"](state["x"])


def _run_gated(state, case):
    with torch.no_grad():
        return state["layer"].forward_silu_mul(state["gate"], state["up"])


def _run_train(state, case):
    layer, x = state["layer"], state["x"]
    x.grad = layer.weight.grad = None
    if layer.bias is not None:
        layer.bias.grad = None
    y = layer(x)
    y.backward(state["grad"])
    return {"y": y, "x": x.grad, "weight": layer.weight.grad, "bias": None if layer.bias is None else layer.bias.grad}


def _run_gptq(state, case):
    layer, rotate, x = state["layer"], state["rotate"], state["x"]
    layer.weight = torch.nn.Parameter(rotate(state["weight"]), requires_grad=False)
    handle = GPTQ(layer, _quantizer(case))
    step = max(1, 16384 // case["length"])
    for i in range(0, case["seqs"], step):
        handle.update(rotate(x[i:i + step]))
    weight, _, scales = handle.quantize(want_grid_values=False)
    return {"weight": weight, "codes": handle.packed_codes, "scales": scales,
            "error": get_relative_mse_error(weight, layer.weight, handle.H)}


def _run_rtn(state, case):
    quantizer = _quantizer(case)
    w = state["rotate"](state["weight"]).float()
    scales, zeros = quantizer.get_quantization_params(w)
    grid = quantizer.quantize(w, scales, zeros)
    return {"codes": pack_fp4_to_uint8(grid), "scales": scales, "weight": quantizer.dequantize(grid, scales, zeros)}


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "rtn":
        e = case["rows"] * case["cols"]
        return {"bytes": 2 * e + e / 2 + 4 * e / GROUP[case["fmt"]] + 4 * e, "flops": 12 * e}
    if kind == "gptq":
        rows, d, tokens = case["rows"], case["cols"], case["seqs"] * case["length"]
        e = rows * d
        return {"bytes": 2 * tokens * d + 2 * e + 2 * e + e / 2 + 4 * e / GROUP[case["fmt"]],
                # Hessian (symmetric), factor and triangular inverse, column loop, error metric
                "flops": tokens * d * (d + 1) + 2 / 3 * d ** 3 + rows * d * d + 2 * rows * d * (d + 1)}
    m, k, n = case["m"], case["k"], case["n"]
    if kind == "train":
        return {"bytes": 2 * (2 * m * k + 2 * n * k + 2 * m * n), "flops": 6 * m * n * k}
    weights = n * k / 2 + n * k / GROUP[case["fmt"]]
    return {"bytes": (4 if kind == "gated" else 2) * m * k + weights + 2 * m * n, "flops": 2 * m * n * k}


def tolerance(case):
    if case["kind"] == "rtn":
        return "exact"
    if case["kind"] == "gptq":
        # The column loop feeds every rounding into the columns that follow, so the last bits of the Hessian move codes.  The
        # same pass over the calibration sequences in another order: weights 1e-3 to 5e-3 (one grid step at most: 0.52 of a
        # value), 3e-5 to 4e-4 of the code bytes, error metric below 1e-5.
        return {"rel": 0.02, "max": 0.95, "differ": 0.0016}
    # bf16 results of fp32 sums: the unrounded fp64 product is 1.66e-3 away, no value by more than 3.9e-3.
    return {"rel": 0.006, "max": 0.016}
