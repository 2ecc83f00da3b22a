"""The calls that users of this framework make, as cases to be timed: single convolutions through both operator
surfaces and the module, matrix products, transposed convolutions, and chains of fused convolutions.

Sizes are those of the repository's own benchmark configurations and layer table, or generic ones. The path is
inference only, so there is one direction; the data types are the three that it computes.
"""
import math

import torch

from tracea_b200 import nn as tnn
from tracea_b200 import ops, resnet50, runner

_DT = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}

# Bounds of a drawn case: far below the largest listed one even where a layer runs at a few per cent of the peak.
_MAX_BYTES = 6e8
_MAX_FLOPS = 3e11


def _conv(name, via, dtype, n, c, h, w, k, r, stride, pad, epilogue, dil=1):
    return {"name": name, "kind": "conv", "via": via, "dtype": dtype, "n": n, "c": c, "h": h, "w": w, "k": k, "r": r,
            "stride": stride, "pad": pad, "dil": dil, "epilogue": epilogue}


def listed():
    return [
        # the smallest call: one image in the framework's default NCHW memory, fp32 -- an interactive request, where
        # latency and launches count
        _conv("conv_one_image_f32", "nchw", "f32", 1, 64, 56, 56, 64, 3, 1, 1, "bias+relu"),
        # a module dropped into a user's own network on one large NCHW image (decoder / super-resolution resolution)
        _conv("conv_large_image_f16", "module", "f16", 1, 64, 224, 224, 128, 3, 1, 0, ""),
        # the reference's own benchmark layer at a serving batch
        _conv("conv_64ch_bf16_n32", "nhwc", "bf16", 32, 64, 56, 56, 64, 3, 1, 1, "bias+relu"),
        # a strided downsampling layer at a throughput batch, with an activation that costs arithmetic
        _conv("conv_down_bf16_n256", "nhwc", "bf16", 256, 128, 56, 56, 256, 3, 2, 1, "bias+silu"),
        # nothing is a multiple of anything: odd channel counts and extents in NCHW memory, as user-written networks have
        _conv("conv_ragged_f16", "nchw", "f16", 3, 20, 61, 83, 50, 5, 1, 2, "gelu"),
        # fp32 storage with a skip connection: networks that are not converted to 16 bits
        _conv("conv_residual_f32_n16", "nhwc", "f32", 16, 128, 28, 28, 128, 3, 1, 1, "bias+residual+relu"),
        # three fused convolutions with a residual: the repeated unit of the network below, at the benchmark's batch
        {"name": "block_bf16_n256", "kind": "block", "dtype": "bf16", "n": 256, "replay": False},
        # one image through the whole convolution stack, replayed from a graph: 53 dependent small launches
        {"name": "stack_bf16_n1", "kind": "stack", "dtype": "bf16", "n": 1, "replay": True},
        # the whole convolution stack at the benchmark's batch: the largest case
        {"name": "stack_bf16_n512", "kind": "stack", "dtype": "bf16", "n": 512, "replay": False},
        # a large square matrix product with the weight in the layout of a linear layer
        {"name": "gemm_square_bf16", "kind": "gemm", "dtype": "bf16", "m": 8192, "n": 8192, "k": 8192, "w": "nk",
         "epilogue": ""},
        # a classifier head on a small batch: few rows, a long reduction
        {"name": "gemm_head_f16", "kind": "gemm", "dtype": "f16", "m": 64, "n": 1000, "k": 2048, "w": "nk",
         "epilogue": "bias"},
        # the upsampling layer of a decoder
        {"name": "conv_transpose_bf16_n128", "kind": "conv_transpose", "dtype": "bf16", "n": 128, "c": 256, "h": 32,
         "w": 32, "k": 128, "r": 4, "stride": 2, "pad": 1, "opad": 0, "epilogue": "bias+relu"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _channels(rng, lo=16, hi=1024):
    """Half of them multiples of 64, a quarter multiples of 8, a quarter anything down to single channels."""
    u = rng.random()
    if u < 0.5:
        return 64 * max(1, _log(rng, max(lo, 64), hi) // 64)
    if u < 0.75:
        return 8 * max(1, _log(rng, lo, hi // 2) // 8)
    return _log(rng, 1, hi // 4)


def _draw_once(rng):
    dtype = rng.choice(["bf16", "bf16", "f16", "f32"])
    u = rng.random()
    if u < 0.55:
        via = rng.choice(["nhwc", "nhwc", "nchw", "module"])
        h = _log(rng, 7, 224)
        r = rng.choice([1, 1, 3, 3, 3, 5, 7])
        epi = rng.choice(["", "bias"]) if via == "module" else rng.choice(
            ["", "bias", "relu", "bias+relu", "bias+silu", "gelu", "residual+relu", "bias+residual+relu"])
        return {"kind": "conv", "via": via, "dtype": dtype, "n": _log(rng, 1, 256), "c": _channels(rng), "h": h,
                "w": h if rng.random() < 0.5 else _log(rng, 7, 224), "k": _channels(rng), "r": r,
                "stride": rng.choice([1, 1, 2]), "pad": rng.choice([r // 2, r // 2, r // 2, 0]),
                "dil": 2 if r == 3 and rng.random() < 0.15 else 1, "epilogue": epi}
    if u < 0.75:
        odd = rng.random() < 0.25
        n, k = _log(rng, 64, 8192), _log(rng, 64, 8192)
        return {"kind": "gemm", "dtype": dtype, "m": _log(rng, 1, 16384), "n": n if odd else 8 * (n // 8),
                "k": k if odd else 8 * (k // 8), "w": rng.choice(["nk", "nk", "kn"]),
                "epilogue": rng.choice(["", "bias", "bias+relu", "gelu", "bias+residual"])}
    if u < 0.9:
        stride = rng.choice([1, 2, 2, 2, 3])
        r = rng.randint(max(2, stride), 5)
        return {"kind": "conv_transpose", "dtype": dtype, "n": _log(rng, 1, 128), "c": _channels(rng, 16, 512),
                "h": _log(rng, 4, 64), "w": _log(rng, 4, 64), "k": _channels(rng, 16, 512), "r": r, "stride": stride,
                "pad": rng.randint(0, (r - 1) // 2), "opad": rng.randint(0, stride - 1),
                "epilogue": rng.choice(["", "bias", "bias+relu", "bias+silu", "bias+residual+relu"])}
    n = _log(rng, 1, 256)
    return {"kind": rng.choice(["block", "stack"]), "dtype": rng.choice(["bf16", "bf16", "f16"]), "n": n,
            "replay": n <= 16}


def draw(rng):
    while True:
        case = _draw_once(rng)
        if case["kind"] in ("block", "stack"):
            return case
        if case["kind"] == "conv" and min(case["h"], case["w"]) + 2 * case["pad"] <= case["dil"] * (case["r"] - 1):
            continue
        wk = work(case)
        if wk["bytes"] <= _MAX_BYTES and wk["flops"] <= _MAX_FLOPS:
            return case


# ---------------------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(gen, shape, dtype, std=1.0):
    return (torch.randn(shape, generator=gen, device="cuda") * std).to(dtype)


def _has(case, op):
    return op in case["epilogue"].split("+")


def _conv_out(case):
    ext = case["dil"] * (case["r"] - 1) + 1
    return tuple((d + 2 * case["pad"] - ext) // case["stride"] + 1 for d in (case["h"], case["w"]))


def _convt_out(case):
    return tuple((d - 1) * case["stride"] - 2 * case["pad"] + case["r"] + case["opad"] for d in (case["h"], case["w"]))


def _prepare_conv(case, gen, dt):
    n, c, k, r = case["n"], case["c"], case["k"], case["r"]
    ho, wo = _conv_out(case)
    std = (2.0 / (c * r * r)) ** 0.5
    bias = _normal(gen, (k,), torch.float32, 0.1) if _has(case, "bias") else None
    if case["via"] == "nhwc":
        x = _normal(gen, (n, case["h"], case["w"], c), dt)
        w = _normal(gen, (k, r, r, c), dt, std)
        res = _normal(gen, (n, ho, wo, k), dt) if _has(case, "residual") else None
    else:
        x = _normal(gen, (n, c, case["h"], case["w"]), dt)
        w = _normal(gen, (k, c, r, r), dt, std)
        res = _normal(gen, (n, k, ho, wo), dt) if _has(case, "residual") else None
    state = {"x": x, "w": w, "bias": bias, "res": res}
    if case["via"] == "module":
        m = tnn.TraceaConv2d(c, k, r, stride=case["stride"], padding=case["pad"], dilation=case["dil"],
                             bias=bias is not None, device="cuda", dtype=dt)
        with torch.no_grad():
            m.weight.copy_(w)
            if bias is not None:
                m.bias.copy_(bias)
        state["module"] = m
    return state


def _prepare_chain(case, gen, dt):
    n = case["n"]
    specs = resnet50.resnet50_convs() if case["kind"] == "stack" else resnet50.stage3_bottleneck()
    cl = torch.channels_last
    if case["kind"] == "stack":
        inputs = {"image": _normal(gen, (n, 224, 224, 3), dt).permute(0, 3, 1, 2),
                  "pooled": _normal(gen, (n, 64, 56, 56), dt).abs().contiguous(memory_format=cl)}
    else:
        inputs = {"input": _normal(gen, (n, 1024, 14, 14), dt).abs().contiguous(memory_format=cl)}
    weights = {}
    for sp in specs:
        weights[sp.name] = (_normal(gen, (sp.K, sp.C, sp.R, sp.S), torch.float32, (2.0 / (sp.C * sp.R * sp.S)) ** 0.5),
                            _normal(gen, (sp.K,), torch.float32, 0.05))
    stack = runner.ConvStack(specs, n, case["dtype"], inputs=inputs, weights=weights)
    if case["replay"]:
        stack.capture()
    return {"stack": stack}


def prepare(case, seed):
    gen, dt = _gen(seed), _DT[case["dtype"]]
    kind = case["kind"]
    if kind in ("block", "stack"):
        return dict(_prepare_chain(case, gen, dt), case=case)
    if kind == "conv":
        return dict(_prepare_conv(case, gen, dt), case=case)
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        w = _normal(gen, (n, k), dt, k ** -0.5).t() if case["w"] == "nk" else _normal(gen, (k, n), dt, k ** -0.5)
        return {"case": case, "x": _normal(gen, (m, k), dt), "w": w,
                "bias": _normal(gen, (n,), torch.float32, 0.1) if _has(case, "bias") else None,
                "res": _normal(gen, (m, n), dt) if _has(case, "residual") else None}
    c, k, r = case["c"], case["k"], case["r"]
    ho, wo = _convt_out(case)
    taps = max(1.0, (r / case["stride"]) ** 2)
    return {"case": case, "x": _normal(gen, (case["n"], case["h"], case["w"], c), dt),
            "w": _normal(gen, (k, r, r, c), dt, (2.0 / (c * taps)) ** 0.5),
            "bias": _normal(gen, (k,), torch.float32, 0.1) if _has(case, "bias") else None,
            "res": _normal(gen, (case["n"], ho, wo, k), dt) if _has(case, "residual") else None}


# ---------------------------------------------------------------------------------------------------- one pass
def run(state):
    case = state.get("case")
    kind = case["kind"]
    if kind in ("block", "stack"):
        stack = state["stack"]
        out = stack.replay() if case["replay"] else stack.forward()
        # the network's first layer feeds a pooling that is not part of the stack: its output is a result too
        return {"out": out, "stem": stack.tensors["stem"]} if kind == "stack" else out
    epi = case["epilogue"] or None
    if kind == "gemm":
        return ops.gemm(state["x"], state["w"], state["bias"], epi, state["res"])
    if kind == "conv_transpose":
        return ops.conv_transpose2d(state["x"], state["w"], state["bias"], state["res"], epi, case["stride"],
                                    case["pad"], case["opad"])
    if case["via"] == "nhwc":
        return ops.conv2d(state["x"], state["w"], state["bias"], state["res"], epi, case["stride"], case["pad"],
                          case["dil"])
    if case["via"] == "nchw":
        return ops.conv2d_nchw(state["x"], state["w"], state["bias"], state["res"], case["stride"], case["pad"],
                               case["dil"], 1, epi)
    with torch.no_grad():
        return state["module"](state["x"])


# ---------------------------------------------------------------------------------------------------- what a pass needs
def work(case):
    es = 4 if case["dtype"] == "f32" else 2
    kind = case["kind"]
    if kind in ("block", "stack"):
        # every layer's output is a tensor that the chain owns and hands out: each is written once and read once
        specs = resnet50.resnet50_convs() if kind == "stack" else resnet50.stage3_bottleneck()
        return {"bytes": sum(resnet50.conv_bytes(s, case["n"], es) for s in specs),
                "flops": sum(resnet50.conv_flops(s, case["n"]) for s in specs)}
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        x, w, out, flops = m * k, n * k, m * n, 2.0 * m * n * k
        ch = n
    elif kind == "conv":
        ho, wo = _conv_out(case)
        n, c, k, r = case["n"], case["c"], case["k"], case["r"]
        # a strided 1x1 layer only reads the pixels that it samples
        x = n * c * (ho * wo if r == 1 and case["pad"] == 0 else case["h"] * case["w"])
        w, out, flops = k * c * r * r, n * k * ho * wo, 2.0 * n * ho * wo * k * c * r * r
        ch = k
    else:
        ho, wo = _convt_out(case)
        n, c, k, r = case["n"], case["c"], case["k"], case["r"]
        # every input pixel meets every tap; taps that fall outside the output are not needed, but are few
        x, w, out = n * c * case["h"] * case["w"], k * c * r * r, n * k * ho * wo
        flops = 2.0 * n * case["h"] * case["w"] * c * k * r * r
        ch = k
    nbytes = (x + w + out * (2 if _has(case, "residual") else 1)) * es + (4 * ch if _has(case, "bias") else 0)
    return {"bytes": float(nbytes), "flops": float(flops)}


# Relative 2-norm errors against 64-bit results over the listed and 80 drawn cases: 1.67e-3 (bf16) and 2.1e-4 (f16), one
# rounding of the output; up to 8.9e-4 for fp32 storage, whose inputs lose bits to TF32. Four times that is stated. A
# chain of layers rounds between them: measured against the same layers with fp32 sums in another library, the block
# differs by less than one more rounding, the 53-layer stack by 8.5e-3 (bf16) and 1.3e-3 (f16).
_REL = {"bf16": 7e-3, "f16": 9e-4, "f32": 3.5e-3}
_REL_STACK = {"bf16": 3.4e-2, "f16": 5e-3}


def tolerance(case):
    return {"rel": (_REL_STACK if case["kind"] == "stack" else _REL)[case["dtype"]]}
