"""What a program does with this package, as timed cases: the W4A4 layer, the quantizer, the packed-int4 product and the
dequantizer, each through the public entry point such a program calls.

Sizes are the projection shapes the benchmark and the tests use: hidden 4096, intermediate 14336 or 11008, and 28672 wide
rows, from one decode token to prefill chunks of thousands.  Activations are N(0, 1) with 1 % of the channels
multiplied by 50, transforms are random orthogonal, weights are N(0, 0.02) quantized per output channel with absmax / 7.
"""
from __future__ import annotations

import math

import torch

import quant_ops_b200 as quant_ops

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
ITEM = {"bf16": 2, "fp16": 2, "fp32": 4}

# (in, out) features of the layers: attention and MLP projections of the benchmark's stack, and the 11008-wide MLP
LAYERS = [(4096, 4096), (4096, 1024), (4096, 14336), (14336, 4096), (4096, 11008), (11008, 4096)]
WIDTHS = [1024, 3072, 4096, 5120, 8192, 11008, 14336, 28672]
MOST_ROWS = 8192
MOST_VALUES = 8192 * 4096  # of one activation matrix
MOST_MACS = 4096 * 14336 * 4096


def _linear(tokens, k, n_out, dtype="bf16", bias=False, keep_int8=False):
    return {"op": "linear", "tokens": tokens, "k": k, "n_out": n_out, "dtype": dtype, "bias": bias, "keep_int8": keep_int8, "clip": 0.9}


def _quantize(tokens, k, dtype, pack, clip):
    return {"op": "quantize", "tokens": tokens, "k": k, "dtype": dtype, "pack": pack, "clip": clip}


def _matmul(tokens, k, n_out, layout, out):
    return {"op": "matmul", "tokens": tokens, "k": k, "n_out": n_out, "layout": layout, "out": out}


def _dequantize(tokens, k, pack):
    return {"op": "dequantize", "tokens": tokens, "k": k, "pack": pack}


def listed():
    return [
        # one decode step of one sequence through an attention projection: latency and launches
        dict(_linear(1, 4096, 4096), name="linear_1x4096x4096"),
        # a decode step of a small batch through the down projection: the packed weights once
        dict(_linear(16, 14336, 4096), name="linear_16x14336x4096"),
        # a large decode batch or a short prompt, between the weight-bound and the compute-bound sizes
        dict(_linear(256, 14336, 4096), name="linear_256x14336x4096"),
        # a prompt of odd length, float16 model with biases
        dict(_linear(777, 4096, 11008, dtype="fp16", bias=True), name="linear_777x4096x11008"),
        # a prefill chunk through the down projection: the largest
        dict(_linear(4096, 14336, 4096), name="linear_4096x14336x4096"),
        # the quantizer alone as its own operator: a small float16 batch to int8 codes
        dict(_quantize(128, 4096, "fp16", False, 1.0), name="quantize_128x4096_fp16"),
        # the benchmark's headline: a prefill chunk to packed codes
        dict(_quantize(8192, 4096, "bf16", True, 0.9), name="quantize_8192x4096_bf16"),
        # float32 activations, as a calibration or evaluation run has them
        dict(_quantize(2048, 4096, "fp32", False, 0.9), name="quantize_2048x4096_fp32"),
        # 28672-wide rows (the down-projection input of the largest dense models), odd token count
        dict(_quantize(1001, 28672, "bf16", True, 0.9), name="quantize_1001x28672_bf16"),
        # the packed product alone, weights kept [out, K/8] and passed as a transposed view
        dict(_matmul(4096, 4096, 4096, "weights", "fp16"), name="matmul_4096x4096x4096"),
        # the same operator with weights in its own [K/8, out] layout and an odd row count
        dict(_matmul(333, 4096, 14336, "columns", "fp16"), name="matmul_333x4096x14336_columns"),
        # codes back to float32, as a check of the quantizer's error or a float fallback does
        dict(_dequantize(8192, 4096, True), name="dequantize_8192x4096"),
    ]


def _rows(rng, most):
    """Row counts spread over the logarithm of 1 .. most; about half of the larger ones are odd."""
    t = int(round(math.exp(rng.uniform(0.0, math.log(most)))))
    if t > 8 and rng.random() < 0.4:
        t = t // 8 * 8
    return max(1, min(most, t))


def draw(rng):
    op = rng.choice(["linear", "linear", "linear", "quantize", "quantize", "matmul", "matmul", "dequantize"])
    if op == "linear":
        k, n_out = rng.choice(LAYERS)
        return _linear(_rows(rng, min(MOST_ROWS, MOST_MACS // (k * n_out))), k, n_out, rng.choice(["bf16", "bf16", "fp16"]),
                       rng.random() < 0.3, rng.random() < 0.3)
    if op == "matmul":
        k, n_out = rng.choice(LAYERS)
        if rng.random() < 0.3:
            n_out -= 8 * rng.randrange(1, 32)
        return _matmul(_rows(rng, min(MOST_ROWS, MOST_MACS // (k * n_out))), k, n_out, rng.choice(["weights", "weights", "columns"]),
                       rng.choice(["fp16", "bf16"]))
    k = rng.choice(WIDTHS)
    tokens = _rows(rng, min(MOST_ROWS, MOST_VALUES // k))
    if op == "dequantize":
        return _dequantize(tokens, k, rng.random() < 0.7)
    dtype = rng.choice(["bf16", "bf16", "fp16", "fp32"])
    if dtype == "fp32":
        k = min(k, 14336)
    return _quantize(tokens, k, dtype, rng.random() < 0.6, rng.choice([1.0, 0.9]))


# ---- inputs ----------------------------------------------------------------------------------------------------------
def _gen(seed, salt):
    return torch.Generator(device="cuda").manual_seed(seed * 1000003 + salt)


def _activations(case, seed):
    g = _gen(seed, 1)
    x = torch.randn(case["tokens"], case["k"], device="cuda", generator=g)
    hot = torch.randperm(case["k"], device="cuda", generator=g)[: case["k"] // 100]
    x[:, hot] *= 50
    return x.to(DTYPES[case["dtype"]])


def _transforms(case, seed):
    g = torch.Generator().manual_seed(seed * 1000003 + 2)
    m, n = quant_ops.get_decompose_dim(case["k"])
    return [torch.linalg.qr(torch.randn(s, s, dtype=torch.float64, generator=g)).Q.contiguous().to("cuda").to(DTYPES[case["dtype"]])
            for s in (m, n)]


def _weights(case, seed):
    """int8 codes [out, K] and float32 scales [out] of N(0, 0.02) weights."""
    w = torch.randn(case["n_out"], case["k"], device="cuda", generator=_gen(seed, 3)) * 0.02
    scale = w.abs().amax(dim=1) / 7
    return torch.round(w / scale[:, None]).clamp_(-8, 7).to(torch.int8), scale


def _codes(case, seed):
    """int8 codes [tokens, K] spread as the quantizer's are, and float32 scales [tokens]."""
    g = _gen(seed, 4)
    z = torch.randn(case["tokens"], case["k"], device="cuda", generator=g)
    scale = z.abs().amax(dim=1) * (0.9 / 7)
    codes = torch.round(z / scale[:, None]).clamp_(-8, 7).to(torch.int8)
    return codes, scale * (4 + torch.rand(case["tokens"], device="cuda", generator=g))


def _pack(codes):
    """[rows, K] int8 codes -> [rows, K/8] int32, nibble i of a word = code + 8."""
    c = (codes.to(torch.int32) + 8).reshape(codes.shape[0], -1, 8)
    word = c[:, :, 0].clone()
    for i in range(1, 8):
        word |= c[:, :, i] << (4 * i)
    return word


def _bias(case, seed):
    return torch.randn(case["n_out"], device="cuda", generator=_gen(seed, 5)).to(DTYPES[case["dtype"]]) if case["bias"] else None


def prepare(case, seed):
    op = case["op"]
    if op == "linear":
        codes, scale = _weights(case, seed)
        left, right = _transforms(case, seed)
        layer = quant_ops.W4A4Linear(case["k"], case["n_out"], bias=case["bias"], clip_ratio=case["clip"], dtype=DTYPES[case["dtype"]],
                                     device="cuda", keep_int8_weights=case["keep_int8"])
        layer.load_quantized(codes, scale, left, right, _bias(case, seed))
        return {"op": op, "layer": layer, "x": _activations(case, seed)}
    if op == "quantize":
        left, right = _transforms(case, seed)
        return {"op": op, "x": _activations(case, seed), "left": left, "right": right, "clip": case["clip"], "pack": case["pack"]}
    codes, sa = _codes(case, seed)
    if op == "dequantize":
        return {"op": op, "codes": _pack(codes) if case["pack"] else codes, "scales": sa, "pack": case["pack"]}
    w, sb = _weights(case, seed)
    b = _pack(w).t()
    return {"op": op, "a": _pack(codes), "b": b.contiguous() if case["layout"] == "columns" else b, "sa": sa, "sb": sb,
            "out": DTYPES[case["out"]]}


def run(state):
    op = state["op"]
    if op == "linear":
        return state["layer"](state["x"])
    if op == "quantize":
        return quant_ops.flatquant_dynamic_quantize(state["x"], state["left"], state["right"], state["clip"], state["pack"])
    if op == "dequantize":
        return quant_ops.dequantize_int4(state["codes"], state["scales"], state["pack"])
    if state["out"] == torch.float16:
        return quant_ops.int4_matmul(state["a"], state["b"], state["sa"], state["sb"])
    return quant_ops.int4_matmul_ex(state["a"], state["b"], state["sa"], state["sb"], state["out"])


def work(case):
    t, k = case["tokens"], case["k"]
    op = case["op"]
    if op == "dequantize":
        return {"bytes": t * k * (0.5 if case["pack"] else 1) + 4 * t + 4 * t * k, "flops": t * k}
    if op == "matmul":
        n = case["n_out"]
        return {"bytes": (t + n) * k / 2 + 4 * (t + n) + 2 * t * n, "flops": 2 * t * k * n}
    m, n = quant_ops.get_decompose_dim(k)
    item = ITEM[case["dtype"]]
    rows = t * k * item + (m * m + n * n) * item
    transform = 2 * t * k * (m + n)
    if op == "quantize":
        return {"bytes": rows + t * k * (0.5 if case["pack"] else 1) + 4 * t, "flops": transform}
    return {"bytes": rows + case["n_out"] * (k / 2 + 4) + 2 * t * case["n_out"], "flops": transform + 2 * t * k * case["n_out"]}


def tolerance(case):
    op = case["op"]
    if op in ("dequantize", "matmul"):
        return "exact"  # whole-number sums, then one or two float32 products in a given order
    if op == "quantize":
        if case["dtype"] == "fp32":
            # another summation order moves a quotient across a rounding boundary on about 2e-6 of the codes (of the
            # packed words, eight times that), and a scale by a few units in the last place
            return {"rel": 1e-6, "max": 4e-6, "differ": 1e-4}
        # another summation order can round a transformed value to its neighbour in 16 bits: where that value is the
        # row's largest the scale moves by one unit in the last place and with it a few codes of the row
        return {"rel": 2e-3, "max": 8e-3 if case["dtype"] == "bf16" else 1e-3, "differ": 4e-3}
    # the layer: the quantizer's ties change a few codes by one, the product's output is rounded to 16 bits (seen between two
    # summation orders: 1.1e-3 and, where a whole row's scale moved, 0.2)
    return {"rel": 5e-3, "max": 0.8}


def _rounded(v, dtype):
    """float64 values rounded to the activation dtype (the operator is defined with these roundings)."""
    return v if dtype == "fp32" else v.to(DTYPES[dtype]).to(torch.float64)


def _exact_quantize(x, left, right, clip, dtype):
    """Codes and scales as float64, every sum in 64 bits, rounded to the activation dtype where the operator rounds."""
    m, n = left.shape[0], right.shape[0]
    y = _rounded(x.to(torch.float64).reshape(-1, m, n) @ right.to(torch.float64), dtype)
    z = _rounded(left.to(torch.float64).t() @ y, dtype).reshape(x.shape)
    top = torch.maximum(_rounded(z.amax(dim=1) * clip, dtype), _rounded(z.amin(dim=1) * clip, dtype).abs())
    scale = _rounded(top / 7, dtype)
    return torch.round(_rounded(z / scale[:, None], dtype)).clamp_(-8, 7), scale


def exact(case, seed):
    op = case["op"]
    if op == "dequantize":
        codes, scale = _codes(case, seed)
        return codes.to(torch.float64) * scale.to(torch.float64)[:, None]
    if op == "matmul":
        a, sa = _codes(case, seed)
        w, sb = _weights(case, seed)
        return (a.to(torch.float64) @ w.to(torch.float64).t()) * sa.to(torch.float64)[:, None] * sb.to(torch.float64)
    left, right = _transforms(case, seed)
    codes, scale = _exact_quantize(_activations(case, seed), left, right, case["clip"], case["dtype"])
    if op == "quantize":
        return None, scale
    w, sb = _weights(case, seed)
    y = (codes @ w.to(torch.float64).t()) * scale[:, None] * sb.to(torch.float64)
    bias = _bias(case, seed)
    return y if bias is None else y + bias.to(torch.float64)
