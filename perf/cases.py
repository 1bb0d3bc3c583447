"""The calls this library is measured on: what a program that uses it has it do, over the range it does it in.

Every case goes through the Python entry points of ``codegendemo_b200.kcg.matmul_op`` (``matmul``, ``bmm``,
``attention_fused``) on GPU tensors, exactly as a program calls them: operands in hand, result allocated by the call.
"""
import math

import torch

from codegendemo_b200.kcg import matmul_op

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def _mm(name, m, n, k, dtype, form="plain"):
    return {"name": name, "op": "matmul", "m": m, "n": n, "k": k, "dtype": dtype, "form": form}


def _attn(name, heads, sq, sk, d, dtype):
    return {"name": name, "op": "attention", "heads": heads, "sq": sq, "sk": sk, "d": d, "dtype": dtype}


def listed():
    return [
        # smallest product: a small projection or a classifier head; launch and latency are all of it
        _mm("small_bf16", 256, 1024, 512, "bf16"),
        # one decode step of a batch of 128 through a square projection: streams the weights once
        _mm("skinny_bf16", 128, 4096, 4096, "bf16"),
        # the same through a weight stored out_features x in_features (how linear layers keep it), 512 rows
        _mm("linear_bf16", 512, 4096, 11008, "bf16", "b_transposed"),
        # prefill of 2048 tokens into a wide layer, bias and ReLU fused into the store
        _mm("prefill_fp16_bias_relu", 2048, 11008, 4096, "fp16", "bias_relu"),
        # no size a multiple of the large tiles
        _mm("ragged_bf16", 1664, 2752, 1472, "bf16"),
        # largest product: the slab a single GPU runs of the 32768-row problem
        _mm("slab_bf16", 32768, 8192, 8192, "bf16"),
        # fp32 at fp32 accuracy: small square, large square, and a rectangle with few rows
        _mm("small_fp32", 1024, 1024, 1024, "fp32"),
        _mm("square_fp32", 4096, 4096, 4096, "fp32"),
        _mm("rect_fp32", 512, 11008, 4096, "fp32"),
        # per-expert or per-group products: many middling ones in one call
        {"name": "bmm_bf16", "op": "bmm", "batch": 24, "m": 384, "n": 768, "k": 640, "dtype": "bf16"},
        # attention over a whole prompt
        _attn("attention_prefill_bf16", 32, 4096, 4096, 128, "bf16"),
        # attention of one new token per head over a long cache
        _attn("attention_decode_bf16", 32, 1, 8192, 128, "bf16"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _step(rng, lo, hi, step):
    return max(lo, min(hi, int(round(_log(rng, lo, hi) / step)) * step))


# what a drawn case may cost, in floating point operations: the largest listed product, and as much time in fp32
_MOST = {"bf16": 2.0 * 32768 * 8192 * 8192, "fp16": 2.0 * 32768 * 8192 * 8192, "fp32": 2.0 * 8192 * 8192 * 4096}


def draw(rng):
    kind = rng.choices(["matmul16", "matmul32", "bmm", "attention"], [6, 3, 1, 2])[0]
    while True:
        # widths of real layers: mostly multiples of 256 or 128, now and then only of 64
        wn, wk = rng.choice([64, 128, 256, 256]), rng.choice([64, 128, 256, 256])
        if kind == "matmul16":
            c = {"op": "matmul", "m": _step(rng, 128, 32768, 128), "n": _step(rng, 512, 16384, wn),
                 "k": _step(rng, 256, 16384, wk), "dtype": rng.choice(["bf16", "bf16", "fp16"]),
                 "form": rng.choice(["plain", "plain", "plain", "bias_relu", "b_transposed", "strided"])}
        elif kind == "matmul32":
            c = {"op": "matmul", "m": _step(rng, 128, 8192, 128), "n": _step(rng, 512, 11008, wn),
                 "k": _step(rng, 256, 11008, wk), "dtype": "fp32", "form": rng.choice(["plain", "plain", "bias_relu"])}
        elif kind == "bmm":
            c = {"op": "bmm", "batch": int(_log(rng, 4, 64)), "m": _step(rng, 128, 2048, 128),
                 "n": _step(rng, 256, 2048, wn), "k": _step(rng, 256, 2048, wk),
                 "dtype": rng.choice(["bf16", "bf16", "fp16"])}
        else:
            # prompts of any length, and (every other draw) a few new tokens over a cache of any length
            sk = int(_log(rng, 256, 16384))
            sq = int(_log(rng, 1, 16)) if rng.random() < 0.5 else int(_log(rng, 64, 8192))
            c = {"op": "attention", "heads": int(_log(rng, 8, 128)), "sq": sq, "sk": sk,
                 "d": rng.choice([64, 128, 128]), "dtype": rng.choice(["bf16", "bf16", "fp16"])}
        if work(c)["flops"] <= _MOST[c["dtype"]] * (0.4 if kind == "attention" else 1.0):
            return c


def _values(gen, shape, dtype, scale):
    """Seeded entries: normal(0,1) * scale for the 16-bit types, uniform[-1,1) for fp32."""
    if dtype == torch.float32:
        return torch.rand(shape, generator=gen, device="cuda", dtype=torch.float32) * 2.0 - 1.0
    return (torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32) * scale).to(dtype)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    dt = DTYPES[case["dtype"]]
    s = {"case": case}
    if case["op"] == "attention":
        h, d = case["heads"], case["d"]
        s["q"] = _values(gen, (h, case["sq"], d), dt, 1.0)
        s["k"] = _values(gen, (h, case["sk"], d), dt, 1.0)
        s["v"] = _values(gen, (h, case["sk"], d), dt, 1.0)
        return s
    m, n, k = case["m"], case["n"], case["k"]
    scale = 1.0 / math.sqrt(k)
    if case["op"] == "bmm":
        s["a"] = _values(gen, (case["batch"], m, k), dt, scale)
        s["b"] = _values(gen, (case["batch"], k, n), dt, scale)
        return s
    form = case["form"]
    if form == "strided":  # operands that are column blocks of wider tensors (one head's or one gate's part)
        s["a"] = _values(gen, (m, 2 * k), dt, scale)[:, k:]
        s["b"] = _values(gen, (k, n + 512), dt, scale)[:, 256:256 + n]
    else:
        s["a"] = _values(gen, (m, k), dt, scale)
        s["b"] = _values(gen, (n, k) if form == "b_transposed" else (k, n), dt, scale)
    if form == "bias_relu":
        s["bias"] = _values(gen, (n,), dt, scale)
    return s


def run(s):
    case = s["case"]
    if case["op"] == "attention":
        return matmul_op.attention_fused(s["q"], s["k"], s["v"])
    if case["op"] == "bmm":
        return matmul_op.bmm(s["a"], s["b"])
    if case["form"] == "bias_relu":
        return matmul_op.matmul(s["a"], s["b"], bias=s["bias"], relu=True)
    if case["form"] == "b_transposed":
        return matmul_op.matmul(s["a"], s["b"], b_transposed=True)
    return matmul_op.matmul(s["a"], s["b"])


def work(case):
    eb = 4 if case["dtype"] == "fp32" else 2
    if case["op"] == "attention":
        h, sq, sk, d = case["heads"], case["sq"], case["sk"], case["d"]
        return {"bytes": eb * h * d * (2.0 * sq + 2.0 * sk), "flops": 4.0 * h * sq * sk * d}
    b, m, n, k = case.get("batch", 1), case["m"], case["n"], case["k"]
    bias = n if case.get("form") == "bias_relu" else 0
    return {"bytes": float(eb) * (b * (m * k + k * n + m * n) + bias), "flops": 2.0 * b * m * n * k}


def tolerance(case):
    """About four times the error of the path against the same product in 64 bits (2-norm, and the largest one)."""
    if case["op"] == "attention":
        return {"bf16": {"rel": 1e-2, "max": 4e-2}, "fp16": {"rel": 1.2e-3, "max": 5e-3}}[case["dtype"]]
    return {"bf16": {"rel": 7e-3, "max": 1.6e-2}, "fp16": {"rel": 9e-4, "max": 2e-3},
            "fp32": {"rel": 4e-6, "max": 1.5e-5}}[case["dtype"]]
