"""What a program that serves a quantized transformer has this library do, as timed cases.

A case is one pass through the public entry points (`kaio_b200.ops`, `kaio_b200.ffn.FfnInt4`):
decode steps and prefills of W4A16, W8A16 and W8A8 projections, the feed-forward chain, and
attention over a prompt or over a cache.  The listed sizes are those of the 7B and 70B layers the
benchmark and the tests use and of the small shapes the tests carry; `draw` spreads the same
operations over the ranges around them, with ragged row counts and widths that no tile divides.
"""
import math

import torch

from kaio_b200 import ops
from kaio_b200.ffn import FfnInt4

GROUP = 128


def listed():
    return [
        # one token through the 7B up projection: the smallest decode step, W4A16
        {"name": "int4 decode m1", "kind": "int4", "m": 1, "n": 11008, "k": 4096},
        # eight sequences' next token through the 7B fused QKV projection, W4A16
        {"name": "qkv int4 decode m8", "kind": "qkv_int4", "m": 8, "n": 4096, "k": 4096},
        # sixteen sequences' next token through the 70B feed-forward block, W4A16
        {"name": "ffn int4 decode m16", "kind": "ffn", "m": 16, "hidden": 8192, "inter": 28672},
        # a batch of 64 tokens through a small model's fused QKV projection, W8A16
        {"name": "qkv int8 m64", "kind": "qkv_int8", "m": 64, "n": 2048, "k": 2048},
        # a small square W8A8 product, where the launch counts
        {"name": "int8 m512", "kind": "int8", "m": 512, "n": 512, "k": 512},
        # a ragged prompt through the 7B fused QKV projection, activations quantised on the way, W8A8
        {"name": "qkv w8a8 m1000", "kind": "qkv_w8a8", "m": 1000, "n": 4096, "k": 4096},
        # a ragged batch through the 70B down projection, W4A16
        {"name": "int4 m250", "kind": "int4", "m": 250, "n": 8192, "k": 28672},
        # a 4096-token prefill through the 7B up projection: quantise the rows, then W8A8
        {"name": "linear w8a8 m4096", "kind": "linear_w8a8", "m": 4096, "n": 11008, "k": 4096},
        # a 4096-token prefill through the 70B feed-forward block, the largest call
        {"name": "ffn int4 m4096", "kind": "ffn", "m": 4096, "hidden": 8192, "inter": 28672},
        # single-head causal attention at the drop-in entry point's longest sequence
        {"name": "attention tc 384", "kind": "attention_tc", "seq": 384, "d": 128, "causal": True},
        # causal prefill attention of the 7B layer over eight 2048-token prompts
        {"name": "attention prefill", "kind": "attention", "batch": 8, "heads": 32, "seq_q": 2048, "seq_k": 2048, "d": 128, "causal": True},
        # one new token of eight sequences attending to its cache
        {"name": "attention decode", "kind": "attention", "batch": 8, "heads": 32, "seq_q": 1, "seq_k": 2000, "d": 128, "causal": False},
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], spread evenly over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["int4", "int4", "qkv_int4", "ffn", "ffn", "qkv_int8", "int8", "qkv_w8a8", "linear_w8a8", "attention_tc", "attention", "attention"])
    if kind == "int4":
        return {"kind": kind, "m": _log(rng, 1, 1024), "n": _log(rng, 1024, 28672, 8), "k": _log(rng, 1024, 28672, 128)}
    if kind in ("qkv_int4", "qkv_int8", "qkv_w8a8"):
        return {"kind": kind, "m": _log(rng, 1, 4096), "n": _log(rng, 1024, 8192, 16), "k": _log(rng, 1024, 8192, 128)}
    if kind == "ffn":
        return {"kind": kind, "m": _log(rng, 1, 2048), "hidden": _log(rng, 1024, 8192, 128), "inter": _log(rng, 2048, 28672, 128)}
    if kind == "int8":
        return {"kind": kind, "m": _log(rng, 64, 4096), "n": _log(rng, 64, 4096, 16), "k": _log(rng, 64, 4096, 32)}
    if kind == "linear_w8a8":
        return {"kind": kind, "m": _log(rng, 1, 4096), "n": _log(rng, 1024, 28672, 16), "k": _log(rng, 1024, 11008, 32)}
    if kind == "attention_tc":
        return {"kind": kind, "seq": _log(rng, 64, 384, 16), "d": rng.choice([64, 128, 128]), "causal": rng.random() < 0.5}
    batch, heads, d = rng.choice([1, 2, 4, 8]), rng.choice([8, 16, 32]), rng.choice([64, 128, 128, 128])
    if rng.random() < 0.5:
        return {"kind": kind, "batch": batch, "heads": heads, "seq_q": 1, "seq_k": _log(rng, 128, 8192), "d": d, "causal": False}
    # head size 64 is bounded in length so that no drawn case costs more than the largest listed one
    seq = _log(rng, 128, 2048 if d == 128 else 512)
    return {"kind": kind, "batch": batch, "heads": heads, "seq_q": seq, "seq_k": seq, "d": d, "causal": rng.random() < 0.75}


def _normal(gen, n, scale=1.0, dtype=torch.float16):
    return torch.randn(n, generator=gen, device="cuda").mul_(scale).to(dtype)


def _int4_weight(dev, gen, k, n):
    """Normally distributed weights, quantised and packed as a checkpoint converter does."""
    w = torch.randn(k * n, generator=gen, device="cuda").mul_(0.02)
    packed = torch.empty(k // 8 * n, dtype=torch.int32, device="cuda")
    scales = torch.empty(k // GROUP * n, dtype=torch.float16, device="cuda")
    ops.quantize_pack_int4(dev, w, packed, scales, k, n)
    return packed, scales


def _int8(gen, n):
    return torch.randn(n, generator=gen, device="cuda").mul_(32.0).round_().clamp_(-127, 127).to(torch.int8)


def _scales(gen, n):
    return torch.rand(n, generator=gen, device="cuda").mul_(0.009).add_(0.001)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dev, kind = ops.KaioDevice(0), case["kind"]
    s = {"case": case, "dev": dev}
    if kind in ("attention_tc", "attention"):
        if kind == "attention_tc":
            nq = nk = case["seq"] * case["d"]
        else:
            width = case["heads"] * case["d"]
            nq, nk = case["batch"] * case["seq_q"] * width, case["batch"] * case["seq_k"] * width
        s["q"], s["k"], s["v"] = _normal(gen, nq), _normal(gen, nk), _normal(gen, nk)
        s["out"] = torch.empty(nq, dtype=torch.float32 if kind == "attention_tc" else torch.float16, device="cuda")
        return s
    m = case["m"]
    if kind == "ffn":
        h, i = case["hidden"], case["inter"]
        w = _int4_weight(dev, gen, h, i) + _int4_weight(dev, gen, h, i) + _int4_weight(dev, gen, i, h)
        s["ffn"] = FfnInt4(ops, dev, h, i, *w, max_m=m)
        s["ffn"].enable_fused_silu()
        s["x"] = _normal(gen, m * h)
        return s
    n, k = case["n"], case["k"]
    if kind == "int4":
        s["x"], s["w"] = _normal(gen, m * k), _int4_weight(dev, gen, k, n)
        s["out"] = torch.empty(m * n, dtype=torch.float16, device="cuda")
    elif kind == "int8":
        s["x"], s["w"] = _int8(gen, m * k), _int8(gen, k * n)
        s["out"] = torch.empty(m * n, dtype=torch.float32, device="cuda")
    elif kind == "linear_w8a8":
        s["x"], s["w"], s["w_scale"] = _normal(gen, m * k, dtype=torch.float32), _int8(gen, k * n), _scales(gen, n)
        s["q"] = torch.empty(m * k, dtype=torch.int8, device="cuda")
        s["q_scale"] = torch.empty(m, dtype=torch.float32, device="cuda")
        s["out"] = torch.empty(m * n, dtype=torch.float32, device="cuda")
    else:
        s["x"] = _normal(gen, m * k)
        if kind == "qkv_int4":
            pairs = [_int4_weight(dev, gen, k, n) for _ in range(3)]
            s["w"], s["scales"] = [p[0] for p in pairs], [p[1] for p in pairs]
        else:
            s["w"] = [_int8(gen, k * n) for _ in range(3)]
            s["scales"] = [_scales(gen, n) for _ in range(3)] if kind == "qkv_w8a8" else [0.001, 0.0015, 0.002]
        s["out"] = [torch.empty(m * n, dtype=torch.float16, device="cuda") for _ in range(3)]
    return s


def run(s):
    case, dev = s["case"], s["dev"]
    kind = case["kind"]
    if kind == "int4":
        ops.matmul_int4(dev, s["x"], *s["w"], s["out"], case["m"], case["n"], case["k"], GROUP)
    elif kind == "qkv_int4":
        ops.qkv_project_int4(dev, s["x"], *s["w"], *s["scales"], *s["out"], case["m"], case["n"], case["k"], GROUP)
    elif kind == "ffn":
        return s["ffn"].run(s["x"], case["m"])
    elif kind == "qkv_int8":
        ops.qkv_project_int8(dev, s["x"], *s["w"], *s["scales"], *s["out"], case["m"], case["n"], case["k"])
    elif kind == "int8":
        ops.matmul_int8(dev, s["x"], s["w"], s["out"], 0.001, case["m"], case["n"], case["k"])
    elif kind == "qkv_w8a8":
        ops.qkv_project_w8a8(dev, s["x"], *s["w"], *s["scales"], *s["out"], case["m"], case["n"], case["k"])
    elif kind == "linear_w8a8":
        ops.quantize_rows_int8(dev, s["x"], s["q"], s["q_scale"], case["m"], case["k"])
        ops.matmul_int8_scaled(dev, s["q"], s["w"], s["out"], s["q_scale"], s["w_scale"], case["m"], case["n"], case["k"])
        return {"out": s["out"], "q": s["q"], "q_scale": s["q_scale"]}
    elif kind == "attention_tc":
        f = ops.attention_tc_causal if case["causal"] else ops.attention_tc
        f(dev, s["q"], s["k"], s["v"], s["out"], case["seq"], case["seq"], case["d"], case["d"])
    else:
        ops.attention_mha_f16(dev, s["q"], s["k"], s["v"], s["out"], case["batch"], case["heads"], case["seq_q"], case["seq_k"],
                              case["d"], case["heads"] * case["d"], case["causal"])
    return s["out"]


def _int4_bytes(k, n):
    return k * n // 2 + 2 * (k // GROUP) * n


def work(case):
    kind = case["kind"]
    if kind in ("attention_tc", "attention"):
        if kind == "attention_tc":
            pairs, sq, sk, out = 1, case["seq"], case["seq"], 4
        else:
            pairs, sq, sk, out = case["batch"] * case["heads"], case["seq_q"], case["seq_k"], 2
        scores = sq * (sq + 1) // 2 if case["causal"] else sq * sk
        return {"bytes": pairs * case["d"] * (2 * sq + 4 * sk + out * sq), "flops": 4 * pairs * case["d"] * scores}
    m = case["m"]
    if kind == "ffn":
        h, i = case["hidden"], case["inter"]
        return {"bytes": 3 * _int4_bytes(h, i) + 2 * m * h + 4 * m * h, "flops": 6 * m * h * i}
    n, k = case["n"], case["k"]
    if kind == "int4":
        return {"bytes": _int4_bytes(k, n) + 2 * m * k + 2 * m * n, "flops": 2 * m * n * k}
    if kind == "int8":
        return {"bytes": m * k + k * n + 4 * m * n, "flops": 2 * m * n * k}
    if kind == "linear_w8a8":
        return {"bytes": 4 * m * k + m * k + 4 * m + k * n + 4 * n + 4 * m * n, "flops": 2 * m * n * k}
    weight = _int4_bytes(k, n) if kind == "qkv_int4" else k * n + (4 * n if kind == "qkv_w8a8" else 0)
    return {"bytes": 2 * m * k + 3 * weight + 6 * m * n, "flops": 6 * m * n * k}


def tolerance(case):
    kind = case["kind"]
    if kind in ("int8", "linear_w8a8"):
        # exact integer sums, then one or two f32 multiplications
        return {"rel": 1e-6}
    if kind == "qkv_w8a8":
        # the same, narrowed to f16
        return {"rel": 1e-3}
    if kind == "ffn":
        # f16 weights, f16 projections and an f16 activation between the products
        return {"rel": 3e-3}
    if kind in ("attention_tc", "attention"):
        # f16 probabilities
        return {"rel": 3e-3}
    # f16 weights and outputs, f32 sums
    return {"rel": 1e-3}
