"""The work a user of this package has it do, as timed cases: FP8 linear layers, MoE grouped GEMMs, a whole
MoE feed-forward layer, and the quantise / dequantise pair on its own -- all through ``primus_turbo_b200.pytorch``.

Sizes are those of ``bench.py`` (its c1 .. c5 shapes and the per-rank shards of c4), of the tests' shape grid, or
generic.  Kinds of case (``"op"``):

  dense    ``gemm_fp8``: forward, or forward + both gradients; raw weights, or weights quantised once
  grouped  ``grouped_gemm_fp8``: the same over per-expert row groups of uneven (and empty) lengths
  moe      ``token_permute`` -> grouped GEMM -> ``swiglu_with_probs`` -> grouped GEMM -> ``token_unpermute``, both ways
  codec    ``quantize_fp8`` followed by ``dequantize_fp8`` (what an FP8 exchange does either side of the wire)
"""

import math

import torch

from primus_turbo_b200.pytorch.core.low_precision import (
    Float8QuantConfig,
    Format,
    ScaleDtype,
    ScalingGranularity,
    float8_e4m3,
    float8_e5m2,
)
from primus_turbo_b200.pytorch.core.quantized_tensor import create_quantized_weight
from primus_turbo_b200.pytorch.ops import dequantize_fp8, gemm_fp8, grouped_gemm_fp8, quantize_fp8
from primus_turbo_b200.pytorch.ops.activation import swiglu_with_probs
from primus_turbo_b200.pytorch.ops.moe import token_permute, token_unpermute

GRANULARITY = {
    "tensor": ScalingGranularity.TENSORWISE,
    "row": ScalingGranularity.ROWWISE,
    "block": ScalingGranularity.BLOCKWISE,
    "mx": ScalingGranularity.MX_BLOCKWISE,
}
BLOCK = {"tensor": None, "row": None, "block": 128, "mx": 32}
DTYPE = {"bf16": torch.bfloat16, "fp16": torch.float16}
FORMAT = {"e4m3": Format.E4M3, "hybrid": Format.HYBRID}


def _dense(name, gran, m, n, k, train, cached=False, trans_b=True, fmt="e4m3", dtype="bf16"):
    return {"name": name, "op": "dense", "gran": gran, "m": m, "n": n, "k": k, "train": train, "cached": cached,
            "trans_b": trans_b, "fmt": fmt, "dtype": dtype}


def _grouped(name, gran, g, rows, n, k, spread, train, cached=False, fmt="e4m3", dtype="bf16"):
    return {"name": name, "op": "grouped", "gran": gran, "groups": g, "rows": rows, "n": n, "k": k, "spread": spread,
            "train": train, "cached": cached, "fmt": fmt, "dtype": dtype}


def _moe(name, tokens, experts, topk, hidden, inter, fmt="e4m3"):
    return {"name": name, "op": "moe", "tokens": tokens, "experts": experts, "topk": topk, "hidden": hidden,
            "inter": inter, "fmt": fmt}


def _codec(name, gran, m, n, fp8="e4m3", dtype="bf16"):
    return {"name": name, "op": "codec", "gran": gran, "m": m, "n": n, "fp8": fp8, "dtype": dtype}


def listed():
    return [
        # bench.py's c1: the smallest call, a small projection in inference; bound by launches and host work
        _dense("dense_small_forward", "block", 256, 512, 1024, train=False),
        # a decode step of an MLP projection: few tokens against weights quantised when the model was loaded
        _dense("dense_decode", "tensor", 32, 14336, 4096, train=False, cached=True),
        # bench.py's c2: prefill of the same projection, weights quantised on the fly
        _dense("dense_prefill", "tensor", 8192, 14336, 4096, train=False),
        # bench.py's c3: a training step of a large square projection, per-row scales
        _dense("dense_train_row", "row", 16384, 8192, 8192, train=True),
        # a training micro-batch with a ragged token count and a width that is no multiple of the tiles; e5m2 gradients
        _dense("dense_train_ragged", "block", 3001, 5760, 2880, train=True, trans_b=False, fmt="hybrid"),
        # the two-GPU shard of bench.py's c4: the largest expert layer, training, weights quantised every step
        _grouped("grouped_train_large", "block", 128, 32768, 4096, 7168, "softmax", train=True),
        # bench.py's c5: many narrow experts with a heavy-tailed load and empty groups, training
        _grouped("grouped_train_skewed", "block", 128, 32768, 1536, 2048, "zipf", train=True),
        # decode through one rank's experts: a handful of rows each, weights quantised when the model was loaded
        _grouped("grouped_decode", "block", 32, 256, 4096, 7168, "softmax", train=False, cached=True),
        # few large experts with one scale per tensor (the default configuration), e5m2 gradients
        _grouped("grouped_train_tensor", "tensor", 8, 8192, 7168, 2048, "softmax", train=True, fmt="hybrid"),
        # the eight-GPU shard of c4 in the MXFP8 format, training
        _grouped("grouped_train_mx", "mx", 32, 8192, 4096, 7168, "softmax", train=True),
        # one MoE feed-forward layer of many narrow experts, training, from routing to merged output and back
        _moe("moe_layer_train", 4096, 64, 8, 2048, 768),
        # activations packed for an exchange and unpacked on the other side
        _codec("codec_activations", "tensor", 16384, 7168),
    ]


def _size(rng, lo, hi, step):
    """A multiple of ``step`` in [lo, hi], even over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi, max(lo, round(v / step) * step)))


def draw(rng):
    op = rng.choice(["dense"] * 7 + ["grouped"] * 8 + ["moe"] * 2 + ["codec"] * 3)
    fmt = rng.choice(["e4m3", "e4m3", "hybrid"])
    dtype = rng.choice(["bf16"] * 5 + ["fp16"])
    if op == "dense":
        gran = rng.choice(["tensor", "row", "block", "block", "mx"])
        train = rng.random() < 0.6
        cached = not train and rng.random() < 0.5
        step = 32 if gran == "mx" else 16
        n, k = _size(rng, 512, 14336, step), _size(rng, 512, 14336, step)
        m = _size(rng, 128 if train else 16, 16384, 1)
        while m * n * k > 16384 * 8192 * 8192 // (2 if gran == "mx" else 1):
            m //= 2
        return {"op": op, "gran": gran, "m": m, "n": n, "k": k, "train": train, "cached": cached,
                "trans_b": cached or gran == "mx" or rng.random() < 0.7, "fmt": fmt, "dtype": dtype}
    if op == "grouped":
        gran = rng.choice(["tensor", "row", "block", "block", "block", "mx"])
        train = rng.random() < 0.7
        n, k = _size(rng, 1024, 7168, 64), _size(rng, 1024, 7168, 64)
        g = _size(rng, 4, 128, 1)
        while g * n * k > 128 * 4096 * 7168 // (4 if gran in ("mx", "row") else 1):
            g //= 2
        rows = _size(rng, 1024, 32768, 1) if train else _size(rng, 32, 8192, 1)
        if gran in ("mx", "row"):
            rows = max(32, rows // 2)
        while rows * n * k > 32768 * 4096 * 7168 // (2 if gran in ("mx", "row") else 1):
            rows //= 2
        return {"op": op, "gran": gran, "groups": g, "rows": rows, "n": n, "k": k,
                "spread": rng.choice(["softmax", "softmax", "zipf", "even"]), "train": train,
                "cached": not train and rng.random() < 0.7, "fmt": fmt, "dtype": dtype}
    if op == "moe":
        tokens, experts, topk = _size(rng, 256, 8192, 1), rng.choice([8, 16, 32, 64, 128]), rng.choice([2, 4, 6, 8])
        hidden, inter = _size(rng, 1024, 4096, 128), _size(rng, 512, 2048, 128)
        while tokens * topk * hidden * inter > 32768 * 2048 * 2048:
            tokens //= 2
        while experts > 8 and experts * hidden * inter > 128 * 2048 * 1024:
            experts //= 2
        return {"op": op, "tokens": tokens, "experts": experts, "topk": topk, "hidden": hidden, "inter": inter, "fmt": fmt}
    gran = rng.choice(["tensor", "row", "block", "mx"])
    return {"op": op, "gran": gran, "m": _size(rng, 64, 32768, 1), "n": _size(rng, 1024, 8192, 32 if gran == "mx" else rng.choice([8, 8, 8, 1])),
            "fp8": rng.choice(["e4m3", "e4m3", "e5m2"]), "dtype": dtype}


def _config(case):
    gran = case.get("gran", "block")
    scale = ScaleDtype.E8M0 if gran == "mx" else ScaleDtype.FP32
    return Float8QuantConfig(format=FORMAT[case["fmt"]], granularity=GRANULARITY[gran], block_size=BLOCK[gran], scale_dtype=scale)


def _counts(case, gen):
    """Rows per expert: a router's uneven load, a heavy tail with empty experts, or an even split."""
    g, rows = case["groups"], case["rows"]
    if case["spread"] == "even":
        return rows // g + (torch.arange(g) < rows % g).to(torch.int64)
    if case["spread"] == "softmax":
        p = torch.softmax(torch.randn(g, generator=gen), 0)
    else:
        p = torch.arange(1, g + 1, dtype=torch.float32).pow(-1.2)[torch.randperm(g, generator=gen)]
    counts = torch.bincount(torch.multinomial(p, rows, replacement=True, generator=gen), minlength=g)
    if case["spread"] == "zipf" and g >= 16:
        order = torch.argsort(counts, stable=True)
        counts[order[-1]] += counts[order[: g // 16]].sum()
        counts[order[: g // 16]] = 0
    return counts


def prepare(case, seed):
    dev = torch.device("cuda")
    host = torch.Generator().manual_seed(seed)
    gen = torch.Generator(dev).manual_seed(seed)
    dtype = DTYPE[case.get("dtype", "bf16")]

    def normal(*shape, std=1.0, grad=False):
        t = torch.randn(shape, dtype=dtype, device=dev, generator=gen)
        if std != 1.0:
            t.mul_(std)
        return t.requires_grad_(grad)

    s = {"case": case}
    if case["op"] == "codec":
        s["x"] = normal(case["m"], case["n"])
        return s
    s["config"] = _config(case)
    if case["op"] == "moe":
        t, e, k, h, i = (case[x] for x in ("tokens", "experts", "topk", "hidden", "inter"))
        logits = torch.randn(t, e, device=dev, generator=gen) + 0.7 * torch.randn(e, device=dev, generator=gen)
        top, index = torch.topk(torch.softmax(logits, -1), k, dim=-1)
        s["map"] = torch.zeros(t, e, dtype=torch.bool, device=dev).scatter_(1, index, True)
        probs = torch.zeros(t, e, device=dev).scatter_(1, index, top / top.sum(-1, keepdim=True))
        s["probs"] = probs.requires_grad_(True)
        s["x"] = normal(t, h, grad=True)
        s["w1"], s["w2"] = normal(e, 2 * i, h, std=0.02, grad=True), normal(e, h, i, std=0.02, grad=True)
        s["gy"] = normal(t, h, std=1e-3)
        return s
    train, n, k = case["train"], case["n"], case["k"]
    if case["op"] == "dense":
        rows = case["m"]
        w = normal(*((n, k) if case["trans_b"] else (k, n)), std=0.02, grad=train)
    else:
        rows = case["rows"]
        w = normal(case["groups"], n, k, std=0.02, grad=train)
        s["lens"] = _counts(case, host).to(dev)
    s["x"] = normal(rows, k, grad=train)
    if case["cached"]:
        w, _ = create_quantized_weight(w, float8_e4m3, s["config"])
    s["w"] = w
    if train:
        s["gy"] = normal(rows, n, std=1e-3)
    return s


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "codec":
        gran, block = GRANULARITY[case["gran"]], BLOCK[case["gran"]]
        axis = None if case["gran"] == "tensor" else 1
        q, scale = quantize_fp8(s["x"], float8_e4m3 if case["fp8"] == "e4m3" else float8_e5m2, gran, block_size=block, axis=axis)
        y = dequantize_fp8(q, s["x"].dtype, gran, block_size=block, axis=axis, scale_inv=scale)
        return {"q": q.view(torch.uint8), "scale": scale.view(torch.uint8) if case["gran"] == "mx" else scale, "y": y}
    cfg = s["config"]
    if op == "moe":
        x, probs, routing, w1, w2 = s["x"], s["probs"], s["map"], s["w1"], s["w2"]
        rows, row_probs, index, counts = token_permute(x, case["tokens"] * case["topk"], probs=probs, routing_map=routing)
        hidden = grouped_gemm_fp8(rows, w1, counts, config=cfg)
        act = swiglu_with_probs(hidden, row_probs)
        y = grouped_gemm_fp8(act, w2, counts, config=cfg)
        out = token_unpermute(y, index, restore_shape=x.shape, routing_map=routing)
        gx, gp, gw1, gw2 = torch.autograd.grad(out, (x, probs, w1, w2), s["gy"])
        return {"out": out.detach(), "grad_x": gx, "grad_probs": gp, "grad_w1": gw1, "grad_w2": gw2}
    if case["train"]:
        if op == "dense":
            out = gemm_fp8(s["x"], s["w"], trans_b=case["trans_b"], config=cfg)
        else:
            out = grouped_gemm_fp8(s["x"], s["w"], s["lens"], config=cfg)
        gx, gw = torch.autograd.grad(out, (s["x"], s["w"]), s["gy"])
        return {"out": out.detach(), "grad_x": gx, "grad_w": gw}
    with torch.no_grad():
        if op == "dense":
            return gemm_fp8(s["x"], s["w"], trans_b=case["trans_b"], config=cfg)
        return grouped_gemm_fp8(s["x"], s["w"], s["lens"], config=cfg)


def work(case):
    """Inputs read once, outputs written once; 2 M N K per product (padding and re-quantisation never count)."""
    op = case["op"]
    if op == "codec":
        e = case["m"] * case["n"]
        return {"bytes": e * (2 + 1 + 2), "flops": 0}
    if op == "moe":
        t, r = case["tokens"], case["tokens"] * case["topk"]
        h, i, e = case["hidden"], case["inter"], case["experts"]
        weights = 3 * e * h * i
        # tokens, their gradient, the output and its gradient; map, probabilities and theirs; weights and their gradients
        return {"bytes": 4 * 2 * t * h + 9 * t * e + 4 * weights, "flops": 3 * 2 * r * 3 * h * i}
    n, k = case["n"], case["k"]
    rows = case["m"] if op == "dense" else case["rows"]
    experts = 1 if op == "dense" else min(case["groups"], rows)
    flops = 2 * rows * n * k
    if case["train"]:
        return {"bytes": 2 * (2 * rows * k + 2 * rows * n + 2 * experts * n * k), "flops": 3 * flops}
    return {"bytes": 2 * rows * (k + n) + (1 if case["cached"] else 2) * experts * n * k, "flops": flops}


def tolerance(case):
    # codec: bytes and scales have one right value.  The products accumulate FP8 operands in fp32 in whatever order
    # and come out in 16 bits.
    return "exact" if case["op"] == "codec" else {"rel": 1e-2}
