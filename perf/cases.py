"""Performance cases of the operator library: what a user's program calls, at the sizes it calls it with.

Eight kinds of work, each through the public entry points (``torch.ops.b200k.*``, ``ops.linear``,
``ops.sdpa``):

  gemm      a matrix product, any storage order of the operands
  rows      a linear layer with bias and activation on a few rows (one decode step of a served model)
  linear    a linear layer with bias, forward and backward (training)
  fp8       an fp8 linear layer: activations quantised on each call, or both operands given in fp8
  attn      attention forward (prefill), causal or not
  train     attention forward and backward
  decode    one step of decoding: paged (new K/V rows appended first) or over a contiguous history
  chunk     one chunk of a prefill over a paged cache (K/V appended, then attention)

``listed()`` are fixed cases, ``draw()`` gives another one of the same ranges.
"""

import math

import torch

from iree_turbine_b200 import ops

DEVICE = "cuda"
DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}
SIZE = {"f16": 2, "bf16": 2, "f32": 4}

# No drawn case costs more than the largest listed ones: the operations of the long causal prefill
# (fp8 ones count half, those of a backward one and a half) and the bytes of the large decode step.
MOST_FLOPS = 5.4e11
FLOP_COST = {"fp8": 0.5, "train": 1.5}
MOST_BYTES = 1.1e9


def listed():
    return [
        # A projection of a decode step: 16 sequences, one token each, bias and activation fused.
        {"name": "rows_16x4096x4096", "kind": "rows", "m": 16, "n": 4096, "k": 4096, "dtype": "bf16", "act": "silu"},
        # The ordinary half-precision product of the benchmark, accumulated and returned in fp32.
        {"name": "gemm_f16_2048", "kind": "gemm", "m": 2048, "n": 2048, "k": 2048, "dtype": "f16", "out": "f32",
         "trans_a": False, "trans_b": True},
        # A training step of a linear layer on a ragged batch of tokens: y, dx, dw and db.
        {"name": "linear_train_3000", "kind": "linear", "m": 3000, "n": 4352, "k": 3840, "dtype": "bf16"},
        # A linear layer served in fp8: fp32 activations of a ragged batch are quantised on each call.
        {"name": "fp8_linear_1000", "kind": "fp8", "m": 1000, "n": 4096, "k": 4096, "quantize": True},
        # The benchmark's fp8 product: both operands in fp8 already, the largest contraction.
        {"name": "fp8_gemm_8192", "kind": "fp8", "m": 8192, "n": 8192, "k": 8192, "quantize": False},
        # Attention of an encoder or a vision model: many short sequences, no mask.
        {"name": "attn_full_8x32x1024", "kind": "attn", "batch": 8, "heads": 32, "kv_heads": 32, "sq": 1024,
         "skv": 1024, "dim": 128, "causal": False, "dtype": "f16"},
        # Prefill of long prompts: the benchmark's headline problem.
        {"name": "attn_causal_4x32x4096", "kind": "attn", "batch": 4, "heads": 32, "kv_heads": 32, "sq": 4096,
         "skv": 4096, "dim": 128, "causal": True, "dtype": "bf16"},
        # A small attention call with head dim 64: 32 sequences of 128 tokens (launch-bound).
        {"name": "attn_short_32x8x128", "kind": "attn", "batch": 32, "heads": 8, "kv_heads": 8, "sq": 128,
         "skv": 128, "dim": 64, "causal": True, "dtype": "bf16"},
        # A training step of a grouped-query attention layer on ragged sequences: output and gradients.
        {"name": "attn_train_2x32x2000", "kind": "train", "batch": 2, "heads": 32, "kv_heads": 8, "sq": 2000,
         "skv": 2000, "dim": 128, "causal": True, "dtype": "bf16"},
        # Decoding for a few users over their own contiguous histories: latency decides.
        {"name": "decode_4_seqs", "kind": "decode", "paged": False, "seqs": 4, "heads": 32, "kv_heads": 8,
         "dim": 128, "min_len": 100, "max_len": 1000, "page": 16, "dtype": "bf16"},
        # A decode step of a loaded server: 64 sequences of 512 to 8192 tokens in pages of 16.
        {"name": "paged_decode_64_seqs", "kind": "decode", "paged": True, "seqs": 64, "heads": 32, "kv_heads": 8,
         "dim": 128, "min_len": 512, "max_len": 8192, "page": 16, "dtype": "f16"},
        # The next 512 prompt tokens of four sequences, appended to the cache and attended to.
        {"name": "paged_prefill_4x512", "kind": "chunk", "batch": 4, "heads": 32, "kv_heads": 8, "sq": 512,
         "max_len": 4000, "dim": 128, "page": 16, "dtype": "bf16"},
    ]


def _log(rng, lo, hi, multiple=1):
    """A whole number between lo and hi, even over the logarithm, rounded to a multiple."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / multiple)) * multiple))


def _heads(rng):
    kv = rng.choice([1, 2, 4, 8, 16])
    group = rng.choice([1, 1, 2, 4, 8])
    return kv * group, kv


def _draw(rng):
    kind = rng.choice(["gemm", "rows", "linear", "fp8", "attn", "train", "decode", "chunk"])
    dtype = rng.choice(["f16", "bf16"])
    if kind == "gemm":
        # The contiguous size of each operand is a multiple of 8.
        ta, tb = rng.choice([(False, True), (False, True), (False, False), (True, False)])
        m, n, k = _log(rng, 64, 8192, 8 if ta else 1), _log(rng, 64, 8192, 1 if tb else 8), _log(rng, 64, 16384, 8)
        return {"kind": kind, "m": m, "n": n, "k": k, "dtype": dtype, "out": rng.choice(["f32", dtype]),
                "trans_a": ta, "trans_b": tb}
    if kind == "rows":
        return {"kind": kind, "m": _log(rng, 1, 256), "n": _log(rng, 1024, 14336, 8), "k": _log(rng, 1024, 14336, 8),
                "dtype": dtype, "act": rng.choice(["none", "relu", "gelu", "silu"])}
    if kind == "linear":
        return {"kind": kind, "m": _log(rng, 256, 8192), "n": _log(rng, 512, 8192, 8), "k": _log(rng, 512, 8192, 8),
                "dtype": dtype}
    if kind == "fp8":
        return {"kind": kind, "m": _log(rng, 16, 8192), "n": _log(rng, 1024, 8192), "k": _log(rng, 1024, 8192, 16),
                "quantize": rng.random() < 0.6}
    if kind in ("attn", "train"):
        heads, kv = _heads(rng)
        causal = rng.random() < 0.6
        sq = _log(rng, 64, 8192)
        skv = sq if causal or rng.random() < 0.5 else _log(rng, 64, 8192)
        return {"kind": kind, "batch": _log(rng, 1, 32), "heads": heads, "kv_heads": kv, "sq": sq, "skv": skv,
                "dim": rng.choice([128, 128, 64]), "causal": causal, "dtype": dtype}
    heads, kv = _heads(rng)
    case = {"kind": kind, "heads": heads, "kv_heads": kv, "dim": rng.choice([128, 128, 64]),
            "page": rng.choice([16, 16, 32, 64]), "dtype": dtype}
    if kind == "decode":
        max_len = _log(rng, 64, 16384)
        return dict(case, paged=rng.random() < 0.7, seqs=_log(rng, 1, 128), min_len=max(1, max_len // 16),
                    max_len=max_len)
    sq = _log(rng, 16, 2048)
    return dict(case, batch=_log(rng, 1, 16), sq=sq, max_len=sq + _log(rng, 16, 8192))


def draw(rng):
    while True:
        case = _draw(rng)
        w = work(case)
        if w["flops"] * FLOP_COST.get(case["kind"], 1.0) <= MOST_FLOPS and w["bytes"] <= MOST_BYTES:
            return case


def _lens(case):
    """Sequence lengths, evenly spread between the two ends (their sum does not depend on a seed)."""
    n = case["batch"] if case["kind"] == "chunk" else case["seqs"]
    lo = case["sq"] if case["kind"] == "chunk" else case["min_len"]
    hi = case["max_len"]
    return [hi - (hi - lo) * i // max(1, n) for i in range(n)]


def _pairs(case):
    """Visible (query, key) pairs of one head and batch element; keys are aligned at the end."""
    if not case["causal"]:
        return case["sq"] * case["skv"]
    return case["sq"] * (case["skv"] - case["sq"]) + case["sq"] * (case["sq"] + 1) // 2


def work(case):
    kind = case["kind"]
    if kind in ("gemm", "rows", "linear", "fp8"):
        m, n, k = case["m"], case["n"], case["k"]
        product = 2.0 * m * n * k
        if kind == "gemm":
            s = SIZE[case["dtype"]]
            return {"bytes": s * (m * k + n * k) + SIZE[case["out"]] * m * n, "flops": product}
        if kind == "rows":
            return {"bytes": 2.0 * (m * k + n * k + m * n + n), "flops": product}
        if kind == "linear":  # x, w, bias, dy read; y, dx, dw, db written
            return {"bytes": 2.0 * (2 * m * k + 2 * n * k + 2 * m * n + 2 * n), "flops": 3 * product}
        return {"bytes": (4 if case["quantize"] else 1) * m * k + n * k + 2.0 * m * n, "flops": product}
    if kind in ("attn", "train"):
        b, h, kv, d = case["batch"], case["heads"], case["kv_heads"], case["dim"]
        q, k = b * h * case["sq"] * d, b * kv * case["skv"] * d
        flops = 4.0 * b * h * d * _pairs(case)
        if kind == "attn":
            return {"bytes": 2.0 * (2 * q + 2 * k), "flops": flops}
        return {"bytes": 2.0 * (4 * q + 4 * k), "flops": 3.5 * flops}  # q, o, do, dq; k, v, dk, dv
    lens, d, h, kv = _lens(case), case["dim"], case["heads"], case["kv_heads"]
    cache = 2.0 * 2 * kv * d * sum(lens)
    if kind == "decode":
        q = 2.0 * len(lens) * h * d
        flops = 4.0 * h * d * sum(lens)
        tables = 4.0 * len(lens)
        if case["paged"]:  # the new rows are read and written, and then are part of the cache
            tables += 4.0 * sum(-(-n // case["page"]) for n in lens) + 2 * 2.0 * len(lens) * kv * d
        return {"bytes": cache + 2 * q + tables, "flops": flops}
    sq = case["sq"]
    pairs = sum(sq * (n - sq) + sq * (sq + 1) // 2 for n in lens)
    q = 2.0 * len(lens) * h * sq * d
    new = 2 * 2.0 * len(lens) * kv * sq * d
    return {"bytes": cache + 2 * q + new + 4.0 * sum(-(-n // case["page"]) for n in lens), "flops": 4.0 * h * d * pairs}


def tolerance(case):
    # fp32 results of 16-bit operands differ by the order of the fp32 sums; 16-bit results by one
    # rounding of the output and, in attention, of the probabilities and their gradients.  A tensor
    # quantised to fp8 may round single values the other way before the product is rounded to bf16.
    if case["kind"] == "gemm" and case["out"] == "f32":
        return {"rel": 2e-5}
    if case["kind"] == "fp8":
        return {"rel": 1e-2}
    return {"rel": 2e-3 if case["dtype"] == "f16" else 1e-2}


def _normal(g, shape, dtype, std=1.0):
    t = torch.randn(shape, generator=g, device=DEVICE, dtype=dtype)
    return t.mul_(std) if std != 1.0 else t


def _to_fp8(t):
    scale = t.abs().max().float().reshape(1) / 448.0
    return (t.float() / scale).to(torch.float8_e4m3fn), scale


def _pages(case, lens, g, dtype):
    """A page pool in random order: caches, block table and lengths, as a serving program keeps them."""
    page, shape = case["page"], (case["kv_heads"], case["page"], case["dim"])
    counts = [-(-n // page) for n in lens]
    order = torch.randperm(sum(counts), generator=g, device=DEVICE).to(torch.int32)
    table = torch.zeros((len(lens), max(counts)), dtype=torch.int32, device=DEVICE)
    for row, part in zip(table, order.split(counts)):
        row[: part.numel()] = part
    return (_normal(g, (sum(counts),) + shape, dtype), _normal(g, (sum(counts),) + shape, dtype), table,
            torch.tensor(lens, dtype=torch.int32, device=DEVICE))


def prepare(case, seed):
    kind = case["kind"]
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    dtype = DTYPES[case.get("dtype", "bf16")]
    s = dict(case)
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        s["a"] = _normal(g, (k, m) if case["trans_a"] else (m, k), dtype)
        s["b"] = _normal(g, (n, k) if case["trans_b"] else (k, n), dtype)
        s["out_dtype"] = DTYPES[case["out"]]
    elif kind in ("rows", "linear"):
        m, n, k = case["m"], case["n"], case["k"]
        s["x"], s["w"] = _normal(g, (m, k), dtype), _normal(g, (n, k), dtype, k ** -0.5)
        s["bias"], s["out_dtype"] = _normal(g, (n,), dtype, 0.1), dtype
        if kind == "linear":
            for name in ("x", "w", "bias"):
                s[name].requires_grad_(True)
            s["dy"] = _normal(g, (m, n), dtype)
    elif kind == "fp8":
        m, n, k = case["m"], case["n"], case["k"]
        x = _normal(g, (m, k), torch.float32)
        s["x"] = x if case["quantize"] else _to_fp8(x)
        s["w"], s["scale_w"] = _to_fp8(_normal(g, (n, k), torch.float32, k ** -0.5))
    elif kind in ("attn", "train"):
        b, h, kv, d = case["batch"], case["heads"], case["kv_heads"], case["dim"]
        s["scale"] = d ** -0.5
        s["q"] = _normal(g, (b, h, case["sq"], d), dtype, 0.5)
        s["k"], s["v"] = (_normal(g, (b, kv, case["skv"], d), dtype, 0.5) for _ in range(2))
        if kind == "train":
            for name in ("q", "k", "v"):
                s[name].requires_grad_(True)
            s["do"] = _normal(g, (b, h, case["sq"], d), dtype)
    else:
        lens, d, h, kv = _lens(case), case["dim"], case["heads"], case["kv_heads"]
        s["scale"] = d ** -0.5
        new = case.get("sq", 1)
        if kind == "chunk":
            s["q"] = _normal(g, (len(lens), h, new, d), dtype)
        else:
            s["q"] = _normal(g, (len(lens), h, d), dtype)
        if kind == "chunk" or case["paged"]:
            s["kc"], s["vc"], s["table"], s["lens"] = _pages(case, lens, g, dtype)
            s["k_new"], s["v_new"] = (_normal(g, (len(lens), new, kv, d), dtype) for _ in range(2))
            s["positions"] = s["lens"] - new
        else:
            s["kc"], s["vc"] = (_normal(g, (len(lens), kv, max(lens), d), dtype) for _ in range(2))
            s["lens"] = torch.tensor(lens, dtype=torch.int32, device=DEVICE)
    return s


def run(s):
    kind, op = s["kind"], torch.ops.b200k
    if kind == "gemm":
        if s["trans_b"] and not s["trans_a"]:
            return op.gemm_nt(s["a"], s["b"], s["out_dtype"])
        return op.gemm(s["a"], s["b"], s["trans_a"], s["trans_b"], s["out_dtype"])
    if kind == "rows":
        return op.linear_act(s["x"], s["w"], s["bias"], s["act"], s["out_dtype"])
    if kind == "linear":
        y = ops.linear(s["x"], s["w"], s["bias"])
        return (y.detach(),) + torch.autograd.grad(y, (s["x"], s["w"], s["bias"]), s["dy"])
    if kind == "fp8":
        x, scale_x = op.quantize_e4m3(s["x"]) if s["quantize"] else s["x"]
        return op.gemm_fp8_nt(x, s["w"], scale_x, s["scale_w"])
    if kind == "attn":
        return op.attention(s["q"], s["k"], s["v"], s["scale"], s["causal"])
    if kind == "train":
        o = ops.sdpa(s["q"], s["k"], s["v"], s["scale"], s["causal"])
        return (o.detach(),) + torch.autograd.grad(o, (s["q"], s["k"], s["v"]), s["do"])
    if kind == "decode" and not s["paged"]:
        return op.decode_attention(s["q"], s["kc"], s["vc"], s["lens"], s["scale"])
    op.kv_append(s["k_new"], s["v_new"], s["kc"], s["vc"], s["table"], s["positions"])
    if kind == "chunk":
        o = op.paged_attention(s["q"], s["kc"], s["vc"], s["table"], s["lens"], s["scale"], True)
    else:
        o = op.paged_decode_attention(s["q"], s["kc"], s["vc"], s["table"], s["lens"], s["scale"])
    return o, s["kc"], s["vc"]
