"""Performance cases of the package's public entry points.

    listed()            the standing cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what a program has in hand before the call (inputs on the GPU; host buffers for the host call)
    run(state)          one call, as a program makes it, and its outputs
    work(case)          bytes and operations one call cannot do without
    tolerance(case)     how far another correct implementation of the same precision may be
    exact(case, seed)   the outputs of that call in 64 bits

Kinds of case ("op"):

* gemm     `custom_kernel((a, b, a_scale, b_scale, c))`, K-major operands ("k") or the [K][M] / [K][N] storage of the
           competition harness with its [K/128][M] scales ("mn")
* kv_down  `kv_down_projection_fp8`: the KV down-projection of an MLA decode step, output allocated by the call
* grouped  `fp8_mm_grouped` with per-group row counts: the expert GEMMs of one MoE layer
* host     `fp8_mm_host`: operands and result in pinned host memory
* rope     `mla_decode` twice, as a decode step calls it: the query in place, the keys gathered out of the KV cache
* softmax  `div_softmax` over the attention scores of a decode step, in place
"""
from __future__ import annotations

import math
import random

import torch

import amd_developer_challenge_2025_b200 as pkg

DEV = "cuda"
MAX_FLOPS = 2.0 * 8192 * 4608 * 7168  # the largest listed case


def gemm(name, m, n, k, layout="k"):
    return {"name": name, "op": "gemm", "m": m, "n": n, "k": k, "layout": layout}


def listed():
    return [
        # A few tokens against a small weight: launch and call overhead are most of the time.
        gemm("gemm_small_32x576x1024", 32, 576, 1024),
        # KV down-projection of one decode step at batch 128.
        {"name": "kv_down_bs128", "op": "kv_down", "m": 128, "n": 576, "k": 7168},
        # A decode-sized batch against a long-K weight: too few tiles for the SMs.
        gemm("gemm_256x1536x7168", 256, 1536, 7168),
        # KV down-projection in prefill: skinny N, long K.
        gemm("gemm_skinny_2048x576x7168", 2048, 576, 7168),
        # Up-projection with a short K: output-heavy, two to four K blocks per tile.
        gemm("gemm_shortk_2048x7168x512", 2048, 7168, 512),
        # Ragged in both dimensions: row and column remainders, rows of c that are not 16-byte aligned.
        gemm("gemm_ragged_1000x4099x2304", 1000, 4099, 2304),
        # The competition harness's own storage of a, b and the scales, one of its large cases.
        gemm("gemm_mn_6144x3072x1536", 6144, 3072, 1536, "mn"),
        # The large prefill GEMM of the benchmark.
        gemm("gemm_large_8192x4608x7168", 8192, 4608, 7168),
        # Expert GEMMs of an MoE layer with uneven loads.
        {"name": "grouped_8x1024x2048x7168", "op": "grouped", "g": 8, "m": 1024, "n": 2048, "k": 7168},
        # A program whose data lives on the host.
        {"name": "host_2048x4608x7168", "op": "host", "m": 2048, "n": 4608, "k": 7168},
        # RoPE of one decode step: 128 sequences, 128 heads, 6145 positions.
        {"name": "rope_bs128_6145", "op": "rope", "bs": 128, "nh": 128, "sl": 6145},
        # Softmax of the same step's scores.
        {"name": "softmax_bs128_6145", "op": "softmax", "bs": 128, "nh": 128, "sl": 6145},
    ]


def _log_int(rng: random.Random, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choices(["gemm", "kv_down", "grouped", "host", "rope", "softmax"], [10, 2, 2, 1, 1, 1])[0]
    while True:
        if op == "gemm":
            layout = rng.choice(["k", "k", "k", "mn"])
            step = 16 if layout == "mn" else 1  # the pitch of MN-major storage is a multiple of 16
            m = max(1, _log_int(rng, 1, 16384) // step) * step
            n = max(1, _log_int(rng, 64, 8192) // step) * step
            c = {"op": op, "m": m, "n": n, "k": 128 * _log_int(rng, 1, 56), "layout": layout}
        elif op == "kv_down":
            c = {"op": op, "m": _log_int(rng, 1, 4096), "n": 576, "k": 7168}
        elif op == "grouped":
            c = {"op": op, "g": rng.randint(2, 32), "m": _log_int(rng, 16, 2048), "n": 64 * _log_int(rng, 4, 64),
                 "k": 128 * _log_int(rng, 2, 56)}
        elif op == "host":
            c = {"op": op, "m": _log_int(rng, 64, 4096), "n": _log_int(rng, 512, 4608), "k": 128 * _log_int(rng, 2, 56)}
        else:
            c = {"op": op, "bs": _log_int(rng, 1, 128), "nh": rng.choice([16, 32, 64, 128]), "sl": _log_int(rng, 64, 8192)}
        if work(c)["flops"] <= MAX_FLOPS and work(c)["bytes"] <= 6e8:
            return c


# DeepSeek-style MLA sizes, as the reference's decode script uses them.
DNOPE, DROPE, DKV = 128, 64, 512


def _scale(g, *shape):
    return 0.01 + 0.99 * torch.rand(*shape, dtype=torch.float32, device=DEV, generator=g)


def _fp8(g, *shape):
    return torch.randn(*shape, dtype=torch.bfloat16, device=DEV, generator=g).to(torch.float8_e4m3fn)


def _group_rows(case):
    """Rows per group, from a fair share down to a fraction of it: the multiset is the case's, its order the seed's."""
    return [max(1, (case["m"] * (i + 1)) // case["g"]) for i in range(case["g"])]


def prepare(case, seed):
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    op = case["op"]
    if op in ("gemm", "kv_down", "host"):
        m, n, k = case["m"], case["n"], case["k"]
        a, b = _fp8(g, m, k), _fp8(g, n, k)
        a_s, b_s = _scale(g, m, k // 128), _scale(g, (n + 127) // 128, k // 128)
        if op == "kv_down":
            return {"op": op, "x": a, "w": b, "xs": a_s, "ws": b_s}
        if op == "host":
            host = [torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t) for t in (a, b, a_s, b_s)]
            return {"op": op, "args": tuple(host) + (torch.zeros(m, n, dtype=torch.bfloat16).pin_memory(),)}
        if case["layout"] == "mn":
            a, b, a_s, b_s = (t.t().contiguous().t() for t in (a, b, a_s, b_s))
        return {"op": op, "data": (a, b, a_s, b_s, torch.zeros(m, n, dtype=torch.bfloat16, device=DEV))}
    if op == "grouped":
        e, m, n, k = case["g"], case["m"], case["n"], case["k"]
        rows = _group_rows(case)
        random.Random(int(seed)).shuffle(rows)
        return {"op": op, "args": (_fp8(g, e, m, k), _fp8(g, e, n, k), _scale(g, e, m, k // 128),
                                   _scale(g, e, (n + 127) // 128, k // 128),
                                   torch.zeros(e, m, n, dtype=torch.bfloat16, device=DEV)),
                "rows": torch.tensor(rows, dtype=torch.int32, device=DEV)}
    bs, nh, sl = case["bs"], case["nh"], case["sl"]
    if op == "rope":
        return {"op": op, "bs": bs, "nh": nh, "sl": sl,
                "q": torch.randn(bs * nh, 1, DNOPE + DROPE, dtype=torch.bfloat16, device=DEV, generator=g),
                "cache": torch.randn(bs, sl, DKV + DROPE, dtype=torch.bfloat16, device=DEV, generator=g),
                "keys": torch.zeros(bs, sl, DROPE, dtype=torch.bfloat16, device=DEV)}
    return {"op": op, "bs": bs, "nh": nh, "sl": sl,
            "qk": torch.randn(bs, nh, sl, dtype=torch.bfloat16, device=DEV, generator=g) * 8}


def run(state):
    op = state["op"]
    if op == "gemm":
        return pkg.custom_kernel(state["data"])
    if op == "kv_down":
        return pkg.kv_down_projection_fp8(state["x"], state["xs"], state["w"], state["ws"])
    if op == "grouped":
        return pkg.fp8_mm_grouped(*state["args"], m_valid=state["rows"])
    if op == "host":
        return pkg.fp8_mm_host(*state["args"])
    bs, nh, sl = state["bs"], state["nh"], state["sl"]
    if op == "rope":
        dq, dc = DNOPE + DROPE, DKV + DROPE
        pkg.mla_decode(state["q"], state["q"], sl - 1, DNOPE, DNOPE, bs * nh, 1, DROPE, dq, dq, dq, dq)
        pkg.mla_decode(state["cache"], state["keys"], 0, DKV, 0, bs, sl, DROPE, sl * dc, dc, sl * DROPE, DROPE)
        return state["q"], state["keys"]
    return pkg.div_softmax(state["qk"], bs, nh, sl, DNOPE, DROPE)


def work(case):
    op = case["op"]
    if op in ("gemm", "kv_down", "host"):
        rows, weights = case["m"], 1
    elif op == "grouped":
        rows, weights = sum(_group_rows(case)), case["g"]
    elif op == "rope":  # the query's rope part in place, the keys' rope part out of the cache; 3 operations an element
        elems = case["bs"] * (case["nh"] + case["sl"]) * DROPE
        return {"bytes": 4 * elems, "flops": 3 * elems}
    else:  # read and written once; scale, exponential, sum, quotient
        elems = case["bs"] * case["nh"] * case["sl"]
        return {"bytes": 4 * elems, "flops": 4 * elems}
    n, k = case["n"], case["k"]
    nb, kb = (n + 127) // 128, k // 128
    return {"bytes": rows * k + weights * n * k + 4 * rows * kb + 4 * weights * nb * kb + 2 * rows * n,
            "flops": 2.0 * rows * n * k}


def tolerance(case):
    # bf16 results of fp32 arithmetic. Measured against the same operation in 64 bits (relative 2-norm / largest
    # difference): GEMM 1.7e-3 / 3.9e-3, softmax 2.4e-3 / 7.8e-3 (it rounds twice); RoPE prescribes every bf16
    # rounding and differs from itself only where cos and sin of another library round the other way.
    if case["op"] == "softmax":
        return {"rel": 9e-3, "max": 3e-2}
    if case["op"] == "rope":
        return {"rel": 2e-3, "max": 3e-2}
    return {"rel": 6e-3, "max": 2e-2}


def _dequantised(t, s, row_block):
    """t * its block scales in 64 bits: one scale per `row_block` rows and 128 columns."""
    rows = torch.arange(t.shape[-2], device=t.device) // row_block
    return t.double() * s.double().index_select(-2, rows).repeat_interleave(128, dim=-1)


def exact(case, seed):
    """What `run` returns for these inputs, evaluated in 64 bits."""
    s = prepare(case, seed)
    op = case["op"]
    if op == "kv_down":
        return _dequantised(s["x"], s["xs"], 1) @ _dequantised(s["w"], s["ws"], 128).t()
    if op in ("gemm", "host"):
        a, b, a_s, b_s, _ = (t.to(DEV) for t in (s["data"] if op == "gemm" else s["args"]))
        c = _dequantised(a, a_s, 1) @ _dequantised(b, b_s, 128).t()
        return c.cpu() if op == "host" else c
    if op == "grouped":
        a, b, a_s, b_s, c = s["args"]
        out = torch.zeros(c.shape, dtype=torch.float64, device=DEV)
        for g, r in enumerate(s["rows"].tolist()):  # rows past a group's count keep what c held: zeros
            out[g, :r] = _dequantised(a[g, :r], a_s[g, :r], 1) @ _dequantised(b[g], b_s[g], 128).t()
        return out
    if op == "softmax":
        return torch.softmax(s["qk"].double() / math.sqrt(DNOPE + DROPE), dim=-1)
    # The angles' bf16 steps belong to the operator (a position of 6144 has a bf16 step of 32): they are taken as
    # they are, the trigonometry and the rotation in 64 bits.
    half = DROPE // 2
    exponent = ((torch.arange(half, device=DEV).bfloat16() * -2.0).float() / DROPE).bfloat16()
    base = torch.pow(torch.tensor(10000.0, device=DEV).bfloat16().double(), exponent.double()).bfloat16()

    def rotated(x, pos, n):
        idx = (torch.tensor(float(pos)).bfloat16().to(DEV).float() + torch.arange(n, device=DEV).bfloat16().float()).bfloat16()
        theta = (idx.float()[:, None] * base.float()[None, :]).bfloat16().double()
        x = x.double()
        lo, hi = x[..., :half], x[..., half:]
        return torch.cat((lo * theta.cos() - hi * theta.sin(), hi * theta.cos() + lo * theta.sin()), dim=-1)

    q = s["q"].double()
    q[..., DNOPE:] = rotated(s["q"][..., DNOPE:], s["sl"] - 1, 1)
    return q, rotated(s["cache"][..., DKV:], 0, s["sl"])
