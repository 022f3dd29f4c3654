"""Launches that may begin under the kernel before them still read and write in stream order: chains in which every call
depends on the one before it, with and without other kernels between, on two streams, and inside a CUDA graph, give the
bits of the same calls run one at a time."""
import random

import pytest
import torch

import amd_developer_challenge_2025_b200 as pkg
from amd_developer_challenge_2025_b200.fp8_mm import check_device_status

pytestmark = pytest.mark.gpu


def chain(a, b, b_s, a_s, c, qk, q, steps, sync):
    """c feeds the next a; qk takes c's first rows before its softmax; q is rotated in place each step."""
    for i in range(steps):
        pkg.custom_kernel((a, b, a_s, b_s, c))
        if sync:
            torch.cuda.synchronize()
        a.copy_((c[:, :a.shape[1]] * 1e-3).to(torch.float8_e4m3fn))
        if sync:
            torch.cuda.synchronize()
        pkg.custom_kernel((a, b, a_s, b_s, c))
        if sync:
            torch.cuda.synchronize()
        qk[0].copy_(c[:qk.shape[1], :qk.shape[2]] * 1e-3)
        pkg.div_softmax(qk, *qk.shape, 128, 64)
        if sync:
            torch.cuda.synchronize()
        pkg.mla_decode(q, q, i, 0, 0, q.shape[0], 1, 64, 64, 64, 64, 64)
        pkg.mla_decode(q, q, i + 1, 0, 0, q.shape[0], 1, 64, 64, 64, 64, 64)
        if sync:
            torch.cuda.synchronize()


def state(m, seed):
    a, b, a_s, b_s, c = pkg.make_inputs(m, 576, 512, seed=seed, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [a, b, b_s, a_s, c, torch.zeros(1, min(m, 64), 500, dtype=torch.bfloat16, device="cuda"),
            torch.randn(300, 1, 64, dtype=torch.bfloat16, device="cuda", generator=g)]


@pytest.mark.parametrize("m", [64, 300, 2048])
@pytest.mark.parametrize("how", ["stream", "two streams", "graph"])
def test_chain_equals_one_call_at_a_time(m, how):
    want = state(m, 1)
    chain(*want, steps=4, sync=True)
    got = state(m, 1)
    if how == "stream":
        chain(*got, steps=4, sync=False)
    elif how == "two streams":
        other = state(m, 2)
        s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
        torch.cuda.synchronize()
        for i in range(4):
            with torch.cuda.stream(s2):
                chain(*other, steps=1, sync=False)
        with torch.cuda.stream(s1):
            chain(*got, steps=4, sync=False)
    else:
        s = torch.cuda.Stream()
        warm = state(m, 3)
        with torch.cuda.stream(s):
            chain(*warm, steps=1, sync=False)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            chain(*got, steps=4, sync=False)
        graph.replay()
    torch.cuda.synchronize()
    check_device_status()
    for g, w in zip(got, want):
        assert torch.equal(g.view(torch.uint8), w.view(torch.uint8))


@pytest.mark.parametrize("seed", range(3))
def test_different_problems_back_to_back(seed):
    """Neighbouring launches differ in shape, kernel, addresses and tensor maps; nothing waits between them."""
    rng = random.Random(seed)
    shapes = [(1, 576, 7168), (300, 2000, 512), (128, 576, 7168), (257, 4099, 384), (2048, 512, 1024), (64, 1536, 2048),
              (1000, 1000, 640), (16, 128, 128), (600, 600, 3584), (513, 3072, 256)]
    rng.shuffle(shapes)
    jobs = []
    for i, (m, n, k) in enumerate(shapes * 2):
        g = torch.Generator(device="cuda").manual_seed(100 * seed + i)
        a, b = (torch.randn(r, k, device="cuda", generator=g).to(torch.float8_e4m3fn) for r in (m, n))
        a_s, b_s = (0.01 + torch.rand(r, k // 128, device="cuda", generator=g) for r in (m, (n + 127) // 128))
        if m % 16 == 0 and n % 16 == 0 and i % 2:
            a, b = (t.t().contiguous().t() for t in (a, b))
        jobs.append((a, b, a_s, b_s))
    want = []
    for (a, b, a_s, b_s) in jobs:
        c = torch.zeros(a.shape[0], b.shape[0], dtype=torch.bfloat16, device="cuda")
        pkg.custom_kernel((a, b, a_s, b_s, c))
        torch.cuda.synchronize()
        want.append(c)
    got = [torch.zeros_like(c) for c in want]
    torch.cuda.synchronize()
    for _ in range(5):
        for (a, b, a_s, b_s), c in zip(jobs, got):
            pkg.custom_kernel((a, b, a_s, b_s, c))
    torch.cuda.synchronize()
    check_device_status()
    for g, w in zip(got, want):
        assert torch.equal(g, w)


def adjacent(step, sync):
    """Calls of this package one directly behind the other; each reads, some in place, what the one before wrote."""
    m, n = 300, 512
    a, b, a_s, b_s, c = pkg.make_inputs(m, n, 1024, seed=step, device="cuda")
    c_aligned, c_odd = c, torch.zeros(m, n + 1, dtype=torch.bfloat16, device="cuda")[:, :n]
    y = torch.zeros(m, n, dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()

    def calls():
        yield lambda: pkg.custom_kernel((a, b, a_s, b_s, c_aligned))
        yield lambda: pkg.mla_decode(c_aligned, c_aligned, step, 0, 0, m, 1, n, n, n, n, n)  # GEMM -> RoPE in place
        yield lambda: pkg.mla_decode(c_aligned, y, step + 1, 0, 0, m, 1, n, n, n, n, n)      # RoPE -> RoPE out of place
        yield lambda: pkg.div_softmax(y, 1, m, n, 128, 64)                                   # RoPE -> softmax
        yield lambda: pkg.div_softmax(y, 1, 1, m * n, 1, 0)                                  # softmax -> softmax, other rows
        yield lambda: pkg.custom_kernel((a, b, a_s, b_s, c_odd))
        yield lambda: pkg.mla_decode(c_odd, c_odd, step, 0, 0, m, 1, n, n + 1, n + 1, n + 1, n + 1)  # the same, rows not aligned
        yield lambda: pkg.custom_kernel((a, b, a_s, b_s, c_aligned))
        yield lambda: pkg.div_softmax(c_aligned, 1, m, n, 1 << 16, 0)                        # GEMM -> softmax in place
        yield lambda: pkg.mla_decode(c_aligned, c_aligned, step, 0, 0, 1, m, n, m * n, n, m * n, n)  # softmax -> RoPE, m positions

    for call in calls():
        call()
        if sync:
            torch.cuda.synchronize()
    return [c_aligned, c_odd, y]


@pytest.mark.parametrize("how", ["stream", "graph"])
def test_directly_adjacent_calls(how):
    for step in range(1, 9):
        want = adjacent(step, sync=True)
        got = adjacent(step, sync=False)
        if how == "graph":
            # the same calls once more, captured, on inputs of their own
            m, n = 300, 512
            a, b, a_s, b_s, c = pkg.make_inputs(m, n, 1024, seed=step, device="cuda")
            s = torch.cuda.Stream()
            torch.cuda.synchronize()
            with torch.cuda.stream(s):
                pkg.custom_kernel((a, b, a_s, b_s, c))  # (the stream's scratch exists before the capture)
            torch.cuda.synchronize()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                for _ in range(4):
                    pkg.custom_kernel((a, b, a_s, b_s, c))
                    pkg.mla_decode(c, c, step, 0, 0, m, 1, n, n, n, n, n)
                    pkg.div_softmax(c, 1, m, n, 1 << 16, 0)
            g.replay()
            torch.cuda.synchronize()
            w = torch.zeros_like(c)
            pkg.custom_kernel((a, b, a_s, b_s, w))
            torch.cuda.synchronize()
            pkg.mla_decode(w, w, step, 0, 0, m, 1, n, n, n, n, n)
            torch.cuda.synchronize()
            pkg.div_softmax(w, 1, m, n, 1 << 16, 0)
            want, got = want + [w], got + [c]
        torch.cuda.synchronize()
        check_device_status()
        for g_, w_ in zip(got, want):
            assert torch.equal(g_.contiguous().view(torch.int16), w_.contiguous().view(torch.int16))


@pytest.mark.parametrize("seed", range(4))
def test_row_counts_written_by_the_kernel_before(seed):
    """Each grouped call's row counts are written by a call of this package directly before it: RoPE at position 0 leaves
    every value as it is, so it copies the counts, seen as bf16 words, into the tensor that the grouped call is given."""
    rng = random.Random(seed)
    g, m, n, k = 8, 300, 320, 256
    parts = [pkg.make_inputs(m, n, k, seed=i, device="cuda") for i in range(g)]
    a, b, a_s, b_s = (torch.stack([p[j] for p in parts]) for j in range(4))
    full = torch.zeros(g, m, n, dtype=torch.bfloat16, device="cuda")
    pkg.fp8_mm_grouped(a, b, a_s, b_s, full)
    rows = [[rng.randint(0, m) for _ in range(g)] for _ in range(12)]
    counts = torch.tensor(rows, dtype=torch.int32, device="cuda")
    m_valid = torch.zeros(g, dtype=torch.int32, device="cuda")
    outs = [torch.full_like(full, 7.0) for _ in rows]
    w = 2 * g  # the counts as 16-bit words
    torch.cuda.synchronize()
    for i, c in enumerate(outs):
        pkg.mla_decode(counts[i].view(torch.bfloat16), m_valid.view(torch.bfloat16), 0, 0, 0, 1, 1, w, w, w, w, w)
        pkg.fp8_mm_grouped(a, b, a_s, b_s, c, m_valid=m_valid)
    check_device_status()
    for c, rs in zip(outs, rows):
        for j, r in enumerate(rs):
            assert torch.equal(c[j, :r], full[j, :r]) and bool((c[j, r:] == 7.0).all())
