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
