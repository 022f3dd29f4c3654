"""What `describe` says is what an automatic call runs: 128-wide single CTAs with one tile each have one staging buffer and a ring
of six stages, in the described plan, in shared memory, and when the plan is handed back."""
import pytest
import torch

import amd_developer_challenge_2025_b200 as pkg
from amd_developer_challenge_2025_b200.fp8_mm import check_device_status, fp8_mm

SHAPES = [(1500, 1000, 2048), (369, 3200, 1792), (1024, 2048, 1024), (1152, 1536, 4096), (186, 4813, 1664)]


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_the_plan(built_library, m, n, k):
    p = pkg.describe(m, n, k)
    assert (p.block_n, p.cta_pair, p.split_k, p.stages, p.store_bufs) == (128, 0, 1, 6, 1)
    # ring and two warpgroups' staging, whole KiB of slack and header beside them
    rest = p.smem_bytes - p.stages * (128 + 128) * 128 - 2 * p.store_bufs * 128 * 64
    assert 0 < rest <= 16384 and rest % 1024 == 0


def kernel_time(call):
    s = torch.cuda.Stream()
    times = []
    with torch.cuda.stream(s):
        call()
        s.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            for _ in range(20):
                call()
        for _ in range(8):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record(s)
            graph.replay()
            e[1].record(s)
            e[1].synchronize()
            times.append(e[0].elapsed_time(e[1]))
    return min(times)


@pytest.mark.gpu
def test_handed_back_it_runs_the_same():
    """Equal results, and equal times: the automatic call once took another store path than its own plan, 8 % slower here."""
    m, n, k = 1024, 2048, 1024
    a, b, a_s, b_s, c = pkg.make_inputs(m, n, k, seed=m, device="cuda")
    d = torch.zeros_like(c)
    plan = pkg.describe(m, n, k)
    auto, forced = [min(t) for t in zip(*((kernel_time(lambda: fp8_mm(a, b, a_s, b_s, c)),
                                           kernel_time(lambda: fp8_mm(a, b, a_s, b_s, d, plan=plan))) for _ in range(3)))]
    check_device_status()
    assert torch.equal(c, d)
    assert auto < 1.05 * forced
