"""The workspace size for a (partly) forced plan is what the launch asks for."""
import ctypes
import math
import random

import pytest
import torch

import amd_developer_challenge_2025_b200 as pkg
from amd_developer_challenge_2025_b200 import _lib
from amd_developer_challenge_2025_b200.fp8_mm import Plan, check_device_status

ONE_FIELD = [Plan(block_n=64), Plan(block_n=128), Plan(block_n=256), Plan(cta_pair=-1), Plan(cta_pair=1), Plan(stages=4),
             Plan(store_bufs=-1), Plan(store_bufs=1), Plan(split_k=2), Plan(split_k=5)]


@pytest.mark.parametrize("plan", [Plan(block_n=64), Plan(cta_pair=-1), Plan(stages=4), Plan(store_bufs=-1)])
def test_cluster_plans_are_sized_as_the_planes_they_replace(built_library, plan):
    # 9 tiles of 64 columns split 14 ways before clusters of eight take their place; run() asks for the former
    assert pkg.workspace_bytes(128, 576, 7168, plan) >= 4096 + 9 * 14 * 128 * 64 * 4
    assert pkg.workspace_bytes(128, 576, 7168) >= 4096 + 9 * 14 * 128 * 64 * 4


def shapes(count, seed):
    rng = random.Random(seed)
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return [(16 * log(1, 64), 16 * log(4, 128), 128 * log(4, 56)) for _ in range(count)]


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(128, 576, 7168), (256, 1536, 7168)] + shapes(16, 1))
def test_the_size_is_enough(m, n, k):
    """The C ABI with a workspace of exactly that size, with K-major and with MN-major operands: never refused for want of it."""
    lib = _lib.load()
    a, b, a_s, b_s, c = pkg.make_inputs(m, n, k, seed=1, device="cuda")
    ta, tb = a.t().contiguous().t(), b.t().contiguous().t()
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    for plan in [None] + ONE_FIELD:
        nbytes = pkg.workspace_bytes(m, n, k, plan)
        ws = torch.zeros(max(nbytes, 256), dtype=torch.uint8, device="cuda")
        cplan = plan.to_c() if plan is not None else None
        for x, y in ((a, b), (ta, tb), (ta, b), (a, tb)):
            rc = lib.b200_fp8_mm_strided(x.data_ptr(), y.data_ptr(), a_s.data_ptr(), b_s.data_ptr(), c.data_ptr(), m, n, k,
                                         *x.stride(), *y.stride(), *a_s.stride(), *b_s.stride(), c.stride(0), 0,
                                         ws.data_ptr() if nbytes else None, nbytes, status.data_ptr(),
                                         torch.cuda.current_stream().cuda_stream, ctypes.byref(cplan) if cplan is not None else None)
            assert rc != 6, (plan, nbytes)
            torch.cuda.synchronize()
    assert status.tolist()[0] == 0
    check_device_status()


@pytest.mark.gpu
def test_a_partly_forced_plan_on_a_fresh_stream():
    a, b, a_s, b_s, c = pkg.make_inputs(128, 576, 7168, seed=1, device="cuda")
    want = pkg.fp8_mm(a, b, a_s, b_s, torch.zeros_like(c))
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        pkg.fp8_mm(a, b, a_s, b_s, c, plan=Plan(block_n=64))
    torch.cuda.synchronize()
    torch.testing.assert_close(c.float(), want.float(), rtol=1e-2, atol=1e-2)
