"""64-wide tiles take two K blocks to a ring stage: odd K ranges (a half-full last stage), rings of every depth a plan may ask for,
fewer rows than a tile, MN-major operands, pairs, split K and groups. Against the CPU oracle with the tolerance of the parity
tests."""
import pytest
import torch

import amd_developer_challenge_2025_b200 as pkg
from amd_developer_challenge_2025_b200.fp8_mm import Plan, check_device_status, fp8_mm, fp8_mm_grouped
from oracle import fp8_mm_oracle as oracle

pytestmark = pytest.mark.gpu


def checked(c, ref, what):
    check_device_status()
    ok, excess, max_err = oracle.check(c, ref)
    assert ok, (what, excess, max_err)


@pytest.mark.parametrize("m,n", [(1, 70), (40, 64), (150, 200)])
@pytest.mark.parametrize("k", [128, 256, 384, 640, 1152])
def test_odd_and_even_ranges(m, n, k):
    a, b, a_s, b_s, c = pkg.make_inputs(m, n, k, seed=k + m, device="cuda")
    ref = oracle.dequant_matmul(a, b, a_s, b_s)
    plans = [Plan(block_n=64, cta_pair=-1, split_k=1, stages=s) for s in range(2, 9)] + [Plan(block_n=64, cta_pair=1, split_k=1)]
    plans += [Plan(block_n=64, cta_pair=-1, split_k=s) for s in (2, 3, 5) if s * 2 <= k // 128]
    for plan in plans:
        c.fill_(float("nan"))
        fp8_mm(a, b, a_s, b_s, c, plan=plan)
        checked(c, ref, plan)


@pytest.mark.parametrize("m,k", [(48, 384), (160, 640)])
def test_mn_major(m, k):
    n = 208
    a, b, a_s, b_s, c = pkg.make_inputs(m, n, k, seed=m, device="cuda")
    ref = oracle.dequant_matmul(a, b, a_s, b_s)
    for x, y in ((a.t().contiguous().t(), b), (a, b.t().contiguous().t()), (a.t().contiguous().t(), b.t().contiguous().t())):
        for split in (1, 2):
            if split * 2 <= k // 128:
                c.fill_(float("nan"))
                fp8_mm(x, y, a_s, b_s, c, plan=Plan(block_n=64, cta_pair=-1, split_k=split))
                checked(c, ref, (x.stride(), y.stride(), split))


# Odd ranges of more than 15 K blocks: their copies bring two blocks each, the last one a block past the end of K (zeros) or the
# first block of the next range.
@pytest.mark.parametrize("m,n,k,split", [(1, 64, 17, 1), (40, 70, 19, 1), (150, 200, 17, 1), (300, 130, 21, 1), (128, 64, 35, 2),
                                         (20, 200, 53, 3), (140, 72, 38, 2), (257, 64, 33, 1)])
def test_two_blocks_a_copy_over_odd_ranges(m, n, k, split):
    a, b, a_s, b_s, c = pkg.make_inputs(m, n, 128 * k, seed=k, device="cuda")
    ref = oracle.dequant_matmul(a, b, a_s, b_s)
    for plan in [Plan(block_n=64, cta_pair=-1, split_k=split, stages=s) for s in (0, 2, 5)] + [Plan(block_n=64, cta_pair=1, split_k=split)]:
        c.fill_(float("nan"))
        fp8_mm(a, b, a_s, b_s, c, plan=plan)
        checked(c, ref, plan)


@pytest.mark.parametrize("m,n,k,split", [(48, 208, 17, 1), (160, 64, 19, 1), (128, 144, 37, 2)])
def test_two_blocks_a_copy_over_odd_ranges_mn_major(m, n, k, split):
    a, b, a_s, b_s, c = pkg.make_inputs(m, n, 128 * k, seed=k, device="cuda")
    ref = oracle.dequant_matmul(a, b, a_s, b_s)
    for x, y in ((a.t().contiguous().t(), b), (a, b.t().contiguous().t()), (a.t().contiguous().t(), b.t().contiguous().t())):
        c.fill_(float("nan"))
        fp8_mm(x, y, a_s, b_s, c, plan=Plan(block_n=64, cta_pair=-1, split_k=split))
        checked(c, ref, (x.stride(), y.stride()))


@pytest.mark.parametrize("g,m,n,k", [(5, 72, 136, 384), (3, 40, 70, 17 * 128), (4, 150, 64, 19 * 128)])
def test_groups(g, m, n, k):
    parts = [pkg.make_inputs(m, n, k, seed=i, device="cuda") for i in range(g)]
    a, b, a_s, b_s = (torch.stack([p[j] for p in parts]) for j in range(4))
    c = torch.zeros(g, m, n, dtype=torch.bfloat16, device="cuda")
    rows = torch.tensor([m, 0, 1, 9, 64][:g], dtype=torch.int32, device="cuda")
    fp8_mm_grouped(a, b, a_s, b_s, c, m_valid=rows, plan=Plan(block_n=64, cta_pair=-1))
    for i, r in enumerate(min(m, r) for r in rows.tolist()):
        if r:
            checked(c[i, :r], oracle.dequant_matmul(a[i, :r], b[i], a_s[i, :r], b_s[i]), i)
