"""Split-K through a thread-block cluster: every cluster size, the tile and row remainders, rows of c that are not
8-byte aligned, both operand layouts. The oracle is the fp32-dequantised product in 64 bits; the bound is the bf16
rounding of the result (2^-8 relative) plus what the tensor core's partial sums inside a K block may lose (the same
allowance as for the unsplit kernels: 2e-2 relative, 1e-3 absolute)."""
import pytest
import torch

import amd_developer_challenge_2025_b200 as pkg
from amd_developer_challenge_2025_b200.fp8_mm import Plan, check_device_status, fp8_mm

pytestmark = pytest.mark.gpu


def reference(a, b, a_s, b_s):
    rows = torch.arange(b.shape[0], device=b.device) // 128
    return (a.double() * a_s.double().repeat_interleave(128, 1)) @ (b.double() * b_s[rows].double().repeat_interleave(128, 1)).T


@pytest.mark.parametrize("split", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("block_n", [64, 128])
@pytest.mark.parametrize("m,n,kblocks", [(1, 64, 16), (128, 576, 17), (129, 131, 16), (33, 70, 23)])
def test_every_cluster_size(split, block_n, m, n, kblocks):
    a, b, a_s, b_s, c = pkg.make_inputs(m, n, 128 * kblocks, seed=m + n + split, device="cuda")
    plan = Plan(block_n=block_n, cta_pair=-1, split_k=split)
    c.fill_(float("nan"))
    fp8_mm(a, b, a_s, b_s, c, plan=plan)
    check_device_status()
    want = reference(a, b, a_s, b_s)
    assert ((c.double() - want).abs() <= 2e-2 * want.abs() + 1e-3).all()
    again = torch.empty_like(c)
    fp8_mm(a, b, a_s, b_s, again, plan=plan)
    assert torch.equal(c, again)  # the ranges are added in a fixed order


@pytest.mark.parametrize("pad,offset", [(0, 1), (1, 0), (3, 2), (4, 4)])
def test_rows_at_any_alignment(pad, offset):
    m, n, guard = 100, 197, 7.0
    a, b, a_s, b_s, _ = pkg.make_inputs(m, n, 2048, seed=3, device="cuda")
    plan = Plan(block_n=64, cta_pair=-1, split_k=4)
    want = torch.zeros(m, 200, dtype=torch.bfloat16, device="cuda")
    fp8_mm(a, b, a_s, b_s, want[:, :n], plan=plan)
    pitch = n + pad
    buf = torch.full((m * pitch + 8,), guard, dtype=torch.bfloat16, device="cuda")
    c = buf[offset:offset + m * pitch].view(m, pitch)[:, :n]
    fp8_mm(a, b, a_s, b_s, c, plan=plan)
    check_device_status()
    assert torch.equal(c, want[:, :n])
    assert bool((buf[:offset] == guard).all()) and bool((buf[offset:offset + m * pitch].view(m, pitch)[:, n:] == guard).all())


def test_mn_major_operands_equal_k_major():
    a, b, a_s, b_s, c = pkg.make_inputs(112, 576, 7168, seed=5, device="cuda")
    mn = [t.t().contiguous().t() for t in (a, b, a_s, b_s)]
    for plan in (Plan(block_n=64, cta_pair=-1, split_k=8), Plan(block_n=128, cta_pair=-1, split_k=5), None):
        d = torch.empty_like(c)
        fp8_mm(a, b, a_s, b_s, c, plan=plan)
        fp8_mm(*mn, d, plan=plan)
        check_device_status()
        assert torch.equal(c, d)


def test_needs_no_workspace_beyond_what_the_size_function_says(built_library):
    """A plan that runs as clusters is chosen beside the one that sizes the workspace, never instead of its demands."""
    for (m, n, k) in ((16, 576, 7168), (128, 576, 7168), (512, 1536, 7168), (16, 4608, 7168), (256, 7168, 2048)):
        p = pkg.describe(m, n, k)
        if p.split_k > 1:
            assert pkg.workspace_bytes(m, n, k) >= 4096 + (p.tiles - p.full_tiles) * p.split_k * 128 * p.block_n * 4
