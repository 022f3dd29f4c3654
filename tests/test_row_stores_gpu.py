"""Rows of c that the TMA store cannot write (odd pitch or base, a row length that is no multiple of 8) and tiles that a group's
row count cuts short leave straight from registers. Each run is compared bit for bit with the same plan's TMA store: an aligned c of
N up to the next multiple of 8, which the parity tests hold against the CPU oracle. The elements around c must keep their value."""
import pytest
import torch

import amd_developer_challenge_2025_b200 as pkg
from amd_developer_challenge_2025_b200.fp8_mm import Plan, check_device_status, fp8_mm, fp8_mm_grouped

pytestmark = pytest.mark.gpu
GUARD = 7.0


def inside(m, n, pitch, offset):
    """A [m, n] view with the given row pitch, `offset` elements into a buffer filled with GUARD."""
    buf = torch.full(((m + 1) * pitch + offset + 8,), GUARD, dtype=torch.bfloat16, device="cuda")
    return buf, buf[offset:offset + m * pitch].view(m, pitch)[:, :n]


def untouched(buf, m, n, pitch, offset):
    mask = torch.ones_like(buf, dtype=torch.bool)
    mask[offset:offset + m * pitch].view(m, pitch)[:, :n] = False
    return bool((buf[mask] == GUARD).all())


@pytest.mark.parametrize("block_n,pair", [(64, -1), (64, 1), (128, -1), (128, 1), (192, -1), (192, 1), (256, -1), (256, 1)])
@pytest.mark.parametrize("m,n,pad,offset", [(1, 1, 0, 0), (129, 65, 0, 0), (33, 96, 1, 0), (128, 255, 0, 1),
                                            (257, 67, 2, 3), (160, 31, 0, 0), (300, 577, 0, 0)])
def test_unaligned_rows_equal_the_aligned_run(block_n, pair, m, n, pad, offset):
    plan = Plan(block_n=block_n, cta_pair=pair, split_k=1)
    a, b, a_s, b_s, _ = pkg.make_inputs(m, n, 384, seed=m + n, device="cuda")
    more = torch.zeros(-n % 8, 384, dtype=torch.uint8, device="cuda")  # (no further scale block and no further tile)
    wide = torch.zeros(m, (n + 7) // 8 * 8, dtype=torch.bfloat16, device="cuda")
    fp8_mm(a, torch.cat((b.view(torch.uint8), more)).view(b.dtype), a_s, b_s, wide, plan=plan)
    pitch = n + pad
    buf, c = inside(m, n, pitch, offset)
    fp8_mm(a, b, a_s, b_s, c, plan=plan)
    check_device_status()
    assert torch.equal(c, wide[:, :n])
    assert untouched(buf, m, n, pitch, offset)


@pytest.mark.parametrize("plan", [None, Plan(block_n=192, cta_pair=-1), Plan(block_n=256, cta_pair=1)])
@pytest.mark.parametrize("n,rows", [(512, [1, 255, 256, 100, 0, 37]), (197, [256, 3, 128, 129])])
def test_groups_cut_short(plan, n, rows):
    g, m, k = len(rows), 256, 256
    parts = [pkg.make_inputs(m, n, k, seed=i, device="cuda") for i in range(g)]
    a, b, a_s, b_s = (torch.stack([p[j] for p in parts]) for j in range(4))
    c = torch.full((g, m, n), GUARD, dtype=torch.bfloat16, device="cuda")
    full = torch.zeros_like(c)
    fp8_mm_grouped(a, b, a_s, b_s, full, plan=plan)
    fp8_mm_grouped(a, b, a_s, b_s, c, m_valid=torch.tensor(rows, dtype=torch.int32, device="cuda"), plan=plan)
    check_device_status()
    for i, r in enumerate(rows):
        assert torch.equal(c[i, :r], full[i, :r])
        assert bool((c[i, r:] == GUARD).all())
