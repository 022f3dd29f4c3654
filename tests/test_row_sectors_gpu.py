"""Rows of c that the TMA store cannot address leave as whole 32-byte sectors and the pieces before and after them; split-K
clusters write 8-byte pieces. Odd pitches give every distance to a sector boundary; column counts lie around the sizes where a
tile, a thread's share of it or a sector ends. Each run equals, bit for bit, the first columns of the same plan's run with as many
more rows of b as the TMA store needs (N a multiple of 8, c aligned), and nothing around c changes."""
import pytest
import torch

import amd_developer_challenge_2025_b200 as pkg
from amd_developer_challenge_2025_b200.fp8_mm import Plan, check_device_status, fp8_mm, fp8_mm_grouped

pytestmark = pytest.mark.gpu
GUARD = 7.0
PLANS = [Plan(block_n=64, cta_pair=-1, split_k=1), Plan(block_n=192, cta_pair=-1, split_k=1), Plan(block_n=256, cta_pair=1, split_k=1),
         Plan(block_n=64, cta_pair=-1, split_k=3), Plan(block_n=128, cta_pair=-1, split_k=2), Plan(block_n=192, cta_pair=1, split_k=2)]


def rows_in_a_guarded_buffer(rows, n, pitch, offset):
    buf = torch.full((rows * pitch + offset + 32,), GUARD, dtype=torch.bfloat16, device="cuda")
    return buf, buf[offset:offset + rows * pitch].view(rows, pitch)[:, :n]


def only_these_changed(buf, c):
    inside = torch.zeros_like(buf, dtype=torch.bool)
    torch.as_strided(inside, c.shape, c.stride(), c.storage_offset()).fill_(True)
    return bool((buf[~inside] == GUARD).all())


def more_rows(b, dim):
    """b with its rows (dimension `dim`) up to the next multiple of 8: no further scale block, no further tile."""
    more = -b.shape[dim] % 8
    shape = list(b.shape)
    shape[dim] = more
    return torch.cat((b.view(torch.uint8), torch.zeros(shape, dtype=torch.uint8, device=b.device)), dim=dim).view(b.dtype)


@pytest.mark.parametrize("plan", PLANS, ids=lambda p: f"{p.block_n}x{p.cta_pair}x{p.split_k}")
@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 33, 48, 63, 66, 95, 112, 127, 129, 191, 194, 255, 271])
def test_every_distance_to_a_sector(plan, n):
    m, k = 35, 1024
    a, b, a_s, b_s, _ = pkg.make_inputs(m, n, k, seed=n, device="cuda")
    aligned = torch.zeros(m, (n + 7) // 8 * 8, dtype=torch.bfloat16, device="cuda")
    fp8_mm(a, more_rows(b, 0), a_s, b_s, aligned, plan=plan)
    for pitch, offset in ((n | 1, 0), (n + 3 - n % 2, 5), ((n + 1) // 2 * 2, 2), ((n + 7) // 8 * 8 + 8, 8)):
        buf, c = rows_in_a_guarded_buffer(m, n, pitch, offset)
        fp8_mm(a, b, a_s, b_s, c, plan=plan)
        check_device_status()
        assert torch.equal(c, aligned[:, :n]) and only_these_changed(buf, c)


@pytest.mark.parametrize("n", [63, 200, 257])
def test_groups_at_odd_rows(n):
    g, m, k = 3, 140, 256
    parts = [pkg.make_inputs(m, n, k, seed=i, device="cuda") for i in range(g)]
    a, b, a_s, b_s = (torch.stack([p[j] for p in parts]) for j in range(4))
    aligned = torch.zeros(g, m, (n + 7) // 8 * 8, dtype=torch.bfloat16, device="cuda")
    fp8_mm_grouped(a, more_rows(b, 1), a_s, b_s, aligned)
    buf, flat = rows_in_a_guarded_buffer(g * m, n, n | 1, 3)
    c = torch.as_strided(buf, (g, m, n), (m * (n | 1), n | 1, 1), 3)
    rows = torch.tensor([140, 5, 129], dtype=torch.int32, device="cuda")
    fp8_mm_grouped(a, b, a_s, b_s, c, m_valid=rows)
    check_device_status()
    for i, r in enumerate(rows.tolist()):
        assert torch.equal(c[i, :r], aligned[i, :r, :n]) and bool((c[i, r:] == GUARD).all())
    assert only_these_changed(buf, flat)
