"""Fewer rows than a tile: the copies of a bring only the rows that exist, and the rest of the stage holds whatever was
there. A launch over NaN operands goes first, so that what is there would show. Reference: the fp32-dequantised product
in 64 bits, within the operator's tolerance (rtol 2e-2, atol 1e-3)."""
import pytest
import torch

import amd_developer_challenge_2025_b200 as pkg
from amd_developer_challenge_2025_b200.fp8_mm import Plan, check_device_status, fp8_mm, fp8_mm_grouped

pytestmark = pytest.mark.gpu


def reference(a, b, a_s, b_s):
    rows = torch.arange(b.shape[0], device=b.device) // 128
    return (a.double() * a_s.double().repeat_interleave(128, 1)) @ (b.double() * b_s[rows].double().repeat_interleave(128, 1)).T


def close(c, want):
    return bool(((c.double() - want).abs() <= 2e-2 * want.abs() + 1e-3).all())


PLANS = [None] + [Plan(block_n=bn, cta_pair=pr, split_k=sp) for bn in (64, 128, 192, 256) for pr in (-1, 1) for sp in (1, 2)]


@pytest.mark.parametrize("plan", PLANS)
@pytest.mark.parametrize("m", [1, 7, 8, 9, 64, 120, 121, 127, 128])
def test_rows(plan, m):
    n, k = 300, 1152
    a, b, a_s, b_s, c = pkg.make_inputs(m, n, k, seed=m, device="cuda")
    nan_a = torch.full((128, k), 0x7f, dtype=torch.uint8, device="cuda").view(torch.float8_e4m3fn)
    fp8_mm(nan_a, b, torch.ones(128, k // 128, device="cuda"), b_s, torch.empty(128, n, dtype=torch.bfloat16, device="cuda"),
           plan=plan)
    c.fill_(float("nan"))
    fp8_mm(a, b, a_s, b_s, c, plan=plan)
    check_device_status()
    assert close(c, reference(a, b, a_s, b_s))


@pytest.mark.parametrize("m,rows", [(1, [1, 0, 1]), (16, [16, 3, 0]), (100, [100, 97, 1])])
def test_groups_of_few_rows(m, rows):
    parts = [pkg.make_inputs(m, 320, 512, seed=i, device="cuda") for i in range(len(rows))]
    a, b, a_s, b_s = (torch.stack([p[j] for p in parts]) for j in range(4))
    c = torch.full((len(rows), m, 320), 7.0, dtype=torch.bfloat16, device="cuda")
    fp8_mm_grouped(a, b, a_s, b_s, c, m_valid=torch.tensor(rows, dtype=torch.int32, device="cuda"))
    check_device_status()
    for i, r in enumerate(rows):
        assert close(c[i, :r], reference(a[i, :r], b[i], a_s[i, :r], b_s[i])) and bool((c[i, r:] == 7.0).all())
