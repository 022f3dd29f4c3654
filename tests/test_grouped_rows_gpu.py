"""The work list of a grouped launch holds only tiles with rows: empty groups first, last and between, negative and too
large counts, counts on both sides of a tile, at every tile shape and with a last wave of every size. Compared bit for
bit with the same groups run whole."""
import random

import pytest
import torch

import amd_developer_challenge_2025_b200 as pkg
from amd_developer_challenge_2025_b200.fp8_mm import Plan, check_device_status, fp8_mm_grouped

pytestmark = pytest.mark.gpu
GUARD = 7.0


def run(g, m, n, k, rows, plan):
    parts = [pkg.make_inputs(m, n, k, seed=i, device="cuda") for i in range(g)]
    a, b, a_s, b_s = (torch.stack([p[j] for p in parts]) for j in range(4))
    full = torch.zeros(g, m, n, dtype=torch.bfloat16, device="cuda")
    c = torch.full_like(full, GUARD)
    fp8_mm_grouped(a, b, a_s, b_s, full, plan=plan)
    fp8_mm_grouped(a, b, a_s, b_s, c, m_valid=torch.tensor(rows, dtype=torch.int32, device="cuda"), plan=plan)
    check_device_status()
    for i, r in enumerate(rows):
        r = max(0, min(m, r))
        assert torch.equal(c[i, :r], full[i, :r])
        assert bool((c[i, r:] == GUARD).all())


PLANS = [None] + [Plan(block_n=bn, cta_pair=-1) for bn in (64, 128, 192, 256)] + [Plan(block_n=bn, cta_pair=1) for bn in (192, 256)]


@pytest.mark.parametrize("plan", PLANS)
@pytest.mark.parametrize("rows", [[0, 0, 0, 0], [0, 256, 0, 1], [512, 300, 0, 0], [-5, 4000, 128, 129], [257, 255, 256, 511]])
def test_counts(plan, rows):
    run(4, 512, 320, 256, rows, plan)


@pytest.mark.parametrize("seed", range(4))
def test_many_groups_and_waves(seed):
    rng = random.Random(seed)
    g, m = 24, 256 * rng.randint(1, 3)
    run(g, m, 64 * rng.randint(6, 40), 256, [rng.randint(0, m) for _ in range(g)], PLANS[rng.choice([0, 4, 6])])
