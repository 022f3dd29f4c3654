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


def operands(g, m, n, k, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    f8 = lambda *s: torch.randn(*s, dtype=torch.bfloat16, device="cuda", generator=gen).to(torch.float8_e4m3fn)
    scale = lambda *s: 0.01 + torch.rand(*s, device="cuda", generator=gen)
    return f8(g, m, k), f8(g, n, k), scale(g, m, k // 128), scale(g, -(-n // 128), k // 128)


# Around the table's 256 marks (one group each, then runs of groups), and with more items per CTA than the list holds: 192-wide
# tiles, whose list of 8 lies in the header, and 60000 groups, for which 384 are not enough.
@pytest.mark.parametrize("g,m,n,plan", [(1, 1, 64, None), (16, 200, 64, None), (17, 200, 64, None), (255, 130, 64, None),
                                        (256, 130, 64, None), (257, 130, 64, None), (700, 40, 192, None), (2000, 9, 128, None),
                                        (200, 130, 768, Plan(block_n=192, cta_pair=-1)), (400, 130, 384, Plan(block_n=192, cta_pair=-1)),
                                        (300, 256, 576, Plan(block_n=192, cta_pair=1)), (60000, 1, 64, None)])
@pytest.mark.parametrize("kind", ["any", "few", "none", "all"])
def test_many_groups(g, m, n, plan, kind):
    ops = operands(g, m, n, 128, seed=g)
    rng = random.Random(g)
    rows = {"any": [rng.randint(0, m) for _ in range(g)], "few": [m if rng.random() < 0.05 else 0 for _ in range(g)],
            "none": [0] * g, "all": [m] * g}[kind]
    full = torch.zeros(g, m, n, dtype=torch.bfloat16, device="cuda")
    c = torch.full_like(full, GUARD)
    fp8_mm_grouped(*ops, full, plan=plan)
    counts = torch.tensor(rows, dtype=torch.int32, device="cuda")
    fp8_mm_grouped(*ops, c, m_valid=counts, plan=plan)
    check_device_status()
    exists = (torch.arange(m, device="cuda")[None, :] < counts[:, None])[:, :, None]
    assert torch.equal(c, torch.where(exists, full, torch.full_like(full, GUARD)))
    for i in {0, g // 2, g - 1}:
        one = torch.zeros(m, n, dtype=torch.bfloat16, device="cuda")
        pkg.fp8_mm(ops[0][i], ops[1][i], ops[2][i], ops[3][i], one)
        torch.testing.assert_close(full[i].float(), one.float(), rtol=1e-2, atol=1e-2)


@pytest.mark.parametrize("g,m,n", [(256, 16, 256), (1024, 64, 128)])
def test_empty_groups_cost_next_to_nothing(g, m, n):
    """A launch whose row counts leave one group in sixteen takes less time than one over all rows (not the time of a walk
    through the groups: that took 2.2 and 1.6 times as long as all rows)."""
    ops = operands(g, m, n, 128, seed=1)
    c = torch.zeros(g, m, n, dtype=torch.bfloat16, device="cuda")
    counts = torch.tensor([m if i % 16 == 0 else 0 for i in range(g)], dtype=torch.int32, device="cuda")

    def best(**kw):
        s, out = torch.cuda.Stream(), []
        torch.cuda.synchronize()
        with torch.cuda.stream(s):
            fp8_mm_grouped(*ops, c, **kw)
            s.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=s):
                for _ in range(20):
                    fp8_mm_grouped(*ops, c, **kw)
            for _ in range(6):
                e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
                e[0].record(s)
                graph.replay()
                e[1].record(s)
                e[1].synchronize()
                out.append(e[0].elapsed_time(e[1]))
        return min(out)

    assert best(m_valid=counts) < best()
