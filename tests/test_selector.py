"""The selector's newer rules, over random shapes (host arithmetic only)."""
import math
import random

import pytest

import amd_developer_challenge_2025_b200 as pkg

# clusters of one-CTA-per-SM kernels on a B200 at the same time, by cluster size
CLUSTERS = {2: 74, 3: 45, 4: 33, 5: 26, 6: 22, 7: 15, 8: 15}


def shapes(count, seed):
    rng = random.Random(seed)
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return [(log(1, 16384), log(1, 8192), 128 * log(1, 64)) for _ in range(count)]


@pytest.mark.parametrize("m,n,k", shapes(300, 1))
def test_plans(built_library, m, n, k):
    p = pkg.describe(m, n, k)
    units = 74 if p.cta_pair else 148
    assert p.tiles == -(-m // (256 if p.cta_pair else 128)) * -(-n // p.block_n)
    assert p.grid <= 148 and p.smem_bytes <= 232448
    if p.full_tiles == p.tiles:
        assert p.split_k == 1 and p.grid == min(p.tiles, units) * (2 if p.cta_pair else 1)
        assert not (p.cta_pair and p.block_n == 64)  # (such a plan becomes single CTAs)
    elif p.full_tiles == 0 and not p.cta_pair and p.block_n <= 128 and p.split_k <= 8 and p.tiles <= CLUSTERS[p.split_k]:
        assert p.grid == p.tiles * p.split_k and p.split_k * 2 <= k // 128       # one cluster per tile, all at once
        assert p.stages * (128 + p.block_n) * 128 >= 128 * (p.block_n + 4) * 4   # the ring holds a partial tile
    if p.split_k > 1:
        assert pkg.workspace_bytes(m, n, k) >= 4096 + (p.tiles - p.full_tiles) * p.split_k * 128 * p.block_n * 4 * (
            2 if p.cta_pair else 1)


@pytest.mark.parametrize("m,n,k", [(1024, 1024, 1024), (300, 2000, 512), (200, 700, 1280)] + shapes(200, 2))
def test_the_estimate_belongs_to_the_plan(built_library, m, n, k):
    """64-wide single CTAs, no tile split: 400 clocks a K block and 1850 a tile, for every wave of tiles, and no cluster of the
    same tiles would be cheaper by its own formula."""
    p = pkg.describe(m, n, k)
    if (m, n, k) == (1024, 1024, 1024):
        assert (p.block_n, p.cta_pair, p.split_k) == (64, 0, 1)
    if (p.block_n, p.cta_pair, p.split_k) != (64, 0, 1):
        return
    cost, kb = -(-p.tiles // 148) * (k // 128 * 400 + 1850), k // 128
    assert pkg.estimate_clocks(m, n, k) == cost
    for split, at_once in CLUSTERS.items():
        if split * 2 <= kb and p.tiles <= at_once:
            rows = min(m, 128) / 128
            assert -(-kb // split) * 400 + 1850 + 2600 + 360 * split * (0.5 + 0.5 * rows) >= cost


@pytest.mark.parametrize("m,n,k", [(369, 3196, 1792), (500, 2385, 4352)] + shapes(100, 3))
def test_two_issuers_get_an_even_ring(built_library, m, n, k):
    p = pkg.describe(m, n, k)
    assert p.block_n > 128 or p.stages % 2 == 0
