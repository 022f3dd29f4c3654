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
        if p.cta_pair and p.block_n == 64:
            assert k // 128 >= 20
    elif p.full_tiles == 0 and not p.cta_pair and p.block_n <= 128 and p.split_k <= 8 and p.tiles <= CLUSTERS[p.split_k]:
        assert p.grid == p.tiles * p.split_k and p.split_k * 2 <= k // 128       # one cluster per tile, all at once
        assert p.stages * (128 + p.block_n) * 128 >= 128 * (p.block_n + 4) * 4   # the ring holds a partial tile
    if p.split_k > 1:
        assert pkg.workspace_bytes(m, n, k) >= 4096 + (p.tiles - p.full_tiles) * p.split_k * 128 * p.block_n * 4 * (
            2 if p.cta_pair else 1)
