"""RoPE's 16-byte kernels on both sides of every line of their dispatch against the scalar kernel, which the same values
reach through rows that are not 16-byte aligned: the same bits (every rounding is prescribed, the angles come from the
same functions)."""
import pytest
import torch

import amd_developer_challenge_2025_b200 as pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d0,d1,d2", [(1, 1, 16), (2, 1, 64), (63, 1, 64), (65, 1, 64), (1000, 1, 64), (1, 31, 64), (7, 33, 64),
                                      (8, 32, 64), (9, 63, 64), (5, 4095, 64), (5, 4096, 64), (1, 8200, 64), (300, 3, 16),
                                      (4, 8, 528), (3, 300, 528), (130, 4100, 64)])
def test_routes_agree(d0, d1, d2):
    g = torch.Generator(device="cuda").manual_seed(d0 + d1)
    x = torch.randn(d0, d1, d2, dtype=torch.bfloat16, device="cuda", generator=g)
    y = torch.full_like(x, float("nan"))
    pkg.mla_decode(x, y, 11, 0, 0, d0, d1, d2, d1 * d2, d2, d1 * d2, d2)
    odd = torch.zeros(d0, d1, d2 + 1, dtype=torch.bfloat16, device="cuda")
    odd[:, :, :d2] = x
    p = d2 + 1
    pkg.mla_decode(odd, odd, 11, 0, 0, d0, d1, d2, d1 * p, p, d1 * p, p)
    torch.cuda.synchronize()
    assert torch.equal(y.view(torch.int16), odd[:, :, :d2].contiguous().view(torch.int16))
    pkg.mla_decode(x, x, 11, 0, 0, d0, d1, d2, d1 * d2, d2, d1 * d2, d2)  # in place
    torch.cuda.synchronize()
    assert torch.equal(y.view(torch.int16), x.view(torch.int16))
