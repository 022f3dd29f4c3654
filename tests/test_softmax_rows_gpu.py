"""Softmax at the edges of its kernels' ranges: one warp per row up to 2048 elements (8, 16, 32 or 64 elements a lane),
one CTA per row beyond, rows at every 2-byte alignment. Reference: softmax in 64 bits. Bound: the exponential and the
quotient are rounded to bf16 one after the other (2^-8 relative each), plus the error of 2^x: 2^-6 relative in all."""
import math

import pytest
import torch

import amd_developer_challenge_2025_b200 as pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sl", [1, 2, 7, 8, 9, 15, 63, 64, 255, 256, 257, 263, 511, 512, 513, 1023, 1024, 1025, 2047, 2048,
                                2049, 8191, 8192, 8193])
@pytest.mark.parametrize("rows", [1, 7, 9])
def test_row_lengths(sl, rows):
    g = torch.Generator(device="cuda").manual_seed(sl)
    qk = torch.randn(1, rows, sl, dtype=torch.bfloat16, device="cuda", generator=g) * 8
    want = torch.softmax(qk.double() / math.sqrt(192), dim=-1)
    buf = torch.full((rows * sl + 16,), 7.0, dtype=torch.bfloat16, device="cuda")
    for offset in (0, 1, 5):
        view = buf[offset:offset + rows * sl].view(1, rows, sl)
        view.copy_(qk)
        pkg.div_softmax(view, 1, rows, sl, 128, 64)
        torch.cuda.synchronize()
        assert ((view.double() - want).abs() <= 2.0 ** -6 * want).all()
        assert bool((buf[:offset] == 7.0).all()) and bool((buf[offset + rows * sl:] == 7.0).all())
        buf.fill_(7.0)
