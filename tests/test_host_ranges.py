"""How the host entry point cuts a problem (arithmetic, no GPU), and every cut against one GEMM over the whole problem."""
import pytest
import torch

import amd_developer_challenge_2025_b200 as pkg
from amd_developer_challenge_2025_b200.fp8_mm import HOST_RANGE_BYTES, _range_rows, check_device_status, host_ranges


def covers(m, n, k, chunk):
    by_columns, cuts = host_ranges(m, n, k, chunk)
    extent = n if by_columns else m
    assert cuts[0] == 0 and cuts[-1] == extent and all(x < y for x, y in zip(cuts, cuts[1:])), (m, n, k, chunk, cuts)
    if by_columns:  # the smaller operand goes first; blocks of columns start on whole scale blocks
        assert n > m and all(x % 128 == 0 for x in cuts[:-1]), (m, n, k, chunk, cuts)
    if m * k + n * k + 2 * m * n < HOST_RANGE_BYTES:
        assert len(cuts) == 2
    if len(cuts) > 2:
        assert max(y - x for x, y in zip(cuts, cuts[1:])) <= max(-(-chunk // 128) * 128, 256), (m, n, k, chunk, cuts)


def test_cuts_cover_the_streamed_operand():
    for m, n, k in ((1, 1, 128), (2048, 4608, 7168), (4608, 2048, 7168), (300, 4096, 1024), (1112, 4288, 2816), (700, 4305, 2816), (8192, 4608, 7168)):
        for chunk in (100, 256, 1024, 4096):
            covers(m, n, k, chunk)


@pytest.mark.parametrize("m,k", [(1, 7168), (512, 1024), (2048, 7168), (4096, 2048)])
@pytest.mark.parametrize("chunk", [128, 256, 384, 1000, 1024, 2048])
def test_cuts_at_every_extent(m, k, chunk):
    """Both operands streamed, at every extent: rounding may not bring two cuts of columns together (2048 x 4650 x 7168)."""
    for extent in range(1, 12001):
        covers(m, extent, k, chunk)
        covers(extent, m, k, chunk)


@pytest.mark.parametrize("chunk", [0, -7, None, 512.0])
def test_what_bounds_nothing(chunk):
    """Up to 512 rows, which are never cut by rows, any value is taken (300 x 640 x 7168 divided by zero); beyond, it is refused."""
    for m, n, k in ((300, 640, 7168), (512, 96, 7168), (512, 4608, 7168)):
        covers(m, n, k, _range_rows(m, chunk))
    with pytest.raises(ValueError):
        _range_rows(513, chunk)
    assert _range_rows(513, 1024) == 1024 and _range_rows(5, 1) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,phase,chunk", [(5, 96, 256, 0, 1024), (40, 2048, 1024, 0, 256), (200, 2112, 1024, 64, 256), (130, 2100, 1024, 96, 256),
                                               (1500, 576, 1024, 32, 256), (640, 1999, 640, 0, 100), (600, 4096, 1152, 0, 1024), (700, 4288, 1152, 64, 1024), (2048, 4650, 7168, 0, 1024),
                                               (2048, 4640, 7168, 32, 1024)])
def test_ranges_equal_the_whole_problem(m, n, k, phase, chunk):
    a, b, a_s, _, _ = pkg.make_inputs(m, n, k, seed=m + n)
    g = torch.Generator().manual_seed(n)
    b_s = torch.rand((n + phase + 127) // 128, k // 128, generator=g) + 0.01
    whole = torch.zeros(m, n, dtype=torch.bfloat16, device="cuda")
    pkg.fp8_mm(a.cuda(), b.cuda(), a_s.cuda(), b_s.cuda(), whole, n_phase=phase)
    for pin in (False, True):
        args = [t.pin_memory() if pin else t for t in (a, b, a_s, b_s)]
        c = torch.full((m, n), 7.0, dtype=torch.bfloat16)
        out = pkg.fp8_mm_host(*args, c.pin_memory() if pin else c, n_phase=phase, chunk_rows=chunk)
        check_device_status()
        # a range whose plan splits K adds its partial sums in another order: one rounding of bf16
        torch.testing.assert_close(out.float(), whole.cpu().float(), rtol=2 ** -7, atol=1e-3)


@pytest.mark.gpu
@pytest.mark.parametrize("scales", [torch.float32, torch.float64])  # the plain call and the converting one
def test_chunk_rows_of_zero(scales):
    for m, n in ((300, 640), (513, 640)):
        a, b, a_s, b_s, c = pkg.make_inputs(m, n, 7168, seed=m)
        want = pkg.fp8_mm_host(a, b, a_s, b_s, torch.zeros_like(c))
        call = lambda: pkg.fp8_mm_host(a, b, a_s.to(scales), b_s, c, chunk_rows=0)
        if m <= 512:
            torch.testing.assert_close(call().float(), want.float(), rtol=2 ** -7, atol=1e-3)
        else:
            with pytest.raises(ValueError):
                call()


@pytest.mark.gpu
def test_other_types_are_converted_as_before():
    m, n, k = 300, 256, 512
    a, b, a_s, b_s, c = pkg.make_inputs(m, n, k, seed=3)
    pkg.fp8_mm_host(a, b, a_s, b_s, c)
    c32 = torch.zeros(m, n)
    assert pkg.fp8_mm_host(a, b, a_s.double(), b_s, c32) is c32
    assert torch.equal(c32, c.float())
    with pytest.raises(Exception):
        pkg.fp8_mm_host(a, b, a_s, b_s, c, n_phase=16)
