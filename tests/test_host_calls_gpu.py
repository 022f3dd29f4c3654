"""The native module's checks against the Python ones, over valid and broken calls. The library's functions are replaced
by stubs that record their arguments, so nothing is launched: whatever the native module would launch must be what the
Python checks accept, with the arguments they would pass."""
import ctypes
import importlib

import pytest
import torch

from amd_developer_challenge_2025_b200 import _lib
host = importlib.import_module("amd_developer_challenge_2025_b200.fp8_mm")  # (the package exports the function)

pytestmark = pytest.mark.gpu


@pytest.fixture
def stubs():
    """Binds recorders in place of the four functions; gives back the list of recorded argument tuples."""
    lib, native, calls, keep = _lib.load(), _lib.host_calls(), [], []
    real = (lib.b200_fp8_mm_strided, lib.b200_fp8_mm_grouped, lib.b200_mla_rope, lib.b200_mla_div_softmax)
    for f in real:
        proto = ctypes.CFUNCTYPE(ctypes.c_int, *[ctypes.c_void_p if t not in (ctypes.c_int, ctypes.c_longlong, ctypes.c_size_t)
                                                 else t for t in f.argtypes])
        keep.append(proto(lambda *a: calls.append(a) or 0))
    host._status_words(torch.device("cuda", torch.cuda.current_device()))
    native.bind(*(ctypes.cast(k, ctypes.c_void_p).value for k in keep))
    yield calls
    native.bind(*(ctypes.cast(f, ctypes.c_void_p).value for f in real))


def parts(m=32, n=160, k=256):
    f8 = lambda r: torch.zeros(r, k, device="cuda").to(torch.float8_e4m3fn)
    return [f8(m), f8(n), torch.ones(m, k // 128, device="cuda"), torch.ones((n + 127) // 128, k // 128, device="cuda"),
            torch.zeros(m, n, dtype=torch.bfloat16, device="cuda")]


def wide(t, extra):
    """The same shape inside rows `extra` elements longer."""
    return torch.zeros(t.shape[0], t.shape[1] + extra, device="cuda").to(t.dtype)[:, :t.shape[1]]


CHANGES = {
    "plain": lambda p: p,
    "a mn": lambda p: [p[0].t().contiguous().t()] + p[1:],
    "both mn, scales transposed": lambda p: [t.t().contiguous().t() for t in p[:4]] + p[4:],
    "a pitch 16": lambda p: [wide(p[0], 16)] + p[1:],
    "c pitch odd": lambda p: p[:4] + [wide(p[4], 3)],
    "a pitch 8": lambda p: [wide(p[0], 8)] + p[1:],
    "a base": lambda p: [torch.zeros(32 * 256 + 8, device="cuda").to(torch.float8_e4m3fn)[8:].view(32, 256)] + p[1:],
    "a every other": lambda p: [wide(p[0], 256)[:, :]] + p[1:],
    "a neither": lambda p: [torch.zeros(32, 512, device="cuda").to(torch.float8_e4m3fn)[:, ::2]] + p[1:],
    "a dtype": lambda p: [p[0].to(torch.float8_e5m2)] + p[1:],
    "a uint8": lambda p: [p[0].view(torch.uint8)] + p[1:],
    "scale dtype": lambda p: p[:2] + [p[2].half()] + p[3:],
    "c dtype": lambda p: p[:4] + [p[4].half()],
    "b k": lambda p: [p[0], p[1][:, :128].contiguous()] + p[2:],
    "a_scale rows": lambda p: p[:2] + [p[2][:31]] + p[3:],
    "b_scale rows": lambda p: p[:3] + [p[3][:1]] + p[4:],
    "c shape": lambda p: p[:4] + [p[4][:, :159]],
    "c transposed": lambda p: p[:4] + [torch.zeros(160, 32, dtype=torch.bfloat16, device="cuda").t()],
    "c cpu": lambda p: p[:4] + [p[4].cpu()],
    "a cpu": lambda p: [p[0].cpu()] + p[1:],
    "rank 3": lambda p: [p[0][None]] + p[1:],
    "k 192": lambda p: [p[0][:, :192], p[1][:, :192], p[2], p[3], p[4]],
    "empty": lambda p: [p[0][:0], p[1], p[2][:0], p[3], p[4][:0]],
}


@pytest.mark.parametrize("name", CHANGES)
@pytest.mark.parametrize("n_phase", [0, 96])
def test_fp8_mm(stubs, name, n_phase):
    p = CHANGES[name](parts())
    taken = _lib.host_calls().fp8_mm(*p, n_phase, host._workspaces, host._status)
    try:
        host._validate(*p, n_phase, None)
        valid = p[0].shape[0] > 0
    except (ValueError, RuntimeError):
        valid = False
    assert taken == valid
    assert len(stubs) == int(taken)
    if taken:
        a, b, a_s, b_s, c = p
        assert stubs[0][:18] == (a.data_ptr(), b.data_ptr(), a_s.data_ptr(), b_s.data_ptr(), c.data_ptr(), 32, 160, 256,
                                 *a.stride(), *b.stride(), *a_s.stride(), *b_s.stride(), c.stride(0), n_phase)


def test_other_types_of_argument_are_left_to_python(stubs):
    p = parts()
    native = _lib.host_calls()
    assert not native.fp8_mm(*p, 0.0, host._workspaces, host._status)
    assert not native.fp8_mm(*p, 128, host._workspaces, host._status) and not native.fp8_mm(*p, -1, host._workspaces, host._status)
    assert not native.fp8_mm(p[0], p[1], None, p[3], p[4], 0, host._workspaces, host._status)
    assert not native.fp8_mm(*p, 0, {}, {}) and not native.fp8_mm(*p)
    q = torch.zeros(8, 1, 64, dtype=torch.bfloat16, device="cuda")
    ok = (q, q, 5, 0, 0, 8, 1, 64, 64, 64, 64, 64)
    assert native.mla_decode(*ok) and len(stubs) == 1
    for i, v in ((0, q.float()), (1, q.cpu()), (2, 2.5), (3, -1), (3, 1), (4, 1), (5, 9), (5, 0), (6, 2), (7, 63), (7, 128), (8, 65)):
        assert not native.mla_decode(*ok[:i], v, *ok[i + 1:])
    s = torch.zeros(2, 3, 5, dtype=torch.bfloat16, device="cuda")
    assert native.div_softmax(s, 2, 3, 5, 128, 64) and len(stubs) == 2
    for bad in ((s, 2, 3, 4, 128, 64), (s.float(), 2, 3, 5, 128, 64), (s.cpu(), 2, 3, 5, 128, 64), (s, 2, 3.0, 5, 128, 64),
                (s.transpose(0, 1), 3, 2, 5, 128, 64), (s, -2, -3, 5, 128, 64)):
        assert not native.div_softmax(*bad)
    g = [torch.stack([t, t]) for t in p]
    rows = torch.tensor([3, 4], dtype=torch.int32, device="cuda")
    assert native.fp8_mm_grouped(*g, None, host._status) and native.fp8_mm_grouped(*g, rows, host._status)
    assert len(stubs) == 4
    for bad in (rows.long(), rows[:1], rows.cpu(), torch.zeros(4, dtype=torch.int32, device="cuda")[::2], 3):
        assert not native.fp8_mm_grouped(*g, bad, host._status)
    assert not native.fp8_mm_grouped(g[0][:1], *g[1:], None, host._status)
    assert not native.fp8_mm_grouped(*p, None, host._status)
    assert len(stubs) == 4


@pytest.mark.parametrize("xs1,xs2,xoff,ok", [(64, 64, 0, True), (-64, 64, 448, True), (-64, 64, 447, False), (-64, 64, 0, False),
                                             (64, -64, 128, True), (64, -64, 127, False), (-64, -64, 576, True),
                                             (-64, -64, 575, False), (64, -64, 129, False),
                                             (-(1 << 40), 64, 0, False), (64, -(1 << 40), 448, False)])
def test_rope_strides_of_either_sign(stubs, xs1, xs2, xoff, ok):
    """8 x 3 rows of 64 in a tensor of 640 elements: rows before its start or past its end are refused, as x and as y."""
    t, whole = torch.zeros(640, dtype=torch.bfloat16, device="cuda"), torch.zeros(8, 3, 64, dtype=torch.bfloat16, device="cuda")
    native = _lib.host_calls()
    assert native.mla_decode(t, whole, 0, xoff, 0, 8, 3, 64, xs1, xs2, 192, 64) == ok
    assert native.mla_decode(whole, t, 0, 0, xoff, 8, 3, 64, 192, 64, xs1, xs2) == ok
    assert len(stubs) == 2 * int(ok)
    if not ok:
        import amd_developer_challenge_2025_b200 as pkg
        with pytest.raises(ValueError, match="x: range outside"):
            pkg.mla_decode(t, whole, 0, xoff, 0, 8, 3, 64, xs1, xs2, 192, 64)
        with pytest.raises(ValueError, match="y: range outside"):
            pkg.mla_decode(whole, t, 0, 0, xoff, 8, 3, 64, 192, 64, xs1, xs2)
        assert len(stubs) == 0


@pytest.mark.parametrize("big", [1 << 62, 1 << 64, -(1 << 64), 1 << 100])
def test_integers_beyond_64_bits_launch_nothing(stubs, big):
    native = _lib.host_calls()
    q = torch.zeros(8, 1, 64, dtype=torch.bfloat16, device="cuda")
    ok = (q, q, 5, 64, 64, 7, 1, 64, 64, 64, 64, 64)
    for i in range(2, 12):
        assert not native.mla_decode(*ok[:i], big, *ok[i + 1:])
    s = torch.zeros(2, 3, 5, dtype=torch.bfloat16, device="cuda")
    for i in range(1, 6):
        call = [s, 2, 3, 5, 128, 64]
        call[i] = big
        assert not native.div_softmax(*call)
    p = parts()
    assert not native.fp8_mm(*p, big, host._workspaces, host._status)
    assert stubs == []


def test_forced_plans_and_checked_calls_are_native_too(stubs, monkeypatch):
    """A plan reaches the library; a call that is to be checked is checked; a numpy n_phase is an integer. (The signature of
    a forced plan used to be remembered; going through the Python checks each time took half as long again.)"""
    import numpy as np
    import amd_developer_challenge_2025_b200 as pkg
    p, checked = parts(), []
    monkeypatch.setattr(host, "check_device_status", checked.append)
    monkeypatch.setattr(host, "_validate", lambda *a: pytest.fail("checked in Python"))
    plan = host.Plan(block_n=64, cta_pair=-1, split_k=2, stages=4)
    assert pkg.fp8_mm(*p, plan=plan) is p[4]
    assert stubs[0][-1] and pkg.fp8_mm(*p) is p[4] and not stubs[1][-1]
    assert pkg.fp8_mm(*p, n_phase=np.int64(96)) is p[4] and stubs[2][17] == 96
    assert checked == [] and pkg.fp8_mm(*p, check=True) is p[4] and checked == [p[0].device]
    assert len(stubs) == 4
