"""The native module belongs to one Python and one torch: it is loaded for these only, and is not needed."""
import os
import warnings

import pytest
import torch

from amd_developer_challenge_2025_b200 import _lib, build


def test_another_torch_gets_another_module(built_library, monkeypatch):
    here = build.host_path()
    assert os.path.exists(here) and not build.needs_build()
    monkeypatch.setattr(torch, "__version__", "99.0")
    assert build.host_path() != here and os.path.dirname(build.host_path()) == os.path.dirname(here)
    assert build.needs_build()


def test_without_the_module_the_python_checks_do(built_library, monkeypatch):
    monkeypatch.setattr(_lib, "_host", None)
    monkeypatch.setattr(torch, "__version__", "99.0")
    with pytest.warns(RuntimeWarning, match="99.0"):
        calls = _lib.host_calls()
    assert not any(f(1, 2) for f in (calls.fp8_mm, calls.fp8_mm_grouped, calls.mla_decode, calls.div_softmax))
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert _lib.host_calls() is calls


@pytest.mark.gpu
def test_results_without_the_module(monkeypatch):
    import amd_developer_challenge_2025_b200 as pkg

    def all_calls():
        a, b, a_s, b_s, c = pkg.make_inputs(64, 256, 512, seed=1, device="cuda")
        g = [t[None].contiguous() for t in (a, b, a_s, b_s, torch.zeros_like(c))]
        x = torch.arange(8 * 64, device="cuda").reshape(8, 1, 64).bfloat16() / 64
        q = torch.arange(6 * 70, device="cuda").reshape(2, 3, 70).bfloat16() / 64
        return [pkg.custom_kernel((a, b, a_s, b_s, c)), pkg.fp8_mm_grouped(*g),
                pkg.mla_decode(x, x, 5, 0, 0, 8, 1, 64, 64, 64, 64, 64), pkg.div_softmax(q, 2, 3, 70, 128, 64)]

    want = all_calls()
    monkeypatch.setattr(_lib, "_host", _lib._PythonChecks)
    for g, w in zip(all_calls(), want):
        assert torch.equal(g, w)
