"""Kernels that may begin under the kernel before them read memory which that kernel may still be writing. Loads through the
read-only path require memory that nothing writes while the kernel lives, and the compiler may move them above the wait for
the earlier kernel, so no source of such kernels asks for them: no __ldg, no ld.global.nc, no `const T* __restrict__`."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "amd_developer_challenge_2025_b200", "csrc")


@pytest.mark.parametrize("name", ["fp8_mm_sm100.cu", "mla_consumers_sm100.cu"])
def test_no_read_only_loads(name):
    with open(os.path.join(CSRC, name)) as f:
        code = re.sub(r"//[^\n]*", "", f.read())
    assert "griddepcontrol.wait" in code
    for form in (r"__ldg\s*\(", r"\bld\.global\.nc", r"\bconst\s+[\w:]+\s*\*\s*__restrict__"):
        assert not re.search(form, code), form
