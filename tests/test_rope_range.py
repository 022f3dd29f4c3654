"""The range check of RoPE's strides against the set of elements that are touched (host only)."""
import itertools

import pytest
import torch

from amd_developer_challenge_2025_b200.mla import _check_range


@pytest.mark.parametrize("start", [0, 5])
def test_every_element_counts(start):
    t = torch.zeros(40, dtype=torch.bfloat16)[start:]
    for off, d0, d1, s1, s2 in itertools.product((-1, 0, 3, 12, 20, 33, 36), (1, 2, 4), (1, 3), (-9, -4, 0, 4, 9), (-7, 0, 7)):
        touched = [off + i0 * s1 + i1 * s2 + j for i0 in range(d0) for i1 in range(d1) for j in range(4)]
        ok = off >= 0 and 0 <= start + min(touched) and start + max(touched) < 40
        if ok:
            _check_range("x", t, off, d0, d1, 4, s1, s2)
        else:
            with pytest.raises(ValueError):
                _check_range("x", t, off, d0, d1, 4, s1, s2)
