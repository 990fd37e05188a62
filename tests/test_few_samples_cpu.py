"""The rule that takes a pass of few samples to FP64 sums instead of digits."""
import ctypes

import pytest

from scp3_b200 import _lib


@pytest.fixture(scope="module")
def rule():
    f = _lib.lib().scp3gpu_internal_few_ranges
    f.argtypes = [ctypes.c_int] * 5 + [ctypes.c_int64]
    f.restype = ctypes.c_int
    return f


@pytest.mark.parametrize("ntiles,half,nsplit,nsum", [(1, 1, 148, 0), (2, 1, 74, 0), (3, 0, 49, 0), (28, 1, 5, 0), (4, 4, 37, 156),
                                                     (114, 0, 5, 2352), (319, 0, 6, 3822), (2000, 3, 1, 0)])
def test_ranges(rule, ntiles, half, nsplit, nsum):
    """Ranges that the plan has and of 8 samples or more; past the first pass that takes the
    digits all larger ones do; the largest do."""
    last = 1
    for k in range(64, 1 << 16, 64):
        r = rule(ntiles, half, nsplit, nsum, 148, k)
        assert 0 <= r <= nsplit and (r <= 1 or k // r >= 8)
        assert last or not r
        last = r
    assert last == 0


def test_bad_arguments(rule):
    assert rule(0, 0, 1, 0, 148, 64) < 0 and rule(1, 0, 1, 0, 148, 0) < 0
