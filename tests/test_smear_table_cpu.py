"""The interval of TTM3-F's smearing table that a distance is looked up in: inside the
table for every value of the argument, none for a NaN."""
import ctypes
import struct

import numpy as np
import pytest

from scp3_b200 import _lib


@pytest.mark.parametrize("fp32,limit", [(0, 37.0), (1, 17.0)])
def test_interval(fp32, limit):
    f = _lib.lib().scp3gpu_internal_tail_span
    f.argtypes = [ctypes.c_double, ctypes.c_int]
    f.restype = ctypes.c_int
    t = np.float32 if fp32 else np.float64
    edges = [1.5, 2, 3, 4, 6, 8, 12, 16, 24, 32, 48]
    for k in range(10):
        lo, hi = t(edges[k]), np.nextafter(t(edges[k + 1]), t(0))
        for x in (lo, np.nextafter(lo, t(100)), t(0.5) * (lo + hi), hi):
            assert f(float(x), fp32) == (k if x <= limit else -1), x
    assert f(limit, fp32) == (8 if fp32 else 9) - (1 if fp32 else 0)
    for x in (0.0, -1.0, 1.0, float(np.nextafter(t(1.5), t(0))), float(np.nextafter(t(limit), t(100))), 1e30, np.inf,
              -np.inf, np.nan, -np.nan):
        assert f(x, fp32) == -1, x
    # NaNs of both signs and other payloads
    for bits in (0x7FF8000000000000, 0xFFF8000000000000, 0x7FFFFFFFFFFFFFFF, 0xFFFFFFFFFFFFFFFF, 0x7FF8000020000000):
        assert f(struct.unpack("<d", struct.pack("<Q", bits))[0], fp32) == -1
