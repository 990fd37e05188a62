"""The digit sweeps of the integer contraction: every pair of digits i + j <= 9 once,
each in the accumulator of its sum."""
import ctypes

from scp3_b200 import _lib


def test_every_pair_once():
    f = _lib.lib().scp3gpu_internal_digit_chain
    f.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.POINTER(ctypes.c_int), ctypes.POINTER(ctypes.c_int)]
    seen = []
    for t in range(4):
        d, large = ctypes.c_int(), ctypes.c_int()
        n = f(t, 0, ctypes.byref(d), ctypes.byref(large))
        chain = [d.value]
        for e in range(1, n):
            assert f(t, e, ctypes.byref(d), ctypes.byref(large)) == n
            assert chain[-1] + d.value == (9 - 2 * t if large.value else 8 - 2 * t)
            seen += [(chain[-1], d.value), (d.value, chain[-1])]
            chain.append(d.value)
        assert 2 * chain[-1] == 8 - 2 * t
        seen.append((chain[-1], chain[-1]))
        assert sorted(chain) == list(range(1, n + 1))
    assert sorted(seen) == [(i, j) for i in range(1, 8) for j in range(1, 8) if i + j <= 9]
    assert f(4, 0, ctypes.byref(d), ctypes.byref(large)) < 0
