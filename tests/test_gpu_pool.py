"""The transfer pool keeps a bounded amount of device memory, whatever the number of threads
that used it."""
import ctypes
import threading

import numpy as np
import pytest

from test_gpu_water_groups import geometries

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    import torch
    assert torch.cuda.is_available()
    import scp3_b200
    return scp3_b200


def idle():
    from scp3_b200 import _lib
    f = _lib.lib().scp3gpu_internal_staging_idle
    f.argtypes = [ctypes.POINTER(ctypes.c_size_t)]
    held = ctypes.c_size_t()
    return f(ctypes.byref(held)), held.value


def test_idle_memory_is_bounded(api):
    """Calls of 17 MB (32 MB slots) from six threads at once, then small ones."""
    X = np.tile(geometries(2, 64, 5), (1600, 1))
    want = api.PES("qtip4pf").energies(X[:64])
    bad = []

    def work():
        for _ in range(3):
            if not np.array_equal(api.PES("qtip4pf").energies(X).reshape(-1, 64), np.tile(want, (1600, 1))):
                bad.append(1)

    ts = [threading.Thread(target=work) for _ in range(6)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
    slots, held = idle()
    assert 1 <= slots <= 8 and held <= 32 << 20
    assert np.array_equal(api.PES("qtip4pf").energies(X[:64]), want)
