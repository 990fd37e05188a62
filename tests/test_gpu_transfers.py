"""Results copied out through the pinned pool: sizes below, at and above its pieces, padded
columns, several threads at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    import torch
    assert torch.cuda.is_available()
    import scp3_b200
    return scp3_b200


# 8 KB (one plain copy), 1.0 MB, 12 MB, 12 MB with padded columns
@pytest.mark.parametrize("n2,pad", [(0, 0), (26, 0), (48, 0), (48, 7)])
def test_read_equals_read_dev(api, n2, pad):
    import torch
    from scp3_b200 import inputs
    nw, x0, MUa, omega = inputs.load("prism_qtip4pf")
    modes = np.arange(48 - max(n2, 30), 48, dtype=np.int32) if n2 < 48 else None
    hb = api.HBuild(nw, x0, MUa, omega, modes=modes, n2=n2, precision="bf16x3", chunk=4096)
    hb.accumulate(3, 4096)
    d = torch.empty(hb.nb, hb.nb, dtype=torch.float64, device="cuda")
    hb.read_dev(d.data_ptr(), hb.nb, 1)
    torch.cuda.synchronize()
    out = np.full((hb.nb + pad, hb.nb), np.nan, order="F")
    hb.read(1, out=out)
    assert np.array_equal(out[:hb.nb].T, d.cpu().numpy())
    assert np.isnan(out[hb.nb:]).all()


@pytest.mark.parametrize("pad", [0, 7])
def test_read_into_pinned_memory(api, pad):
    """A pinned destination takes one copy: the same bytes as a pageable one, padding untouched."""
    import torch
    from scp3_b200 import inputs
    nw, x0, MUa, omega = inputs.load("prism_qtip4pf")
    hb = api.HBuild(nw, x0, MUa, omega, n2=48, precision="bf16x3", chunk=4096)
    hb.accumulate(3, 4096)
    block = torch.full((hb.nb, hb.nb + pad), float("nan"), dtype=torch.float64).pin_memory()
    out = block.numpy().T
    hb.read(1, out=out)
    assert np.array_equal(out[:hb.nb], hb.read(1))
    assert np.isnan(out[hb.nb:]).all()


# one call's buffers within a pool slot's pinned memory, its device memory, and neither
@pytest.mark.parametrize("n", [3, 20000, 60000])
def test_potential_from_several_threads(api, n):
    from scp3_b200 import constants as C, inputs
    nw, x0, MUa, omega = inputs.load("prism_qtip4pf")
    rng = np.random.default_rng(n)
    sets = [C.bohr * (x0 + 0.05 * rng.normal(size=(n, x0.size))) for _ in range(3)]
    pes = api.qtip4pf()
    alone = [pes.energies_grad(x) for x in sets]
    got = [None] * 3

    def call(k):
        got[k] = pes.energies_grad(sets[k])

    for _ in range(3):
        ts = [threading.Thread(target=call, args=(k,)) for k in range(3)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        for (e, g), (e0, g0) in zip(got, alone):
            assert np.array_equal(e, e0) and np.array_equal(g, g0)
