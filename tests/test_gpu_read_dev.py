"""Where a read-out on the device may go: memory of the device, pinned memory by a copy, and
not into memory that the driver does not know."""
import numpy as np
import pytest

from conftest import load_hbuild_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("estimator", ["direct", "gradient"])
def test_destinations(estimator):
    import torch
    import scp3_b200
    c = load_hbuild_case("dimer_qtip4pf")
    hb = scp3_b200.HBuild(2, c["x0"], c["MUa"], c["omega"], modes=c["modes"], n2=int(c["n2"]), estimator=estimator)
    hb.accumulate(5, 2000)
    want, nb = hb.read(1), hb.nb
    for d in (torch.full((nb, nb + 5), -1.0, dtype=torch.float64, device="cuda"),
              torch.full((nb, nb + 5), -1.0, dtype=torch.float64).pin_memory()):
        hb.read_dev(d.data_ptr(), nb + 5, 1)
        torch.cuda.synchronize()
        out = d.cpu().numpy()
        assert np.array_equal(out[:, :nb], want) and (out[:, nb:] == -1).all()
    plain = np.full((nb, nb), -1.0)
    with pytest.raises(Exception, match="device memory"):
        hb.read_dev(plain.ctypes.data, nb, 1)
    assert (plain == -1).all()
    assert np.array_equal(hb.read(1), want)
    hb.close()
