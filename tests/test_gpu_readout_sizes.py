"""Read-outs of bases of few tiles, whose sums lie in up to one sample range per SM."""
import numpy as np
import pytest

from conftest import load_hbuild_case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    import torch
    assert torch.cuda.is_available()
    import scp3_b200
    return scp3_b200


# functions: 2, 13, 23, 91, 127, 136, 253, 288: on both sides of 128 and 256
@pytest.mark.parametrize("nm,n2,n3", [(1, 0, 0), (12, 0, 0), (12, 4, 0), (12, 12, 0), (14, 14, 0), (15, 15, 0), (21, 21, 0), (21, 21, 5)])
def test_every_range(api, nm, n2, n3):
    """FP64 products of 2000 samples against the estimators' rules in FP64 (n roundings of
    terms of ~250 at most); the split form's within 2^-16 of the terms' sum, and some; a
    leading dimension of its own on the device."""
    import oracle
    import torch
    n = 2000
    rng = np.random.default_rng(nm + n3)
    q, V, Vq = rng.normal(scale=np.sqrt(0.5), size=(n, nm)), rng.normal(size=n), rng.normal(size=(n, nm))
    c = load_hbuild_case("dimer_qtip4pf" if nm <= 12 else "hexamer_qtip4pf")
    for estimator in ("direct", "gradient"):
        ref = oracle.accumulate(q, V, n2, n3) if estimator == "direct" else oracle.accumulate_stein(q, V, Vq, n2, n3)
        scale = oracle.accumulate(q, V, n2, n3, absolute=True)
        for precision in ("fp64", "bf16x3"):
            hb = api.HBuild(2 if nm <= 12 else 6, c["x0"], c["MUa"], c["omega"], modes=np.arange(nm), n2=n2, n3=n3,
                            precision=precision, estimator=estimator)
            hb.add_epot_grad(q, V, Vq) if estimator == "gradient" else hb.add_epot(q, V)
            M, nb = hb.read(0), hb.nb
            iu = np.triu_indices(nb)
            tol = n * 2.0 ** -53 * 250 if precision == "fp64" else 1e-4 * scale.max() if estimator == "direct" else 2e-4 * scale.max()
            assert np.abs(M[iu] - ref[iu]).max() <= tol
            assert np.array_equal(M, M.T)
            d = torch.full((nb, nb + 3), -1.0, dtype=torch.float64, device="cuda")
            hb.read_dev(d.data_ptr(), nb + 3, 0)
            torch.cuda.synchronize()
            out = d.cpu().numpy()
            assert np.array_equal(out[:, :nb], M) and (out[:, nb:] == -1).all()
            hb.close()
