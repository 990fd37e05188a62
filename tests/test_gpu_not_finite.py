"""Samples whose geometry is not finite, or has two sites in one place: they read NaN and
are counted, and the others of their group of four are what they are without them."""
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


def spoil(x, kind):
    x = x.copy()
    if kind == "coincident":
        x[12:15] = x[3:6]                    # H1 of the second water on H1 of the first
    elif kind == "same water":
        x[9:18] = x[0:9]
    else:
        x[4] = {"nan": np.nan, "-nan": -np.nan, "inf": np.inf, "-inf": -np.inf}[kind]
    return x


# four geometries a warp up to eight waters, two above
@pytest.mark.parametrize("pes,nw", [("ttm3f", 2), ("ttm3f", 6), ("ttm3f", 9), ("qtip4pf", 3)])
@pytest.mark.parametrize("kind", ["nan", "-nan", "inf", "-inf", "coincident", "same water"])
def test_energies(api, pes, nw, kind):
    p = api.PES(pes)
    X = geometries(nw, 7, 11)
    good = p.energies(X)
    assert np.isfinite(good).all()
    for at in (0, 5):
        Y = X.copy()
        Y[at] = spoil(Y[at], kind)
        E = p.energies(Y)
        assert not np.isfinite(E[at])
        keep = np.arange(7) != at
        assert np.array_equal(E[keep], good[keep])


@pytest.mark.parametrize("pes", ["ttm3f", "qtip4pf"])
def test_gradients_of_coincident_hydrogens(api, pes):
    """Hydrogens do not enter the dipoles' tensors, so these converge and the call returns."""
    X = geometries(3, 6, 12)
    p = api.PES(pes)
    E0, G0 = p.energies_grad(X)
    X[2] = spoil(X[2], "coincident")
    E, G = p.energies_grad(X)
    keep = np.arange(6) != 2
    assert not np.isfinite(E[2]) and not np.isfinite(G[2, 3:6]).any()
    assert np.array_equal(E[keep], E0[keep]) and np.array_equal(G[keep], G0[keep])


@pytest.mark.parametrize("kind", ["nan", "inf"])
def test_gradients_not_finite(api, kind):
    """The dipoles of such a geometry do not converge, which the call reports."""
    X = geometries(3, 6, 12)
    X[2] = spoil(X[2], kind)
    with pytest.raises(RuntimeError):
        api.PES("ttm3f").energies_grad(X)


@pytest.mark.parametrize("precision,estimator", [("fp64", "direct"), ("bf16x3", "direct"), ("bf16x3_pes64", "direct"),
                                                 ("fp64", "gradient"), ("bf16x3", "gradient")])
@pytest.mark.parametrize("name", ["dimer", "hexamer"])
def test_build_from_point_zero(api, precision, estimator, name):
    """Point 0 of the unscrambled sequence is u = 0: its normals are -infinity."""
    from scp3_b200 import inputs, modes
    nw, x0, MUa, omega = inputs.load({"dimer": "cluster_2_800", "hexamer": "cluster_6_100"}[name])
    sel = np.arange(omega.size)[-6:]
    hb = api.HBuild(nw, x0, MUa, omega, modes=sel, n2=6, n3=0, pes="ttm3f", precision=precision, estimator=estimator)
    hb.accumulate(0, 70)
    rc, nonfinite, notconv = hb.status()
    assert nonfinite == 1 and notconv == 1 and rc != 0
    assert np.isnan(hb.read(0)[0, 0])
    hb.reset()
    hb.accumulate(1, 69)
    assert hb.status() == (0, 0, 0) and np.isfinite(hb.read(0)).all()
    hb.close()


def test_normals_not_finite(api):
    from scp3_b200 import inputs
    nw, x0, MUa, omega = inputs.load("cluster_3_700")
    rng = np.random.default_rng(1)
    y = rng.normal(size=(50, omega.size))
    y[7, 3], y[20, 0], y[49, 1] = np.nan, np.inf, -np.inf
    for precision in ("fp64", "bf16x3"):
        hb = api.HBuild(nw, x0, MUa, omega, modes=np.arange(4), n2=4, pes="ttm3f", precision=precision)
        hb.accumulate_normals(y)
        assert hb.status()[1:] == (3, 3)
        hb.close()


def test_batch_and_scp1(api):
    from scp3_b200 import inputs
    nw, x0, MUa, omega = inputs.load("cluster_2_800")
    b = api.Batch([dict(nw=nw, x0=x0, MUa=MUa, omega=omega)] * 2, pes="ttm3f")
    b.accumulate(0, 40)
    assert b.status(0)[1:] == (1, 1) and b.status(1)[1:] == (1, 1)
    b.close()
    s = api.SCP1Average("ttm3f", 2)
    q, d, U = geometries(2, 1, 3)[0] / 0.5291772, np.full(18, 1e-4), np.eye(18)
    v, ux, uxq = s.sums(q, d, U, 0, 0, 30)
    assert np.isnan(v) and np.isnan(ux).any() and s.not_converged() == 1
    v, ux, uxq = s.sums(q, d, U, 0, 1, 30)
    assert np.isfinite(v) and np.isfinite(ux).all() and np.isfinite(uxq).all()
    s.close()
