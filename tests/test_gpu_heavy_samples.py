"""The plain FP64 form where a few samples dwarf the others: a sample whose own terms vanish
in an element leaves that element as it is without the sample, whatever its size."""
import numpy as np
import pytest

from conftest import load_hbuild_case
from test_gpu_integer_products import bra

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    import torch
    assert torch.cuda.is_available()
    import scp3_b200
    return scp3_b200


def handle(api, estimator, nm=8, n3=3, chunk=0):
    c = load_hbuild_case("dimer_qtip4pf")
    return api.HBuild(2, c["x0"], c["MUa"], c["omega"], modes=np.arange(nm), n2=nm, n3=n3, estimator=estimator,
                      chunk=chunk)


def add(hb, q, V, Vq):
    hb.reset()
    if hb.estimator == "gradient":
        hb.add_epot_grad(q, V, Vq)
    else:
        hb.add_epot(q, V)
    return hb.read(0)


def data(n, nm, seed):
    rng = np.random.default_rng(seed)
    return rng.normal(scale=np.sqrt(0.5), size=(n, nm)), rng.normal(size=n), rng.normal(size=(n, nm))


# the first and last samples, whole blocks of 32, more than one batch of 32 in a unit,
# several passes
@pytest.mark.parametrize("estimator", ["direct", "gradient"])
@pytest.mark.parametrize("n,at", [(1000, [0]), (1000, [999]), (4096, [31, 32, 63, 64]), (4096, range(64, 128)),
                                  (16384, range(5, 16384, 150)), (9000, [0, 4095, 4096, 8999])])
@pytest.mark.parametrize("size", [1e4, 1e12, 1e200])
def test_vanishing_terms(api, estimator, n, at, size):
    """The heavy samples sit at q = 0, where the functions with an odd level vanish, and
    carry V = size.  Their exact zeros are all that the other elements see: the same
    bits as with V = 0 there (the others' digits do not depend on samples left out)."""
    at = list(at)
    hb = handle(api, estimator, chunk=4096)
    q, V, Vq = data(n, 8, 7)
    q[at], Vq[at], V[at] = 0.0, 0.0, 0.0
    light = add(hb, q, V, Vq)
    V[at] = size
    full = add(hb, q, V, Vq)
    V1 = np.zeros(n)
    V1[at] = V[at]
    alone = add(hb, q, V1, np.zeros_like(Vq))
    zero = alone == 0
    assert zero.any() and not zero.all()
    assert np.array_equal(full[zero], light[zero])
    # the other elements: two sums of FP64 values, rounded where the units of up to four
    # passes and the heavy samples, at most 110 of them, are added
    assert np.abs(full - (light + alone)).max() <= 2.0 ** -43 * (np.abs(light).max() + np.abs(alone).max())
    hb.close()


@pytest.mark.parametrize("size", [50.0, 1e6, 1e100])
def test_heavy_coordinates(api, size):
    """One coordinate far out where V = 0: the functions of that mode are huge there, their
    terms zero."""
    hb = handle(api, "direct")
    q, V, Vq = data(3000, 8, 8)
    V[1234], q[1234] = 0.0, 0.0
    light = add(hb, q, V, Vq)
    q[1234, 3] = size
    assert np.array_equal(add(hb, q, V, Vq), light)
    hb.close()


@pytest.mark.parametrize("outlier", [1.0, 1e2, 1e3, 1e6, 1e9, 1e12])
def test_error_beside_an_outlier(api, outlier):
    """One sample of 2^14 with V = outlier where the functions of mode 0 vanish; their
    elements' error against extended precision.  A row's values are at most ~2^10 times its
    rms (V within 2^8 of its geometric mean, the functions within 8) and are rounded at
    2^-55 of the largest: two rows' roundings over 2^14 random terms come to 2^-55 2^10
    2^-7 = 2^-52 of the terms' sum, the largest of ~10^3 elements to 4 times that."""
    n = 1 << 14
    hb = handle(api, "direct", nm=8, n3=0)
    q, V, _ = data(n, 8, 9)
    q[5000, 0], V[5000] = 0.0, outlier
    M = add(hb, q, V, None)
    P = bra(q, 8, 0)
    i = [1] + [9 + 8 + k for k in range(7)]         # h1(q_0), h1(q_0) h1(q_k)
    assert not P[i, 5000].any()
    W = P * V
    ref, A = P[i] @ W.T, np.abs(P[i]) @ np.abs(W).T
    assert (np.abs(M[i] - ref) / A).max() <= 1e-15
    hb.close()


@pytest.mark.parametrize("estimator", ["direct", "gradient"])
def test_every_scale(api, estimator):
    """V and dV/dq spread evenly over 24 decades: most samples are over the limit of some
    value."""
    import oracle
    rng = np.random.default_rng(10)
    n, nm = 700, 6
    q, V, Vq = data(n, nm, 11)
    V *= 10.0 ** rng.uniform(-12, 12, size=n)
    Vq *= 10.0 ** rng.uniform(-12, 12, size=n)[:, None]
    hb = handle(api, estimator, nm=nm, n3=2)
    M = add(hb, q, V, Vq)
    iu = np.triu_indices(hb.nb)
    if estimator == "direct":
        P = bra(q, nm, 2)
        ref, A = P @ (P * V).T, np.abs(P) @ np.abs(P * V).T
        # FP64's own bound for n terms of three roundings, and the digits' 2^-44 of a row's
        # typical value for those within the limits
        assert (np.abs(M - ref) / A).max() <= (n + 4) * 2.0 ** -53
    else:
        ref = oracle.accumulate_stein(q, V, Vq, nm, 2)
        assert np.abs(M[iu] - ref[iu]).max() <= (n + 8) * 2.0 ** -53 * 2500 * max(np.abs(V).max(), np.abs(Vq).max())
    hb.close()


def test_nan_reaches_only_its_functions(api):
    """A NaN in dV/dq_m enters the gradient estimator's terms of mode m alone."""
    hb = handle(api, "gradient", nm=6, n3=0)
    q, V, Vq = data(300, 6, 12)
    good = add(hb, q, V, Vq)
    Vq[17, 2] = np.nan
    M = add(hb, q, V, Vq)
    has = np.array([False] + [m == 2 for m in range(6)] * 2 + [2 in (m, k) for m in range(6) for k in range(m + 1, 6)])
    assert np.isnan(M[has]).all()
    clean = M[np.ix_(~has, ~has)]
    assert np.isfinite(clean).all() and np.allclose(clean, good[np.ix_(~has, ~has)], rtol=0, atol=1e-11)
    hb.close()
