"""The plain form's integer products at their edges: k-block and tile remainders, wide
ranges of V, values that are not finite, runs longer than one accumulator holds."""
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


def bra(q, n2, n3):
    nm, n = q.shape[1], q.shape[0]
    h1, h2, h3 = np.sqrt(2) * q, (2 * q * q - 1) / np.sqrt(2), (2 * q * q - 3) * q / np.sqrt(3)
    f = [np.ones(n)] + [h1[:, m] for m in range(nm)] + [h2[:, m] for m in range(n2)]
    f += [h1[:, m] * h1[:, k] for m in range(n2) for k in range(m + 1, n2)] + [h3[:, m] for m in range(n3)]
    for m in range(n3):
        for k in range(m + 1, n3):
            f += [h2[:, m] * h1[:, k], h1[:, m] * h2[:, k]]
    f += [h1[:, m] * h1[:, k] * h1[:, l] for m in range(n3) for k in range(m + 1, n3) for l in range(k + 1, n3)]
    return np.array(f, dtype=np.longdouble)


def check(M, q, V, n2, n3):
    """Every value is rounded at 2^-55 of its row's power of two, at most twice the row's
    largest, and the digit pairs left out of a product lie below 2^-52 of it:
    |error| <= n 2^-51 max|Phi_i| max|V Phi_j| (either row may be the one with V), with
    FP64's own rounding of the values and of the sum beside it."""
    P = bra(q, n2, n3)
    W = P * V
    A = np.abs(P) @ np.abs(W).T
    big, wbig = np.abs(P).max(1), np.abs(W).max(1)
    bound = q.shape[0] * 2.0 ** -51 * np.maximum(np.outer(big, wbig), np.outer(wbig, big)) + 2.0 ** -49 * A
    err = np.abs(M - (P @ W.T))
    assert np.all(err <= bound), float((err / bound).max())


# bases on both sides of one and two 128-row panels; samples on both sides of a k-block
@pytest.mark.parametrize("nm,n2,n3,n", [(1, 0, 0, 1), (12, 12, 0, 63), (14, 14, 2, 64), (14, 14, 4, 65),
                                        (21, 21, 1, 4097), (21, 20, 8, 129)])
def test_add_epot_edges(api, nm, n2, n3, n):
    rng = np.random.default_rng(n)
    q = rng.normal(scale=np.sqrt(0.5), size=(n, nm))
    V = rng.normal(size=n) * np.exp(3 * rng.normal(size=n))
    me = api.ScaledMatrixElements(np.linspace(0.001, 0.02, nm), n2, n3)
    nb = me.getBasisSize()
    M = me.addEpot(q.T, V, np.zeros((nb, nb), order="F"))
    check(M, q, V, n2, n3)
    # a second call on the handle starts from zero again
    assert np.array_equal(me.addEpot(q.T, V, np.zeros((nb, nb), order="F")), M)


@pytest.mark.parametrize("scale", [1e-250, 1e-30, 1e60, 1e250])
def test_scales_of_v(api, scale):
    rng = np.random.default_rng(3)
    q = rng.normal(scale=np.sqrt(0.5), size=(300, 9))
    V = rng.normal(size=300)
    me = api.ScaledMatrixElements(np.linspace(0.001, 0.02, 9), 9, 3)
    nb = me.getBasisSize()
    M = me.addEpot(q.T, V * scale, np.zeros((nb, nb), order="F"))
    check(M / scale, q, V, 9, 3)


def test_zero_and_not_finite(api):
    rng = np.random.default_rng(4)
    q = rng.normal(scale=np.sqrt(0.5), size=(200, 12))
    me = api.ScaledMatrixElements(np.linspace(0.001, 0.02, 12), 12, 0)
    nb = me.getBasisSize()
    assert not me.addEpot(q.T, np.zeros(200), np.zeros((nb, nb), order="F")).any()
    for bad in (np.nan, np.inf, -np.inf):
        V = rng.normal(size=200)
        V[77] = bad
        assert not np.isfinite(me.addEpot(q.T, V, np.zeros((nb, nb), order="F"))).any()
    # a mode at rest: rows of zeros inside the panels
    V = rng.normal(size=200)
    qz = q.copy()
    qz[:, 4] = 0.0
    check(me.addEpot(qz.T, V, np.zeros((nb, nb), order="F")), qz, V, 12, 0)
    qb = q.copy()
    qb[5, 3] = np.nan            # only the functions that excite mode 3
    M = me.addEpot(qb.T, V, np.zeros((nb, nb), order="F"))
    has = np.array([False] + [m == 3 for m in range(12)] * 2 + [3 in (m, k) for m in range(12) for k in range(m + 1, 12)])
    assert not np.isfinite(M[has]).any() and np.isfinite(M[np.ix_(~has, ~has)]).all()


def test_long_runs(api):
    """A pass of 2^17 samples gives a unit 26215 of them, more than the 18432 a 32-bit
    accumulator is allowed: the same sums as in passes of 2^16."""
    from scp3_b200 import inputs
    nw, x0, MUa, omega = inputs.load("prism_qtip4pf")
    out = []
    for chunk in (1 << 17, 1 << 16):
        hb = api.HBuild(nw, x0, MUa, omega, chunk=chunk)
        hb.accumulate(5, (1 << 17) - 100)
        out.append(hb.read(0))
        hb.close()
    d = np.sqrt(np.abs(np.diag(out[0])))
    assert np.abs(out[0] - out[1]).max() <= 1e-12 * np.abs(out[1]).max()
    assert (np.abs(out[0] - out[1]) / np.outer(d, d)).max() <= 1e-12


@pytest.mark.parametrize("n3", [0, 2])
def test_gradient_products(api, n3):
    """Both estimators' sums of one build against the oracle's rule: pair sums as products
    and summed rows (doubles basis), levels up to three."""
    import oracle
    rng = np.random.default_rng(8)
    nm, n = 10, 131
    q = rng.normal(scale=np.sqrt(0.5), size=(n, nm))
    V, Vq = rng.normal(size=n), rng.normal(size=(n, nm))
    c = load_hbuild_case("dimer_qtip4pf")
    hb = api.HBuild(2, c["x0"], c["MUa"], c["omega"], modes=np.arange(nm), n2=nm, n3=n3, estimator="gradient")
    hb.add_epot_grad(q, V, Vq)
    M = hb.read(0)
    ref = oracle.accumulate_stein(q, V, Vq, nm, n3)
    iu = np.triu_indices(hb.nb)
    # terms of one sample are at most ~50 |V| or |Vq|; n 2^-51 of the rows' largest as above
    assert np.abs(M[iu] - ref[iu]).max() <= n * 2.0 ** -51 * 50 * 50 * max(np.abs(V).max(), np.abs(Vq).max())


@pytest.mark.parametrize("estimator", ["direct", "gradient"])
@pytest.mark.parametrize("nm,n", [(9, 1), (12, 65), (12, 4097)])
def test_reset_leaves_nothing(api, estimator, nm, n):
    """After a reset the sums are those of a new handle, bit for bit, also where the next
    pass is too small to reach every unit of the plan; passes add up; nothing
    accumulated reads as zero."""
    c = load_hbuild_case("dimer_qtip4pf")
    new = lambda: api.HBuild(2, c["x0"], c["MUa"], c["omega"], modes=np.arange(nm), n2=nm, n3=0, estimator=estimator)
    hb = new()
    assert not hb.read(0).any()
    hb.accumulate(3, 20000)
    full = hb.read(0)
    hb.reset()
    assert not hb.read(0).any()
    hb.accumulate(50000, n)
    small = hb.read(0)
    other = new()
    other.accumulate(50000, n)
    assert np.array_equal(small, other.read(0)) and small.any()
    hb.accumulate(3, 20000)
    both = hb.read(0)
    # two sums of FP64 values: a rounding of each of at most 148 partials
    assert np.abs(both - (full + small)).max() <= 150 * 2.0 ** -53 * (np.abs(full) + np.abs(small)).max() * 2
