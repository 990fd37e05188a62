"""The potentials in groups of four geometries per warp: every number of waters and
ragged groups, against the oracle's energies and their differences."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    import torch
    assert torch.cuda.is_available()
    import scp3_b200
    return scp3_b200


def geometries(nw, n, seed):
    """n geometries of nw waters on a 3.1 A grid, each water turned and its bonds and
    angle moved by a few per cent."""
    rng = np.random.default_rng(seed)
    cells = np.array([(i, j, k) for i in range(3) for j in range(3) for k in range(3)])[:nw] * 3.1
    out = np.empty((n, nw, 3, 3))
    for s in range(n):
        for w in range(nw):
            r1, r2 = 0.96 * (1 + 0.03 * rng.normal(size=2))
            th = np.radians(104.5) * (1 + 0.03 * rng.normal())
            q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
            x = np.array([[0, 0, 0], [r1, 0, 0], [r2 * np.cos(th), r2 * np.sin(th), 0]]) @ q
            out[s, w] = x + cells[w] + 0.1 * rng.normal(size=3)
    return out.reshape(n, 9 * nw)


def energy(pes, x):
    return oracle.qtip4pf(x) if pes == "qtip4pf" else oracle.ttm3f(x)


# TTM3-F takes eight waters four geometries at a time, more of them two at a time
@pytest.mark.parametrize("pes,nw,n", [("qtip4pf", 1, 1), ("qtip4pf", 9, 5), ("qtip4pf", 16, 3), ("ttm3f", 1, 7),
                                      ("ttm3f", 2, 4), ("ttm3f", 5, 2), ("ttm3f", 8, 9), ("ttm3f", 9, 3), ("ttm3f", 10, 1)])
def test_energies(api, pes, nw, n):
    X = geometries(nw, n, nw)
    E, it = api.PES(pes).energies(X, return_iters=True)
    ref = np.array([energy(pes, x) for x in X])
    # each side sums ~10 terms per pair of waters of up to ~100 kcal/mol in FP64, and the
    # monomer's ~2e5 cm^-1 terms; 1e-12 of their sum covers a few hundred roundings
    assert np.abs(E - ref).max() <= 1e-12 * (1000.0 * nw + 1000.0 * nw * nw)
    assert np.all(it == 0) if pes == "qtip4pf" else np.all((it >= 1) & (it <= 500))


@pytest.mark.parametrize("pes,nw,n", [("qtip4pf", 1, 2), ("qtip4pf", 11, 5), ("ttm3f", 1, 3), ("ttm3f", 3, 5), ("ttm3f", 8, 2)])
def test_gradients(api, pes, nw, n):
    X = geometries(nw, n, 40 + nw)
    E, G = api.PES(pes).energies_grad(X)
    h = 1e-3
    for s in (0, n - 1):
        assert abs(E[s] - energy(pes, X[s])) <= 1e-12 * (1000.0 * nw + 1000.0 * nw * nw)
        for c in np.random.default_rng(s).choice(9 * nw, 6, replace=False):
            d = np.zeros(9 * nw)
            d[c] = h
            num = (8 * (energy(pes, X[s] + d) - energy(pes, X[s] - d)) -
                   (energy(pes, X[s] + 2 * d) - energy(pes, X[s] - 2 * d))) / (12 * h)
            # fourth-order differences: h^4 / 30 of the fifth derivative, ~1e7 kcal/mol/A^5
            # for an O-H stretch (2.3^5 of its 4e4 kcal/mol well over 1 A)
            assert abs(G[s, c] - num) <= 1e-6 * max(1.0, np.abs(G[s]).max()), (s, c)


def test_groups_do_not_mix(api):
    """A geometry's energy and gradient do not depend on the group it is in."""
    X = geometries(6, 11, 3)
    for pes in ("qtip4pf", "ttm3f"):
        p = api.PES(pes)
        E, G = p.energies_grad(X)
        for s in range(11):
            e, g = p.energies_grad(X[s:s + 1])
            assert e[0] == E[s] and np.array_equal(g[0], G[s])
        assert np.allclose(p.energies(X), E, rtol=0, atol=1e-9)
