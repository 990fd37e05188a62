"""Passes of few samples of the plain FP64 form, whose products are added in FP64, at the
edges of their ranges, batches and tiles, and next to passes that take the digits; and the
digits at the sizes that they are left."""
import ctypes

import numpy as np
import pytest

from conftest import load_hbuild_case
from test_gpu_digit_sums import test_single_digits as single_digits
from test_gpu_integer_products import bra, check

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    import torch
    assert torch.cuda.is_available()
    import scp3_b200
    return scp3_b200


def one_tile_takes_digits(n):
    """A basis of one panel (direct estimator): one tile, as many ranges as SMs."""
    import torch
    from scp3_b200 import _lib
    f = _lib.lib().scp3gpu_internal_few_ranges
    f.argtypes, f.restype = [ctypes.c_int] * 5 + [ctypes.c_int64], ctypes.c_int
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return f(1, 1, sms, 0, sms, (n + 63) // 64 * 64) == 0


def handle(api, estimator, nm, n2, n3):
    c = load_hbuild_case("dimer_qtip4pf" if nm <= 12 else "hexamer_qtip4pf")
    return api.HBuild(2 if nm <= 12 else 6, c["x0"], c["MUa"], c["omega"], modes=np.arange(nm), n2=n2, n3=n3,
                      estimator=estimator)


def data(n, nm, seed):
    rng = np.random.default_rng(seed)
    return rng.normal(scale=np.sqrt(0.5), size=(n, nm)), rng.normal(size=n) * np.exp(3 * rng.normal(size=n)), rng.normal(size=(n, nm))


def size(q, n2, n3):
    """bra with every sum's terms taken absolutely"""
    a = np.abs(q)
    nm, n = q.shape[1], q.shape[0]
    h1, h2, h3 = np.sqrt(2) * a, (2 * a * a + 1) / np.sqrt(2), (2 * a * a + 3) * a / np.sqrt(3)
    f = [np.ones(n)] + [h1[:, m] for m in range(nm)] + [h2[:, m] for m in range(n2)]
    f += [h1[:, m] * h1[:, k] for m in range(n2) for k in range(m + 1, n2)] + [h3[:, m] for m in range(n3)]
    for m in range(n3):
        for k in range(m + 1, n3):
            f += [h2[:, m] * h1[:, k], h1[:, m] * h2[:, k]]
    f += [h1[:, m] * h1[:, k] * h1[:, l] for m in range(n3) for k in range(m + 1, n3) for l in range(k + 1, n3)]
    return np.array(f)


# one, two, three and five panels; one range and several; on both sides of a batch of 32
@pytest.mark.parametrize("nm,n2,n3,n", [(1, 0, 0, 1), (12, 12, 0, 8), (12, 12, 0, 65), (12, 12, 0, 4800), (14, 14, 4, 129), (21, 20, 8, 1000),
                                        (21, 20, 8, 257), (30, 30, 4, 63)])
def test_direct(api, nm, n2, n3, n):
    """A function is a product of three factors at most, each within 6 roundings of the sum
    of its terms' sizes, a product of two functions and V within 40, and a sum of n of them
    within n more: |error| <= (n + 40) 2^-53 sum |terms|."""
    q, V, _ = data(n, nm, n)
    hb = handle(api, "direct", nm, n2, n3)
    hb.add_epot(q, V)
    M = hb.read(0)
    hb.close()
    P, S = bra(q, n2, n3), size(q, n2, n3)
    bound = (n + 40) * 2.0 ** -53 * ((S * np.abs(V)) @ S.T)
    err = np.abs(M - P @ (P * V).T)
    assert np.all(err <= bound), float((err / bound).max())


@pytest.mark.parametrize("nm,n2,n3,n", [(9, 9, 0, 1), (10, 10, 2, 71), (12, 12, 0, 800), (10, 4, 0, 300), (21, 21, 3, 130)])
def test_gradient(api, nm, n2, n3, n):
    """Products, pair sums and summed rows; terms of one sample are at most 2500 |V| or
    |dV/dq|, with 60 roundings."""
    import oracle
    q, V, Vq = data(n, nm, n + 1)
    hb = handle(api, "gradient", nm, n2, n3)
    hb.add_epot_grad(q, V, Vq)
    M = hb.read(0)
    ref = oracle.accumulate_stein(q, V, Vq, n2, n3)
    iu = np.triu_indices(hb.nb)
    hb.close()
    assert np.abs(M[iu] - ref[iu]).max() <= (n + 60) * 2.0 ** -53 * 2500 * np.abs(V).max()


@pytest.mark.parametrize("estimator,nm,n3", [("direct", 12, 0), ("direct", 21, 5), ("gradient", 12, 0), ("gradient", 10, 3)])
def test_passes_add_up(api, estimator, nm, n3):
    """Few samples before and after a pass of digits, in units that hold sums and that do
    not: the sums of the passes alone, to a rounding of each of up to 148 partials and of
    the products behind them."""
    hb = handle(api, estimator, nm, nm, n3)
    total, scale = 0, 0
    for ranges in ([(0, 100)], [(200, 20000)], [(50000, 3)], [(60000, 900)]):
        hb.reset()
        hb.accumulate(ranges[0][0] + 7, ranges[0][1])
        M = hb.read(0)
        total, scale = total + M, scale + np.abs(M).max()
    hb.reset()
    for first, n in [(0, 100), (200, 20000), (50000, 3), (60000, 900)]:
        hb.accumulate(first + 7, n)
    assert np.abs(hb.read(0) - total).max() <= 160 * 2.0 ** -53 * scale
    hb.close()


def test_not_finite(api):
    """As FP64 sums have it: NaN in the functions of the modes concerned."""
    hb = handle(api, "direct", 12, 12, 0)
    q, V, _ = data(100, 12, 3)
    q[5, 3] = np.nan
    hb.add_epot(q, V)
    M = hb.read(0)
    has = np.array([False] + [m == 3 for m in range(12)] * 2 + [3 in (m, k) for m in range(12) for k in range(m + 1, 12)])
    assert np.isnan(M[has]).all() and np.isfinite(M[np.ix_(~has, ~has)]).all()
    V[6] = np.inf
    hb.reset()
    hb.add_epot(q, V)
    assert not np.isfinite(hb.read(0)).any()
    hb.close()


# ---------------------------------------------------------------- the digits beyond
@pytest.mark.parametrize("nm,n2,n3,n", [(9, 9, 0, 16384), (12, 12, 0, 16447), (14, 12, 0, 20033), (21, 20, 8, 8193)])
def test_digits_edges(api, nm, n2, n3, n):
    assert nm > 20 or one_tile_takes_digits(n)
    q, V, _ = data(n, nm, n)
    hb = handle(api, "direct", nm, n2, n3)
    hb.add_epot(q, V)
    check(hb.read(0), q, V, n2, n3)
    hb.close()


@pytest.mark.parametrize("i,j", [(1, 1), (1, 2), (2, 2), (1, 4), (3, 3), (2, 5), (1, 7), (4, 4), (2, 6), (3, 5), (2, 7), (7, 2),
                                 (3, 6), (6, 3), (4, 5), (5, 4), (7, 1), (6, 2)])
def test_digits_single(api, i, j):
    assert one_tile_takes_digits(16001)
    single_digits(api, i, j, 16001)


# heavy samples among the digits: the first and last, whole blocks of 32, more than a batch
# of 32 in a unit
@pytest.mark.parametrize("estimator", ["direct", "gradient"])
@pytest.mark.parametrize("at", [[0], [19999], [31, 32, 63, 64], range(64, 200), range(5, 20000, 150)])
@pytest.mark.parametrize("big", [1e4, 1e200])
def test_digits_vanishing_terms(api, estimator, at, big):
    """Heavy samples at q = 0: the elements whose terms vanish there keep their bits."""
    at, n = list(at), 20000
    assert one_tile_takes_digits(n)
    hb = handle(api, estimator, 8, 8, 3)
    rng = np.random.default_rng(7)
    q, V, Vq = rng.normal(scale=np.sqrt(0.5), size=(n, 8)), rng.normal(size=n), rng.normal(size=(n, 8))
    q[at], Vq[at], V[at] = 0.0, 0.0, 0.0

    def add(V, Vq):
        hb.reset()
        hb.add_epot_grad(q, V, Vq) if estimator == "gradient" else hb.add_epot(q, V)
        return hb.read(0)

    light = add(V, Vq)
    V[at] = big
    full = add(V, Vq)
    V1 = np.zeros(n)
    V1[at] = big
    alone = add(V1, np.zeros_like(Vq))
    zero = alone == 0
    assert zero.any() and not zero.all() and np.array_equal(full[zero], light[zero])
    # two sums of FP64 values, rounded where units and up to 136 heavy samples are added
    assert np.abs(full - (light + alone)).max() <= 2.0 ** -43 * (np.abs(light).max() + np.abs(alone).max())
    hb.close()


@pytest.mark.parametrize("estimator", ["direct", "gradient"])
def test_digits_every_scale(api, estimator):
    """V and dV/dq spread evenly over 24 decades, most samples heavy."""
    import oracle
    n, nm = 16100, 6
    assert one_tile_takes_digits(n)
    rng = np.random.default_rng(10)
    q, V, Vq = rng.normal(scale=np.sqrt(0.5), size=(n, nm)), rng.normal(size=n), rng.normal(size=(n, nm))
    V *= 10.0 ** rng.uniform(-12, 12, size=n)
    Vq *= 10.0 ** rng.uniform(-12, 12, size=n)[:, None]
    hb = handle(api, estimator, nm, nm, 2)
    if estimator == "direct":
        hb.add_epot(q, V)
        P, S = bra(q, nm, 2), size(q, nm, 2)
        bound = (n + 40) * 2.0 ** -53 * ((S * np.abs(V)) @ S.T)
        assert np.all(np.abs(hb.read(0) - P @ (P * V).T) <= bound)
    else:
        hb.add_epot_grad(q, V, Vq)
        ref = oracle.accumulate_stein(q, V, Vq, nm, 2)
        iu = np.triu_indices(hb.nb)
        assert np.abs(hb.read(0)[iu] - ref[iu]).max() <= (n + 60) * 2.0 ** -53 * 2500 * max(np.abs(V).max(), np.abs(Vq).max())
    hb.close()


def test_digits_not_finite(api):
    n = 16100
    assert one_tile_takes_digits(n)
    hb = handle(api, "direct", 12, 12, 0)
    q, V, _ = data(n, 12, 3)
    q[5, 3] = np.nan
    hb.add_epot(q, V)
    M = hb.read(0)
    has = np.array([False] + [m == 3 for m in range(12)] * 2 + [3 in (m, k) for m in range(12) for k in range(m + 1, 12)])
    assert np.isnan(M[has]).all() and np.isfinite(M[np.ix_(~has, ~has)]).all()
    V[6] = np.inf
    hb.reset()
    hb.add_epot(q, V)
    assert not np.isfinite(hb.read(0)).any()
    hb.close()


def test_digits_gradient_not_finite(api):
    """A NaN in dV/dq_m, or V = inf at a sample of digits: as FP64 sums have it."""
    n = 16100
    hb = handle(api, "gradient", 6, 6, 0)
    rng = np.random.default_rng(12)
    q, V, Vq = rng.normal(scale=np.sqrt(0.5), size=(n, 6)), rng.normal(size=n), rng.normal(size=(n, 6))
    hb.add_epot_grad(q, V, Vq)
    good = hb.read(0)
    Vq[17, 2] = np.nan
    hb.reset()
    hb.add_epot_grad(q, V, Vq)
    M = hb.read(0)
    has = np.array([False] + [m == 2 for m in range(6)] * 2 + [2 in (m, k) for m in range(6) for k in range(m + 1, 6)])
    assert np.isnan(M[has]).all()
    clean = M[np.ix_(~has, ~has)]
    # the marked sample's terms, added in FP64 now: a rounding each of sums of 1e5 at most
    assert np.isfinite(clean).all() and np.abs(clean - good[np.ix_(~has, ~has)]).max() <= 1e-9
    V[18] = np.inf
    hb.reset()
    hb.add_epot_grad(q, V, Vq)
    assert not np.isfinite(hb.read(0)).any()
    hb.close()
