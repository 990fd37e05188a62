"""The accuracy of the plain FP64 form's digit products: every digit sum that is formed
reaches the matrix, the last one included."""
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


def digit(k):
    """One unit of digit k (1 = most significant) of a row whose largest value is 1: the
    integers are x 2^54, digit k weighs 256^(7 - k)."""
    return 2.0 ** (8 * (7 - k) - 54)


# every group i + j of digits that is formed
@pytest.mark.parametrize("i,j", [(1, 1), (1, 2), (2, 2), (1, 4), (3, 3), (2, 5), (1, 7), (4, 4), (2, 6), (3, 5), (2, 7),
                                 (7, 2), (3, 6), (6, 3), (4, 5), (5, 4), (7, 1), (6, 2)])
@pytest.mark.parametrize("n", [640, 1345])
def test_single_digits(api, i, j, n):
    """V = 1; in one sample of 64 h1(q_0) holds digit i alone and h1(q_1) digit j alone (as
    near as FP64's sqrt(2) q comes); in half of the others the one is 1 and the other zero,
    in half the reverse, which sets the rows' scales (and their geometric means, so that no
    sample is set apart).  <1_0|V|1_1> is then the digit product (i, j) and nothing else: a
    pair that does not reach the matrix is missing altogether."""
    rng = np.random.default_rng(100 * i + j)
    kind = np.arange(n) % 2
    kind[17::64] = 2
    q = np.zeros((n, 3))
    q[:, 0] = np.choose(kind, [np.ones(n), np.zeros(n), rng.integers(20, 61, size=n) * digit(i)])
    q[:, 1] = np.choose(kind, [np.zeros(n), np.ones(n), rng.integers(20, 61, size=n) * digit(j)])
    q /= 1.4142135623730951
    x = 1.4142135623730951 * q                  # h1 in FP64
    c = load_hbuild_case("dimer_qtip4pf")
    hb = api.HBuild(2, c["x0"], c["MUa"], c["omega"], modes=np.arange(3), n2=0, n3=0)
    hb.add_epot(q, np.ones(n))
    M = hb.read(0)
    hb.close()
    want = float(np.sum(x[:, 0].astype(np.longdouble) * x[:, 1].astype(np.longdouble)))
    # the smallest digits are 20 units of their row: half a unit of each is at most 1/40 + 1/40
    assert want > 0 and abs(M[1, 2] - want) <= 0.06 * want


@pytest.mark.parametrize("estimator", ["direct", "gradient"])
def test_norm_of_the_error(api, estimator):
    """2^13 random samples against extended precision.  The integers' rounding and the digit
    sums left out come to ~2e-16 of the matrix's norm; without the pairs i + j = 9 the
    direct form's error is 2.5e-15, the gradient's 5e-16."""
    nm, n = 12, 1 << 13
    rng = np.random.default_rng(5)
    q = rng.normal(scale=np.sqrt(0.5), size=(n, nm))
    V, Vq = rng.normal(size=n), rng.normal(size=(n, nm))
    c = load_hbuild_case("dimer_qtip4pf")
    hb = api.HBuild(2, c["x0"], c["MUa"], c["omega"], modes=np.arange(nm), n2=nm, n3=0, estimator=estimator)
    if estimator == "direct":
        hb.add_epot(q, V)
        P = bra(q, nm, 0)
        ref = P @ (P * V).T
        M = hb.read(0)
    else:
        # <1_m|V|1_k>, m != k: the mean of sum_s dV/dq_m q_k and sum_s dV/dq_k q_m
        hb.add_epot_grad(q, V, Vq)
        T = Vq.astype(np.longdouble).T @ q.astype(np.longdouble)
        off = ~np.eye(nm, dtype=bool)
        ref = (0.5 * (T + T.T))[off]
        M = hb.read(0)[1:1 + nm, 1:1 + nm][off]
    hb.close()
    err = np.linalg.norm((M - ref).astype(float).ravel()) / np.linalg.norm(ref.astype(float).ravel())
    print("error", estimator, err)
    assert err <= 4e-16
