"""The per-sample kernels over the cluster sizes, with groups of four samples cut short: the
normals of a group lie where its geometries go."""
import numpy as np
import pytest

from scp3_b200 import constants as C

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    import torch
    assert torch.cuda.is_available()
    import scp3_b200
    return scp3_b200


def cluster(nw):
    """Waters 3.1 A apart on a grid, every one turned; modes that displace each coordinate
    by ~0.03 bohr."""
    rng = np.random.default_rng(nw)
    w = np.array([[0, 0, 0], [0.9572, 0, 0], [-0.24, 0.9266, 0]])
    x = [w @ np.linalg.qr(rng.normal(size=(3, 3)))[0].T + 3.1 * np.array([i % 3, i // 3 % 3, i // 9]) for i in range(nw)]
    nm0 = 9 * nw - 6
    return np.concatenate(x).ravel() / C.bohr, rng.normal(size=(9 * nw, nm0)) * 0.04 / np.sqrt(nm0), np.linspace(0.001, 0.017, nm0)


@pytest.mark.parametrize("pes,nw", [("qtip4pf", n) for n in (1, 2, 7, 8, 12, 16)] + [("ttm3f", n) for n in (1, 4, 5, 8)])
@pytest.mark.parametrize("precision,estimator", [("fp64", "direct"), ("bf16x3", "direct"), ("fp64", "gradient"), ("bf16x3", "gradient")])
def test_potential_of_points(api, pes, nw, precision, estimator):
    """<0|V|0> of 1 to 3000 points is the sum of the potentials at the back-transformed
    points.  FP64: coordinates to 1e-14 A under forces of up to ~10^3 kcal/mol/A over 9 nw
    of them, 1e-10 kcal/mol, or 2e-13 hartree a point; FP32: 10^9 times that."""
    x0, MUa, omega = cluster(nw)
    hb = api.HBuild(nw, x0, MUa, omega, modes=np.arange(3), n2=0, n3=0, pes=pes, precision=precision, scramble_seed=3,
                    estimator=estimator)
    for n in (1, 3, 70, 3000):
        q = api.std_normals(omega.size, 11, n, scramble_seed=3) / np.sqrt(2.0)
        E = api.PES(pes).energies(C.bohr * (x0 + q @ MUa.T))
        V = E / C.autokcalpmol - 0.5 * (omega * q * q).sum(1)
        hb.reset()
        hb.accumulate(11, n)
        assert hb.status() == (0, 0, 0)
        tol = 2e-13 if precision == "fp64" else 2e-4
        assert abs(hb.read(0)[0, 0] - V.sum()) <= tol * n * (1 + np.abs(V).max())
    hb.close()
