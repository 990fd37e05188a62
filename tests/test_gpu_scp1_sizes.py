"""The SCP1 sums over the cluster sizes: from 64 groups of threads per block (one water) to
two (eight), few samples and many."""
import numpy as np
import pytest

from scp3_b200 import constants as C
from test_gpu_sample_slots import cluster

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    import torch
    assert torch.cuda.is_available()
    import scp3_b200
    return scp3_b200


@pytest.mark.parametrize("nw", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("n", [1, 40, 9000])
def test_sums(api, nw, n):
    """Sums of V, g and g dq^T over the points, each formed in FP64 from potentials that the
    same kernels give: a rounding per term and addition, and 10^-12 of the forces for
    the points' own rounding."""
    dim = 9 * nw
    rng = np.random.default_rng(nw)
    q = cluster(nw)[0]
    d, U = rng.uniform(0.1, 1.0, size=dim), np.linalg.qr(rng.normal(size=(dim, dim)))[0] * 0.03
    s = api.SCP1Average("qtip4pf", nw, chunk=4096)
    v, ux, uxq = s.sums(q, d, U, 5, 2, 2 + n)
    s.close()
    dq = (api.std_normals(dim, 7, n) * np.sqrt(d)) @ U.T
    E, G = api.PES("qtip4pf").energies_grad(C.bohr * (q + dq))
    V, G = E / C.autokcalpmol, G * C.bohr / C.autokcalpmol
    tol = n * 2.0 ** -52 + 1e-12
    assert abs(v - V.sum()) <= tol * np.abs(V).sum()
    assert np.all(np.abs(ux - G.sum(0)) <= tol * (np.abs(G).sum(0) + n * np.abs(G).max()))
    assert np.all(np.abs(uxq - G.T @ dq) <= tol * (np.abs(G).T @ np.abs(dq) + n * np.abs(G).max() * np.abs(dq).max()))
