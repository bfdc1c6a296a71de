"""Spectra over the row counts of the cluster-resident tridiagonalisation and
the Sturm eigenvalues: every power of two, one matrix (several CTAs each) and
many (one or four), reduced row counts from measured sites, rank-deficient
and degenerate spectra.

Entropies against numpy's FP64 eigenvalues of the same states, within 1e-10.
"""
import numpy as np
import pytest

from tests.gpu_util import random_state

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mg():
    from mipt_gb300 import build
    build.build()
    import mipt_gb300
    return mipt_gb300


@pytest.fixture(scope="module")
def orc():
    from oracle import pyoracle
    return pyoracle


def entropy(rho):
    lam = np.linalg.eigvalsh(rho)
    lam = lam[lam > 1e-15]
    return float(-(lam * np.log2(lam)).sum())


@pytest.mark.parametrize("k", [5, 6, 7, 8, 9])
def test_one_matrix(mg, orc, k):
    n = 2 * k
    e = mg.Engine(fp64=True)
    ghz = np.zeros(1 << n, complex)
    ghz[0] = ghz[-1] = 2 ** -0.5
    bell = np.zeros((1 << k, 1 << k), complex)
    np.fill_diagonal(bell, 2 ** (-0.5 * k))
    kept = list(range(k))
    for psi in (random_state(n, k), ghz, bell.reshape(-1), np.eye(1, 1 << n, 3, dtype=complex)[0]):
        e.set_state(psi)
        assert abs(mg.entropy_svd(e.data, n, kept, fp64=True) - entropy(orc.rdm(psi, kept))) < 1e-10


@pytest.mark.parametrize("n,count,p", [(10, 170, 0.1), (12, 80, 0.3), (14, 160, 0.05), (16, 3, 0.1), (16, 40, 0.2)])
def test_batches(mg, orc, n, count, p):
    """Half-chain spectra of 32 to 256 rows, the measured layers' smaller ones among them."""
    seeds = np.array([mg.trajectory_seed(31, i) for i in range(count)], np.uint64)
    b = mg.Batch(n, 2, count, fp64=True, observables=mg.OBS_SVN_HALF, observe_every=1)
    got = b.run(seeds, p)["obs"][:, :, 0]
    for i in (0, count // 2, count - 1):
        ref = orc.run_trajectory(int(seeds[i]), n, 2, p, True, 16, 1, 1)
        np.testing.assert_allclose(got[i], ref["obs"][:, 0], rtol=0, atol=1e-10)


@pytest.mark.parametrize("n,count", [(6, 2), (10, 9), (10, 10), (12, 19), (12, 20), (16, 4), (16, 5)])
def test_lanes_per_eigenvalue(mg, orc, n, count):
    """Around the counts at which an eigenvalue is searched by 32 to 4 lanes or by one."""
    test_batches(mg, orc, n, count, 0.15)
