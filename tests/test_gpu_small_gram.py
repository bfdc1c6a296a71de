"""Entropies of kept sets of up to six modes (the small-set Gram) against the
CPU FP64 oracle, at the edges of its chunks, sub-blocks and splits.

Tolerances: FP64 entropies 1e-10, FP32 1e-5 (the method's |dS| bound).
"""
import numpy as np
import pytest

from tests.gpu_util import random_state

pytestmark = pytest.mark.gpu

TOL = {True: 1e-10, False: 1e-5}


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


def kept_sets(n):
    """One mode to six, low, high, scattered and unordered ones."""
    rng = np.random.default_rng(n)
    out = []
    for k in range(1, min(6, n) + 1):
        out += [list(range(k)), list(range(n - k, n)), [int(q) for q in rng.permutation(n)[:k]]]
    return out


@pytest.mark.parametrize("fp64", [True, False])
@pytest.mark.parametrize("fermion", [False, True])
@pytest.mark.parametrize("n", [2, 5, 7, 11, 12, 15])
def test_single_states(mg, orc, fp64, fermion, n):
    psi = random_state(n, 50 + n)
    e = mg.Engine(fp64=fp64)
    e.set_state(psi)
    stored = e.state()
    for kept in kept_sets(n):
        rho = orc.rdm(stored, kept, fermion)
        assert abs(mg.entropy_svd(e.data, n, kept, fermion, fp64) - orc.entropy(rho, 1)) < TOL[fp64], kept
        assert abs(mg.renyi2(e.data, n, kept, fermion, fp64) - orc.entropy(rho, 2)) < TOL[fp64], kept
        if 2 * len(kept) <= n:
            np.testing.assert_allclose(mg.rdm_subsystem(e.data, n, kept, fermion, fp64), rho, rtol=0,
                                       atol=1e-12 if fp64 else 1e-6)


@pytest.mark.parametrize("fp64", [True, False])
@pytest.mark.parametrize("n,count", [(8, 90), (12, 3)])
def test_measured_batches(mg, orc, fp64, n, count):
    """Regions reduced by measured sites; 90 trajectories give the launches of
    the many-job purity sums."""
    periods, p = 3, 0.4
    seeds = np.array([mg.trajectory_seed(21, i) for i in range(count)], np.uint64)
    b = mg.Batch(n, periods, count, fp64=fp64, observables=15, observe_every=1)
    got = b.run(seeds, p)
    for i in (0, 1, count - 1):
        ref = orc.run_trajectory(int(seeds[i]), n, periods, p, True, 16, 15, 1)
        np.testing.assert_allclose(got["obs"][i], ref["obs"], rtol=0, atol=TOL[fp64])
