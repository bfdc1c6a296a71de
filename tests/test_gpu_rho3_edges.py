"""Three-site blocks at the edges of the sweep's column counter (fewer modes
than a thread index, one step, odd sizes), both sign conventions, unordered
triples, and batches whose pending collapse measures the triple's sites,
against the CPU oracle (FP64 1e-12, FP32 2e-6)."""
import numpy as np
import pytest

from tests.gpu_util import random_state

pytestmark = pytest.mark.gpu

TOL = {True: 1e-12, False: 2e-6}


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


@pytest.mark.parametrize("fp64", [True, False])
@pytest.mark.parametrize("fermion", [False, True])
@pytest.mark.parametrize("n", [3, 4, 9, 10, 11, 15, 17])
def test_single_states(mg, orc, fp64, fermion, n):
    psi = random_state(n, 70 + n)
    e = mg.Engine(fp64=fp64)
    e.set_state(psi)
    rng = np.random.default_rng(n)
    subs = [[0, 1, 2], [n - 1, 0, 1]] + [[int(q) for q in rng.permutation(n)[:3]] for _ in range(4)]
    got = mg.rho3_subsystems(e.data, n, subs, fermion, fp64)
    np.testing.assert_allclose(got, orc.rho3(e.state(), subs, fermion).reshape(-1), rtol=0, atol=TOL[fp64])


@pytest.mark.parametrize("fp64", [True, False])
@pytest.mark.parametrize("n,count", [(8, 3), (14, 2)])
def test_measured_batches(mg, orc, fp64, n, count):
    """Blocks with the last layer's collapse pending, and a run of fewer
    trajectories than the batch has room for."""
    seeds = np.array([mg.trajectory_seed(51, i) for i in range(count)], np.uint64)
    b = mg.Batch(n, 2, count + 60, fp64=fp64, observe_every=1, rho3=True)
    b.run(seeds, 0.5)
    points = b.fetch_rho3_points()
    subs = [[i, (i + 1) % n, (i + 2) % n] for i in range(n)]
    for i in range(count):
        ref = orc.run_trajectory(int(seeds[i]), n, 2, 0.5, True, 16, 0, 0, want_state=True)
        want = orc.rho3(ref["psi"], subs).reshape(n, 128)
        np.testing.assert_allclose(points[i, -1], want, rtol=0, atol=TOL[fp64])
