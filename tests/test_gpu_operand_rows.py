"""Renyi-2 of FP32 states by pre-split operand rows: row blocks of 128 and
more rows, the fewest environment columns, scattered and fermionic kept sets,
rows past the reduced block of measured states.

S_2 against the FP64 oracle on the same state, within 1e-5 (the FP32 Gram's
documented error).
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


@pytest.mark.parametrize("fermion", [False, True])
@pytest.mark.parametrize("n,k", [(11, 7), (12, 7), (14, 7), (15, 8), (16, 9)])
def test_scattered_sets(mg, orc, n, k, fermion):
    psi = random_state(n, 70 + n)
    e = mg.Engine(fp64=False)
    e.set_state(psi)
    stored = e.state()
    rng = np.random.default_rng(n)
    for kept in (list(range(k)), list(range(n - k, n)), [int(q) for q in rng.permutation(n)[:k]]):
        want = orc.entropy(orc.rdm(stored, kept, fermion), 2)
        assert abs(mg.renyi2(e.data, n, kept, fermion, False) - want) < 1e-5, kept


@pytest.mark.parametrize("count,p", [(1, 0.6), (5, 0.4), (33, 0.2)])
def test_measured_batches(mg, orc, count, p):
    n = 16
    seeds = np.array([mg.trajectory_seed(77, i) for i in range(count)], np.uint64)
    b = mg.Batch(n, 2, count, fp64=False, observables=mg.OBS_S2_HALF, observe_every=1)
    got = b.run(seeds, p)["obs"][:, :, 1]
    for i in (0, count - 1):
        ref = orc.run_trajectory(int(seeds[i]), n, 2, p, True, 16, orc.OBS_S2, 1)
        np.testing.assert_allclose(got[i], ref["obs"][:, 1], rtol=0, atol=1e-5)
