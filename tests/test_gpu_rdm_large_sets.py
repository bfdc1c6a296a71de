"""Reduced density matrices of kept sets larger than their environment: the
entries on the kept modes, in their order, not only the spectrum. Small-set
and tiled Grams, no environment mode left, both sign conventions, against the
CPU oracle (FP64 1e-12, FP32 1e-6)."""
import numpy as np
import pytest

from tests.gpu_util import random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fp64", [True, False])
@pytest.mark.parametrize("fermion", [False, True])
@pytest.mark.parametrize("n,k", [(1, 1), (2, 2), (3, 2), (5, 3), (6, 6), (8, 6), (9, 7), (8, 8), (11, 8)])
def test_entries(n, k, fermion, fp64):
    from mipt_gb300 import build
    build.build()
    import mipt_gb300 as mg
    from oracle import pyoracle as orc
    e = mg.Engine(fp64=fp64)
    e.set_state(random_state(n, 10 * n + k))
    rng = np.random.default_rng(n + k)
    for kept in (list(range(k)), list(range(n - k, n)), [int(q) for q in rng.permutation(n)[:k]]):
        want = orc.rdm(e.state(), kept, fermion)
        got = mg.rdm_subsystem(e.data, n, kept, fermion, fp64)
        np.testing.assert_allclose(got, want, rtol=0, atol=1e-12 if fp64 else 1e-6)
