"""Von Neumann entropies -sum l log2 l of states that are not normalised: the
eigenvalue search must not depend on the norm's range.

Several lanes per eigenvalue (up to 512 rows) and one (2048 rows), against
numpy's FP64 eigenvalues. Both are exact to about d eps |T| per eigenvalue:
1e-11 of the entropy.
"""
import numpy as np
import pytest

from tests.gpu_util import random_state

pytestmark = pytest.mark.gpu


CASES = [(k, scale) for k in (2, 3, 5, 6, 7, 8, 9) for scale in (2.0 ** -10, 1.0, 1e9, 1e10, 1e12, 1e40)]
CASES += [(11, 1.0), (11, 1e10)]


@pytest.mark.parametrize("k,scale", CASES)
def test_entropy(k, scale):
    from mipt_gb300 import build
    build.build()
    import mipt_gb300 as mg
    n = 2 * k
    e = mg.Engine(fp64=True)
    e.set_state(scale * random_state(n, k))
    m = e.state().reshape(1 << k, 1 << k)  # environment x kept modes 0..k-1
    lam = np.linalg.eigvalsh(m @ m.conj().T)
    lam = lam[lam > 1e-15]
    want = float(-(lam * np.log2(lam)).sum())
    got = mg.entropy_svd(e.data, n, list(range(k)), False, True)
    assert abs(got - want) <= 1e-11 * max(1.0, abs(want))
