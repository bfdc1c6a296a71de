"""Single-state layers over the sizes where the engine's tile and the streamed
histogram change (9 to 20 qubits, odd ones too; measured sites among the tile's
lowest bits, elsewhere, and all of them), against the CPU oracle: outcomes
equal, amplitudes 1e-12 (FP64) and 2e-5 (FP32)."""
import numpy as np
import pytest

from tests.gpu_util import haar_layer, random_state

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


@pytest.mark.parametrize("fp64", [True, False])
@pytest.mark.parametrize("n", [8, 9, 10, 11, 13, 15, 16, 17, 20])
def test_layer(mg, orc, fp64, n):
    rng = np.random.default_rng(n)
    psi = random_state(n, 80 + n)
    e = mg.Engine(fp64=fp64)
    e.set_state(psi)
    pairs, mats = haar_layer(n - n % 2, 11 + n, start=1)
    e.apply_bonds(pairs, mats)
    want = psi.copy()
    for (a, b), m in zip(pairs, mats):
        want = orc.apply_bond(want, int(a), int(b), m.reshape(4, 4))
    tol = 1e-12 if fp64 else 2e-5
    np.testing.assert_allclose(e.state(), want, rtol=0, atol=tol)
    for sites in ([0], [1, 3], [n - 1], list(range(0, n, 3)), sorted(int(q) for q in rng.permutation(n)[: n // 2]),
                  list(range(n))):
        u = rng.random((len(sites) + 15) // 16)
        before = e.state()
        out, sp = e.measure_layer(sites, u)
        ref = orc.measure_layer(before, sites, u)
        np.testing.assert_array_equal(out, ref[1])
        np.testing.assert_allclose(e.state(), ref[0], rtol=0, atol=tol)
