"""A withheld half tile: the FP32 pass gives up with a status, whichever half
is missing.

Two bonds away from the tile's edges make a pass of one round whose halves are
loaded apart, and 256 tiles give its first CTA a second tile, so with the upper
half missing the wait runs out while the next tile's lower half is on its way.
Nothing faults, and the next call gives the right state (FP32, 1e-6).
"""
import numpy as np
import pytest

from tests.gpu_util import random_state

pytestmark = pytest.mark.gpu

E_INTERNAL = 9004
N, PAIRS = 22, [(4, 5), (6, 7)]


@pytest.fixture(scope="module")
def mg():
    from mipt_gb300 import build
    build.build()
    import mipt_gb300
    return mipt_gb300


@pytest.mark.parametrize("halves", [1, 2, 3])
def test_withheld_half(mg, halves):
    rng = np.random.default_rng(halves)
    psi = random_state(N, halves)
    u = [np.linalg.qr(rng.normal(size=(4, 4)) + 1j * rng.normal(size=(4, 4)))[0] for _ in PAIRS]
    e = mg.Engine(fp64=False)
    e.set_state(psi)
    assert mg.lib().mipt_gb300_test_withhold_tile_halves(1, halves) == 0
    with pytest.raises(mg.MiptError) as ei:
        e.apply_bonds(PAIRS, u)
    assert ei.value.status == E_INTERNAL, ei.value
    assert "tile load wait timed out" in str(ei.value)
    e.set_state(psi)
    e.apply_bonds(PAIRS, u)
    want = psi
    for (q, _), m in zip(PAIRS, u):
        want = np.einsum("ij,ajb->aib", m, want.reshape(-1, 4, 1 << q)).reshape(-1)
    np.testing.assert_allclose(e.state(), want, rtol=0, atol=1e-6)


def test_arguments(mg):
    for count, halves in ((-1, 3), (1, 0), (1, 4)):
        assert mg.lib().mipt_gb300_test_withhold_tile_halves(count, halves) != 0
    assert mg.lib().mipt_gb300_test_withhold_tile_loads(-1) != 0
