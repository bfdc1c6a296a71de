"""FP32 layer passes at the edges of their tiles (10 to 14 local qubits, whole
chains inside one tile, second passes with few bonds, rounds that cannot split
the tile in halves), with fused histograms of few to all sites, open and
closed, Haar and parity-preserving gates, against the CPU oracle: outcomes
equal, amplitudes within 2e-5."""
import numpy as np
import pytest

from tests.gpu_util import mask_of

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


def state_of(mg, batch, i, n):
    e = mg.Engine(fp64=False)
    e.adopt(batch.state_ptr(i), n)
    return e.state()


@pytest.mark.parametrize("n,tile,closed,p", [(10, 0, True, 0.3), (10, 0, False, 1.0), (12, 0, True, 0.05),
                                             (12, 10, True, 0.4), (12, 11, False, 0.4), (14, 0, True, 0.5),
                                             (14, 12, True, 0.2), (16, 0, True, 0.25), (16, 0, False, 0.9),
                                             (16, 13, True, 0.25), (18, 0, True, 0.1), (18, 11, False, 0.3)])
def test_haar_batches(mg, orc, n, tile, closed, p):
    periods, count = 2, 3
    seeds = np.array([mg.trajectory_seed(61, i) for i in range(count)], np.uint64)
    b = mg.Batch(n, periods, count, closed=closed, fp64=False, tile_qubits=tile)
    got = b.run(seeds, p)
    for i in range(count):
        d = orc.haar_draw(int(seeds[i]), n, periods, p, closed, 16)
        r = orc.run_trajectory(int(seeds[i]), n, periods, p, closed, 16, 0, 0, want_state=True)
        for t in range(2 * periods):
            sites = d["sites"][t, : d["sites_per_layer"][t]]
            assert int(got["outcomes"][i, t]) == mask_of(sites, r["outcomes"][t, : len(sites)])
        np.testing.assert_allclose(state_of(mg, b, i, n), r["psi"], rtol=0, atol=2e-5)


@pytest.mark.parametrize("circuit", [2, 4])
@pytest.mark.parametrize("n", [12, 16, 18])
def test_parity_sector_states(mg, circuit, n):
    """Half-size parity-sector states (parity-selected gates in the rounds)
    against the same trajectories on full states."""
    seeds = np.array([mg.trajectory_seed(71, i) for i in range(2)], np.uint64)
    out = []
    for full in (False, True):
        b = mg.Batch(n, 2, 2, fp64=False, circuit=circuit, full_state=full)
        r = b.run(seeds, 0.3)
        out.append((r["outcomes"], [state_of(mg, b, i, n) for i in range(2)]))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    for x, y in zip(out[0][1], out[1][1]):
        np.testing.assert_allclose(x, y, rtol=0, atol=2e-5)
