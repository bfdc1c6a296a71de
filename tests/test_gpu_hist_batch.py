"""A trajectory's Born sums are the same whatever the rest of its batch.

Layers of several chunks (stand-alone histograms), with measurement rates at
which some trajectories' chunks stream and others' need a staged tile: the
surprisals are the same numbers alone and in the batch.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fp64", [True, False])
@pytest.mark.parametrize("n,chunk_bits", [(10, 3), (12, 4), (14, 5), (16, 8), (18, 6)])
def test_surprisals_do_not_depend_on_the_batch(n, chunk_bits, fp64):
    from mipt_gb300 import build
    build.build()
    import mipt_gb300 as mg
    p = np.repeat([0.3, 0.5, 0.7, 0.8, 0.9, 0.95], 3)
    seeds = np.array([mg.trajectory_seed(83, i) for i in range(len(p))], np.uint64)
    together = mg.Batch(n, 2, len(p), fp64=fp64, chunk_bits=chunk_bits).run(seeds, p)
    one = mg.Batch(n, 2, 1, fp64=fp64, chunk_bits=chunk_bits)
    for i in range(len(p)):
        alone = one.run(seeds[i:i + 1], p[i:i + 1])
        np.testing.assert_array_equal(alone["outcomes"][0], together["outcomes"][i])
        np.testing.assert_array_equal(alone["surprisal"][0], together["surprisal"][i])
