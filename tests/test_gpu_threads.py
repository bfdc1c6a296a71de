"""Host threads that launch the same kernel with different shared-memory sizes
at the same time: every call succeeds and gives what it gives alone."""
import threading

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


def together(calls, rounds):
    """Each call `rounds` times in a thread of its own; [(thread's results)]."""
    start = threading.Barrier(len(calls))
    results = [[] for _ in calls]
    errors = []

    def loop(i):
        start.wait()
        try:
            for _ in range(rounds):
                results[i].append(calls[i]())
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=loop, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
    return results


def test_free_fermion_blocks(mg):
    """Blocks of 64 modes (129 KB) beside blocks of 4 (0.6 KB)."""
    seeds = np.array([mg.trajectory_seed(5, 0)], np.uint64)

    def block(n, size):
        return lambda: float(mg.ff_run(seeds, 0.2, n, 2, blocks=[size], tmi=False, host_threads=1)["s_blocks"][0, 0])

    calls = [block(128, 64), block(16, 4)]
    alone = [c() for c in calls]
    for got, want in zip(together(calls, 300), alone):
        assert got == [want] * 300


def test_spectra(mg):
    """Spectra of 128 rows: one CTA per matrix (a batch) beside eight per matrix (one state)."""
    seeds = np.array([mg.trajectory_seed(6, i) for i in range(100)], np.uint64)
    batches = threading.local()

    def batch():
        if not hasattr(batches, "b"):
            batches.b = mg.Batch(14, 1, len(seeds), fp64=True, observables=mg.OBS_SVN_HALF)
        return float(batches.b.run(seeds, 0.0)["obs"][0, 0, 0])

    e = mg.Engine(fp64=True)
    e.set_state(random_state(14, 3))
    calls = [batch, lambda: mg.entropy_svd(e.data, 14, list(range(7)), False, True)]
    alone = [c() for c in calls]
    for got, want in zip(together(calls, 60), alone):
        assert got == [want] * 60
