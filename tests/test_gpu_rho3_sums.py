"""How the three-site blocks' environment sums are added up.

States whose squared amplitudes are powers of two, on columns of chosen
threads, so that the right sum is known exactly: threads' sums are added in
FP64, a plain FP32 run is no longer than 2^(n-11) columns up to n = 14 and 16
from n = 15 on, and a sum that leaves the range is infinite.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SUBS = [[0, 1, 2]]  # environment column e of row 0 is amplitude 8 e


def first_entry(n, amplitudes, fp64):
    from mipt_gb300 import build
    build.build()
    import mipt_gb300 as mg
    psi = np.zeros(1 << n, complex)
    for column, a in amplitudes.items():
        psi[8 * column] = a
    e = mg.Engine(fp64=fp64)
    e.set_state(psi)
    got = np.asarray(mg.rho3_subsystems(e.data, n, SUBS, False, fp64)).reshape(-1)
    return got.view(np.float64)[0]


@pytest.mark.parametrize("fp64", [True, False])
@pytest.mark.parametrize("n", [6, 10, 14, 20])
def test_threads_are_added_in_fp64(n, fp64):
    assert first_entry(n, {0: 1.0, 1: 2.0 ** -13, 2: 2.0 ** -26}, fp64) == 1.0 + 2.0 ** -26 + 2.0 ** -52


@pytest.mark.parametrize("n", [10, 11, 12, 13, 14, 15, 20])
def test_fp32_run_length(n):
    """Squares of 2^-26 are lost beside a 1 in one FP32 run, and only there."""
    columns = max(1, 1 << (n - 10))
    run = max(1, min(16, 1 << max(0, n - 11)))
    amplitudes = {128 * j: 2.0 ** -13 for j in range(1, columns)}
    amplitudes[0] = 1.0
    lost = 1.0 + (columns - 1) * 2.0 ** -26 - first_entry(n, amplitudes, False)
    assert 0.0 <= lost <= (run - 1) * 2.0 ** -26


@pytest.mark.parametrize("fp64", [True, False])
def test_overflow_is_infinite(fp64):
    assert first_entry(12, {0: 2.0 ** (600 if fp64 else 70), 5: 1.0}, fp64) == np.inf


@pytest.mark.parametrize("exponent", [-60, -63, -65, -70, -74])
def test_small_sums_are_exact(exponent):
    """Sums around and below the smallest normal FP32 number."""
    assert first_entry(12, {0: 2.0 ** exponent, 1: 2.0 ** exponent}, False) == 2.0 ** (2 * exponent + 1)
