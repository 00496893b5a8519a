"""Complex128 tensor-core passes with infinities and NaN in many rows of many
tiles: rows finished apart and the other lanes of their warps meet again, with
the lowest positions as rows (straight to memory) and as gates.

Tolerance: test_gpu_tc_c128's, 2^-45 of a row's largest amplitude."""
import numpy as np
import pytest

from test_gpu_parity import rand_state, rand_unitary
from test_gpu_tc_c128 import ROW_TOL, _apply, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,qubits", [(12, [0, 1, 2, 3, 4]), (12, [11, 10, 9, 8, 7]), (16, [3, 5, 7, 9, 1]),
                                      (21, [2, 4, 6, 8, 0]), (21, [20, 19, 18, 3, 4])])
def test_many_rows_with_infinities(n, qubits):
    rng = np.random.default_rng(n + qubits[0])
    amps, m = rand_state(n, rng), rand_unitary(32, rng)
    hit = rng.integers(0, 1 << n, (1 << n) // 150)
    amps[hit] = np.array([np.inf, -np.inf, complex(0.0, np.nan), complex(np.inf, 1.0)])[rng.integers(0, 4, len(hit))]
    want, top = _apply(amps, m, qubits, n)
    got = _run(amps, m, qubits, n)
    fine = np.isfinite(want)
    assert np.array_equal(fine, np.isfinite(got)) and 0 < fine.sum() < fine.size
    assert np.all(np.abs(got[fine] - want[fine]) <= ROW_TOL * top[fine])
