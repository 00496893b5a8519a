"""Phase runs whose angles are not numbers: in complex64 plans of several runs
(which share a pass) the NaN reaches the amplitudes that it reaches gate by
gate, and no others."""
import numpy as np
import pytest

from q1tsim_gb300 import Plan, VectorState
from q1tsim_gb300 import gates as G
from test_gpu_parity import rand_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("at", [0, 1, 2])
def test_nan_phase_spreads_as_gate_by_gate(at):
    n = 10
    gates = []
    for k in range(3):                            # three ladders and a gate after each
        for q in range(k + 1, n):
            gates.append([G.CU1(0.3 * q + k).matrix(), [q, k], Plan.KIND_DIAGONAL])
        gates.append([G.RX(0.4).matrix(), [k], Plan.KIND_GENERAL])
    first = [0, n, 2 * n - 1][at]
    gates[first + 2][0] = np.diag([1, 1, 1, complex(np.nan, np.nan)])
    amps = rand_state(n, np.random.default_rng(1))
    run, one = (VectorState.from_amplitudes(amps, 1, "c64") for _ in range(2))
    flat = np.concatenate([np.ascontiguousarray(m, dtype=np.complex128).ravel() for m, _, _ in gates]).view(np.float64)
    run.apply_plan(Plan(n, [b for _, b, _ in gates], 5, kinds=[k for _, _, k in gates]), flat)
    for m, b, _ in gates:
        one.apply_gate(m, b)
    a, b = run.states()[:, 0], one.states()[:, 0]
    assert np.isnan(b).any() and not np.isnan(b).all()
    np.testing.assert_array_equal(np.isnan(a), np.isnan(b))
    fine = ~np.isnan(b)
    np.testing.assert_allclose(a[fine], b[fine], rtol=0, atol=2e-6)
