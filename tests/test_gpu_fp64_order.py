"""With FP64 arithmetic requested a plan rounds as its gates one by one do,
whichever of them share a tile pass.  (No tolerance: equal bits.)"""
import numpy as np
import pytest

from q1tsim_gb300 import Plan, VectorState
from test_gpu_parity import rand_state, random_gate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 5, 9, 11, 13, 16, 20])
def test_fp64_arithmetic_rounds_in_the_gates_order(n):
    rng = np.random.default_rng(n)
    gates = [random_gate(n, rng) for _ in range(80)]
    amps = rand_state(n, rng)
    run, one = (VectorState.from_amplitudes(amps, 1, "c128") for _ in range(2))
    for s in (run, one):
        s.set_fp64_exact(True)
    flat = np.concatenate([np.ascontiguousarray(g.matrix()).ravel() for g, _ in gates]).view(np.float64)
    run.apply_plan(Plan(n, [b for _, b in gates], 0), flat)
    for g, b in gates:
        one.apply_gate(g, b)
    got, want = (np.ascontiguousarray(s.states()).view(np.uint64) for s in (run, one))
    np.testing.assert_array_equal(got, want)
