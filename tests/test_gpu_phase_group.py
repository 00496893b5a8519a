"""Groups of phase runs in one pass (k_phase_group) against the oracle: the
group's positions at the edges (2 is the lowest it takes), pivots inside and
outside the group, constant and linear phases, a leading plain gate, repeated
positions (which end a group; one step left over is no group) and several
columns."""
import numpy as np
import pytest

from oracle import oracle as orc
from q1tsim_gb300 import Plan, VectorState
from q1tsim_gb300 import gates as G
from test_gpu_parity import TOL64, rand_state

pytestmark = pytest.mark.gpu


def _steps(n, targets, rng, leading):
    """(gate, qubits): per target position a run of phases around a pivot,
    then a gate on the target."""
    at = lambda p: n - 1 - p  # noqa: E731
    out = []
    if leading:
        out.append((G.H(), [0]))
    for k, t in enumerate(targets):
        pivot = targets[k - 1] if k % 2 else int(rng.integers(n))
        for q in range(n):
            if at(q) == at(pivot):
                continue
            if rng.random() < 0.7:
                out.append((G.CU1(float(rng.uniform(0, 6.28))), [at(q), at(pivot)]))
        out += [(G.CZ(), [at(pivot), at((pivot + 1) % n)]) for _ in range(3)]   # at least kMinPhaseRun gates
        if k % 3 == 1:
            out += [(G.RZ(0.7), [at(t)]), (G.U1(1.1), [at(pivot)]), (G.T(), [0])]
        out.append((G.H() if k % 2 else G.U3(*rng.uniform(0, 6.28, 3)), [at(t)]))
    return out


def _plan(n, gates):
    flat = np.concatenate([np.ascontiguousarray(g.matrix()).ravel() for g, _ in gates]).view(np.float64)
    return Plan(n, [b for _, b in gates], 5, kinds=[g.plan_kind() for g, _ in gates]), flat


@pytest.mark.parametrize("leading", [False, True])
@pytest.mark.parametrize("n,targets,groups", [
    (4, [2, 3], 1), (5, [4, 3, 2], 1), (10, [9, 8, 7, 6], 1), (11, [2, 10, 5, 3, 7], 1), (13, [12, 4, 4, 2, 11, 3], 2),
    (13, [5, 1, 6, 0, 8], 0), (16, [15, 14, 13, 12, 11, 10, 9, 8, 7], 2)])
def test_groups_match_oracle(n, targets, groups, leading):
    rng = np.random.default_rng(n + len(targets))
    gates = _steps(n, targets, rng, leading)
    amps = rand_state(n, rng)
    o = orc.OracleState.from_amplitudes(amps, 1)
    for g, b in gates:
        o.apply_gate(g.matrix(), b)
    s = VectorState.from_amplitudes(amps, 1, "c64")
    s.profile(True)
    plan, flat = _plan(n, gates)
    s.apply_plan(plan, flat)
    rep = s.profile_report()
    if not leading:
        assert rep.get("phase_group_c64", {"launches": 0})["launches"] == groups
    np.testing.assert_allclose(s.states()[:, 0], o.states()[:, 0], rtol=0, atol=TOL64)


def test_group_on_several_columns():
    n = 9
    rng = np.random.default_rng(1)
    gates = _steps(n, [8, 6, 2, 5], rng, False)
    both = [orc.OracleState.new(n, 16), VectorState(n, 16, "c64")]
    for s in both:
        for q in range(n):
            s.apply_gate(G.U3(0.3 + q, 0.2, 0.1).matrix(), [q])
    for s in both:
        s.measure_into(4, 0, np.zeros(16, dtype=np.uint64), uniforms=np.full(1, 0.5))
    plan, flat = _plan(n, gates)
    both[1].apply_plan(plan, flat)
    for g, b in gates:
        both[0].apply_gate(g.matrix(), b)
    assert both[1].ncols == 2
    np.testing.assert_allclose(both[1].states(), both[0].states(), rtol=0, atol=TOL64)
