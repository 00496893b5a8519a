"""Runs of plain gates in one tile pass (gate_run.cu) against the gates
applied one by one and the oracle, at the edges of its range: states smaller
than a block of threads, than a tile, of one and of several tiles, several
columns, and amplitudes that the double-float split does not take."""
import numpy as np
import pytest

from oracle import oracle as orc
from q1tsim_gb300 import Plan, VectorState
from q1tsim_gb300 import gates as G
from test_gpu_parity import TOL64, TOL128, rand_state, random_gate

pytestmark = pytest.mark.gpu


def _gates(n, count, seed):
    rng = np.random.default_rng(seed)
    return [random_gate(n, rng) for _ in range(count)]


def _flat(gates):
    return np.concatenate([np.ascontiguousarray(g.matrix()).ravel() for g, _ in gates]).view(np.float64)


def _both(n, gates, prec, amps, exact=False):
    """(by one plan, gate by gate, launches of tile passes)."""
    run, one = (VectorState.from_amplitudes(amps, 1, prec) for _ in range(2))
    for s in (run, one):
        s.set_fp64_exact(exact)
    run.profile(True)
    # dense gates of three qubits take the same kernel on both sides
    run.apply_plan(Plan(n, [b for _, b in gates], 0, tensor_cores=False), _flat(gates))
    tiles = sum(v["launches"] for k, v in run.profile_report().items() if k.startswith("gate_run"))
    for g, b in gates:
        one.apply_gate(g, b)
    return run.states()[:, 0], one.states()[:, 0], tiles


@pytest.mark.parametrize("prec,exact", [("c128", False), ("c128", True), ("c64", False)])
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 10, 11, 12, 13, 16, 21])
def test_runs_match_single_gates(prec, exact, n):
    gates = _gates(n, 90 if n < 16 else 60, 100 * n)
    amps = rand_state(n, np.random.default_rng(n))
    run, one, tiles = _both(n, gates, prec, amps, exact)
    assert tiles > 0
    # gates on disjoint qubits may change places, so roundings differ: the
    # precisions' bounds for whole circuits
    tol = TOL64 if prec == "c64" else TOL128
    np.testing.assert_allclose(run, one, rtol=0, atol=tol)
    o = orc.OracleState.from_amplitudes(amps, 1)
    for g, b in gates:
        o.apply_gate(g.matrix(), b)
    np.testing.assert_allclose(run, o.states()[:, 0], rtol=0, atol=tol)


@pytest.mark.parametrize("prec", ["c128", "c64"])
def test_runs_on_several_columns(prec):
    n, shots = 10, 64
    gates = _gates(n, 40, 5)
    run, one = (VectorState(n, shots, prec) for _ in range(2))
    for s in (run, one):
        s.apply_gate(G.H(), [3])
        s.apply_gate(G.RY(1.0), [8])
        s.measure(3, uniforms=np.full(1, 0.5))
        s.measure(8, uniforms=np.full(2, 0.5))
    assert run.ncols == 4
    run.apply_plan(Plan(n, [b for _, b in gates], 0), _flat(gates))
    for g, b in gates:
        one.apply_gate(g, b)
    np.testing.assert_allclose(run.states(), one.states(), rtol=0,
                               atol=TOL128 if prec == "c128" else TOL64)


@pytest.mark.parametrize("n", [9, 14])
def test_runs_on_extreme_magnitudes(n):
    """Amplitudes of 2^63 and more, infinities and NaN go through FP64 (whole
    tiles), far smaller ones keep an absolute error under 2^-98."""
    rng = np.random.default_rng(3)
    amps = rand_state(n, rng)
    amps[: 1 << (n - 2)] *= 2.0 ** 70
    amps[1 << (n - 1):] *= 2.0 ** -80
    gates = [(G.U3(*rng.uniform(0, 6, 3)), [q]) for q in range(2, n)] + [(G.CX(), [n - 2, n - 1]), (G.T(), [n - 1])]
    run, one, tiles = _both(n, gates, "c128", amps)
    assert tiles > 0
    for part, tol in ((slice(0, 1 << (n - 2)), 2.0 ** 70 * 1e-12), (slice(1 << (n - 2), 1 << (n - 1)), 1e-12),
                      (slice(1 << (n - 1), None), 2.0 ** -80 * 1e-5)):
        assert np.max(np.abs(run[part] - one[part])) <= tol
    amps[5] = np.inf
    amps[1 << (n - 1)] = np.nan
    run, one, _ = _both(n, gates, "c128", amps)
    assert np.array_equal(np.isfinite(run), np.isfinite(one))
