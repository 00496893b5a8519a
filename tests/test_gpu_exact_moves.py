"""Complex128 plans keep what no arithmetic touches: gates of 0, +-1 and +-i
move amplitudes bit for bit, and amplitudes outside a gate's controls keep their
bits.  Amplitudes span 540 to 600 binary orders, with all of their 53 bits; TOP is the
highest (from 2^63 on a tile is done in FP64).  (No tolerance: equal bits.)"""
import numpy as np
import pytest

from oracle import oracle as orc
from q1tsim_gb300 import Plan, VectorState
from q1tsim_gb300 import gates as G
from test_gpu_parity import TOL128, rand_state

pytestmark = pytest.mark.gpu


def _flat(gates):
    return np.concatenate([np.ascontiguousarray(g.matrix()).ravel() for g, _ in gates]).view(np.float64)


TOP = [40, 100]


def _wide_state(n, rng, top):
    a = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    return a * np.exp2(rng.integers(-500, top + 1, 1 << n))


def _bits(a):
    return np.ascontiguousarray(a).view(np.uint64)


def _run(n, gates, amps, width=0, exact=False, tensor_cores=True):
    s = VectorState.from_amplitudes(amps, 1, "c128")
    s.set_fp64_exact(exact)
    s.apply_plan(Plan(n, [b for _, b in gates], width, tensor_cores=tensor_cores), _flat(gates))
    return s.states()[:, 0]


def _one_by_one(n, gates, amps, exact=False):
    s = VectorState.from_amplitudes(amps, 1, "c128")
    s.set_fp64_exact(exact)
    for g, b in gates:
        s.apply_gate(g, b)
    return s.states()[:, 0]


def _unit_gates(n, count, rng):
    one, two = [G.X(), G.Y(), G.Z(), G.S(), G.Sdg()], [G.CX(), G.CY(), G.CZ(), G.Swap()]
    out = []
    for _ in range(count):
        k = int(rng.integers(1, min(n, 3) + 1))
        g = one[rng.integers(5)] if k == 1 else two[rng.integers(4)] if k == 2 else G.CCX()
        out.append((g, [int(q) for q in rng.choice(n, k, replace=False)]))
    return out


@pytest.mark.parametrize("top", TOP)
@pytest.mark.parametrize("width", [0, 2, 5])
@pytest.mark.parametrize("n,count", [(1, 5), (3, 30), (8, 90), (11, 60), (12, 70), (14, 90), (21, 60), (22, 24), (23, 70)])
def test_unit_gates_move_amplitudes(n, count, width, top):
    rng = np.random.default_rng(10 * n + width)
    gates, amps = _unit_gates(n, count, rng), _wide_state(n, rng, top)
    if width and n < 12:
        pytest.skip("blocks of fewer than 12 qubits are dense products")
    np.testing.assert_array_equal(_bits(_run(n, gates, amps, width)), _bits(_one_by_one(n, gates, amps)))


@pytest.mark.parametrize("top", TOP)
@pytest.mark.parametrize("n,count", [(4, 20), (9, 60), (12, 60), (16, 80), (22, 160), (23, 60)])
def test_amplitudes_outside_the_controls_keep_their_bits(n, count, top):
    rng = np.random.default_rng(n)
    gates = []
    for i in range(count):
        c, t = int(rng.integers(0, 2)), int(rng.integers(2, n))
        kind = rng.integers(4)
        ang = rng.uniform(0, 6, 3)
        gates.append((G.CU3(*ang) if kind < 2 else G.CU1(ang[0]) if kind == 2 else G.CX(), [c, t]))
    amps = _wide_state(n, rng, top)
    quarter = 1 << (n - 2)                        # both controls 0: no gate applies
    amps[quarter:] = rng.normal(size=3 * quarter) + 1j * rng.normal(size=3 * quarter)
    got = _run(n, gates, amps)
    np.testing.assert_array_equal(_bits(got[:quarter]), _bits(amps[:quarter]))
    o = orc.OracleState.from_amplitudes(amps, 1)
    for g, b in gates:
        o.apply_gate(g.matrix(), b)
    scale = np.abs(amps[quarter:]).max() * 2
    np.testing.assert_allclose(got[quarter:], o.states()[quarter:, 0], rtol=0, atol=TOL128 * scale)


@pytest.mark.parametrize("n", [9, 14])
def test_controlled_gates_on_infinities(n):
    """Controlled gates alone in a pass: infinities and NaN spread as gate by
    gate, and stay where the controls leave them."""
    rng = np.random.default_rng(n)
    amps = rand_state(n, rng)
    amps[3], amps[-5], amps[1 << (n - 1)] = np.inf, complex(0.0, np.nan), 2.0 ** 200
    gates = [(G.CU3(*rng.uniform(0, 6, 3)), [0, int(t)]) for t in rng.integers(1, n, 12)]
    got, want = _run(n, gates, amps), _one_by_one(n, gates, amps)
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    half = 1 << (n - 1)
    np.testing.assert_array_equal(_bits(got[:half]), _bits(amps[:half]))
    fine = np.isfinite(want) & (np.abs(want) < 2.0 ** 100)
    assert np.max(np.abs(got[fine] - want[fine])) <= 2.0 ** 200 * 1e-12
