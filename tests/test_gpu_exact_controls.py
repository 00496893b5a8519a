"""Dense gates with controls in complex128 plans: the amplitudes that the
controls leave out keep their bits, for single gates of three and more targets
and for fused blocks whose gates share a control.  (No tolerance there: equal
bits; the others against numpy.)"""
import numpy as np
import pytest

from oracle import oracle as orc
from q1tsim_gb300 import Plan, VectorState
from q1tsim_gb300 import gates as G
from test_gpu_parity import TOL128, rand_state, rand_unitary

pytestmark = pytest.mark.gpu


def _controlled(u, controls):
    m = np.eye(u.shape[0] << controls, dtype=np.complex128)
    m[-u.shape[0]:, -u.shape[0]:] = u
    return m


def _check(n, width, mats, bits, keep):
    """keep: the basis states (by their index) that no gate may touch."""
    rng = np.random.default_rng(n + width)
    amps = rand_state(n, rng) * np.exp2(rng.integers(-300, 1, 1 << n))
    s = VectorState.from_amplitudes(amps, 1, "c128")
    flat = np.concatenate([np.ascontiguousarray(m, dtype=np.complex128).ravel() for m in mats]).view(np.float64)
    s.apply_plan(Plan(n, bits, width), flat)
    got = s.states()[:, 0]
    np.testing.assert_array_equal(got[keep].view(np.uint64), amps[keep].view(np.uint64))
    o = orc.OracleState.from_amplitudes(amps, 1)
    for m, b in zip(mats, bits):
        o.apply_gate(m, b)
    np.testing.assert_allclose(got, o.states()[:, 0], rtol=0, atol=TOL128 * np.abs(amps).max())


@pytest.mark.parametrize("width", [0, 3, 5])
@pytest.mark.parametrize("n,targets,controls", [(12, 3, 1), (12, 3, 2), (14, 4, 1), (9, 3, 1), (22, 3, 1)])
def test_one_controlled_gate(n, targets, controls, width):
    rng = np.random.default_rng(7)
    qubits = [int(q) for q in rng.choice(n, targets + controls, replace=False)]
    index = np.arange(1 << n)
    keep = np.zeros(1 << n, dtype=bool)
    for q in qubits[:controls]:
        keep |= ((index >> (n - 1 - q)) & 1) == 0
    _check(n, width, [_controlled(rand_unitary(1 << targets, rng), controls)], [qubits], keep)


@pytest.mark.parametrize("width", [3, 4, 5])
@pytest.mark.parametrize("n", [12, 16, 22])
def test_blocks_of_gates_with_a_common_control(n, width):
    rng = np.random.default_rng(n)
    mats, bits = [], []
    for _ in range(24):
        t = int(rng.integers(1, 5)) * 2
        mats.append(G.CU3(*rng.uniform(0, 6, 3)).matrix())
        bits.append([0, t])
        if rng.random() < 0.5:
            mats.append(G.CCX().matrix())
            bits.append([0, t, 1 + int(rng.integers(4)) * 2])
    _check(n, width, mats, bits, np.arange(1 << n) < (1 << (n - 1)))
