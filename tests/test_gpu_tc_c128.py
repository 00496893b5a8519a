"""Dense blocks of a complex128 state on the tensor cores (k_fused_tc_c128)
against numpy: every kind of gate position, one tile and many per SM, several
columns, rows of zeros, of far different magnitudes and with infinities.

Tolerance: a row's result is off by at most the dropped digit products, 7 of
64 components each: 7 * 2^22 units of 2^-70 of the row's largest amplitude,
and roundings far below: 2^-45 of it."""
import numpy as np
import pytest

from q1tsim_gb300 import DeviceTimeout, Plan, Rng, VectorState
from test_gpu_parity import rand_state, rand_unitary

pytestmark = pytest.mark.gpu

ROW_TOL = 2.0 ** -45


def _apply(amps, m, qubits, n):
    """(result, each amplitude's row maximum) in complex128."""
    k = len(qubits)
    v = amps.reshape([2] * n)
    v = np.moveaxis(v, qubits, range(k)).reshape(1 << k, -1)
    with np.errstate(all="ignore"):
        y = m @ v
        top = np.broadcast_to(np.abs(v).max(axis=0), y.shape)
    back = lambda a: np.moveaxis(a.reshape([2] * n), range(k), qubits).reshape(-1)  # noqa: E731
    return back(y), back(top)


def _run(amps, m, qubits, n):
    s = VectorState.from_amplitudes(amps, 1, "c128")
    s.profile(True)
    s.apply_plan(Plan(n, [qubits], 5), np.ascontiguousarray(m).ravel().view(np.float64))
    assert s.profile_report()["fused_tc_c128"]["launches"] == 1
    return s.states()[:, 0]


@pytest.mark.parametrize("n,qubits", [
    (12, [0, 1, 2, 3, 4]), (12, [11, 10, 9, 8, 7]), (12, [5, 0, 11, 6, 3]), (12, [11, 2, 9]), (13, [12, 1, 11, 0]),
    (14, [13, 12, 11, 10, 9]), (16, [0, 4, 8, 12, 15]), (17, [1, 0, 2, 16, 15]), (20, [19, 18, 0, 1, 10]),
    (21, [3, 20, 7, 19, 11]), (23, [22, 0, 9, 4, 17]), (23, [18, 19, 20, 21, 22])])
def test_block_matches_numpy(n, qubits):
    rng = np.random.default_rng(n * 100 + len(qubits) + qubits[0])
    amps, m = rand_state(n, rng), rand_unitary(1 << len(qubits), rng)
    want, top = _apply(amps, m, qubits, n)
    got = _run(amps, m, qubits, n)
    assert np.all(np.abs(got - want) <= ROW_TOL * top)
    # and typically far closer: 1e-15 of the norm
    assert np.linalg.norm(got - want) <= 2.5e-15


@pytest.mark.parametrize("scale", [1.0, 2.0 ** 900, 2.0 ** -900])
def test_rows_of_any_magnitude(scale):
    n, qubits = 13, [2, 12, 6, 0, 9]
    rng = np.random.default_rng(8)
    amps = rand_state(n, rng) * scale
    amps[: 1 << 10] = 0.0
    amps[1 << 10: 1 << 11] *= np.exp2(rng.integers(-40, 41, 1 << 10))
    amps[rng.integers(0, 1 << n, 200)] = 0.0
    m = rand_unitary(32, rng)
    want, top = _apply(amps, m, qubits, n)
    got = _run(amps, m, qubits, n)
    assert np.all(np.abs(got - want) <= ROW_TOL * top)


def test_permutation_block_moves_amplitudes_exactly():
    n, qubits = 12, [1, 3, 5, 7, 11]
    rng = np.random.default_rng(2)
    # 40 significant bits: every digit product is kept
    amps = np.round(rng.uniform(-1, 1, 1 << n) * 2.0 ** 40) + 1j * np.round(rng.uniform(-1, 1, 1 << n) * 2.0 ** 40)
    m = np.zeros((32, 32), dtype=np.complex128)
    m[np.arange(32), rng.permutation(32)] = np.array([1, -1, 1j, -1j])[rng.integers(0, 4, 32)]
    want, _ = _apply(amps, m, qubits, n)
    np.testing.assert_array_equal(_run(amps, m, qubits, n), want)


def test_infinities_and_nans_stay_in_their_rows():
    n, qubits = 13, [0, 3, 8, 12, 5]
    rng = np.random.default_rng(4)
    amps, m = rand_state(n, rng), rand_unitary(32, rng)
    amps[77] = np.inf
    amps[4100] = complex(0.0, np.nan)
    want, top = _apply(amps, m, qubits, n)
    got = _run(amps, m, qubits, n)
    fine = np.isfinite(want)
    assert np.array_equal(fine, np.isfinite(got)) and (~fine).sum() == 64
    assert np.all(np.abs(got[fine] - want[fine]) <= ROW_TOL * top[fine])


def test_block_on_several_columns():
    n = 12
    rng = np.random.default_rng(6)
    s = VectorState(n, 8, "c128")
    from q1tsim_gb300 import gates as G
    for q in range(n):
        s.apply_gate(G.U3(0.4 + 0.1 * q, 0.3, 0.2), [q])
    s.measure(2, uniforms=np.full(1, 0.5))
    s.measure(7, uniforms=np.full(2, 0.5))
    before = s.states()
    m, qubits = rand_unitary(32, rng), [1, 4, 6, 9, 11]
    s.apply_plan(Plan(n, [qubits], 5), np.ascontiguousarray(m).ravel().view(np.float64))
    after = s.states()
    assert after.shape[1] > 1
    for c in range(after.shape[1]):
        want, top = _apply(np.ascontiguousarray(before[:, c]), m, qubits, n)
        assert np.all(np.abs(after[:, c] - want) <= ROW_TOL * top)


@pytest.mark.parametrize("n,shots,depth,width", [(22, 1, 3, 0), (22, 1, 6, 0), (21, 5, 4, 0), (22, 1, 3, 3),
                                                 (22, 1, 4, 2)])
def test_plain_gates_as_blocks(n, shots, depth, width):
    """Gates of a plan without fusion, or with narrow blocks, multiplied into blocks where that is
    faster, against the same plan on the CUDA cores.  Tolerance: 2^-45 per pass
    of either (both are some 20 passes of 1e-15)."""
    rng = np.random.default_rng(n + depth)
    bits, mats = [], []
    for layer in range(depth):
        for q in range(n):
            bits.append([q])
            mats.append(rand_unitary(2, rng))
        for q in range(layer % 2, n - 1, 2):
            bits.append([q, q + 1] if q % 3 else [q + 1, q])
            kind = rng.integers(3)
            mats.append(np.eye(4)[[0, 1, 3, 2]] if kind == 0 else np.diag([1, 1, 1, -1]) if kind == 1
                        else np.diag([1, 1, 1, np.exp(1j * rng.uniform(0, 6))]))
    flat = np.concatenate([np.ascontiguousarray(m, dtype=np.complex128).ravel().view(np.float64) for m in mats])
    out = []
    for tc in (True, False):
        s = VectorState(n, shots, "c128")
        s.fill_random_normal(7)
        if shots > 1:                       # several columns
            s.measure(3, rng=Rng(1))
        s.profile(True)
        s.profile_report(reset=True)
        s.apply_plan(Plan(n, bits, width, tensor_cores=tc), flat)
        assert ("fused_tc_c128" in s.profile_report()) == tc
        out.append(s.states())
    assert np.linalg.norm(out[0] - out[1]) <= 40 * 2.0 ** -45 * np.linalg.norm(out[1])


@pytest.mark.parametrize("n", [12, 16, 22])
def test_expired_wait_is_reported_and_the_state_usable(n):
    """A limit that every wait for the MMAs exceeds: an error, nothing left
    behind, and the same plan runs with the default limit."""
    rng = np.random.default_rng(n)
    amps, m, qubits = rand_state(n, rng), rand_unitary(32, rng), [n - 1, 3, 0, 7, 5]
    s = VectorState.from_amplitudes(amps, 1, "c128")
    s.set_wait_limit(1e-9)
    plan, flat = Plan(n, [qubits], 5), np.ascontiguousarray(m).ravel().view(np.float64)
    with pytest.raises(DeviceTimeout):
        s.apply_plan(plan, flat)
    s.set_wait_limit(0)
    s.reset_all()
    s.apply_plan(plan, flat)
    start = np.zeros(1 << n, dtype=np.complex128)
    start[0] = 1.0
    assert np.linalg.norm(s.states()[:, 0] - _apply(start, m, qubits, n)[0]) <= 1e-14
    np.testing.assert_allclose(_run(amps, m, qubits, n), _apply(amps, m, qubits, n)[0], rtol=0, atol=1e-14)
