"""Basis states and collapsed columns: the tables that go as kernel parameters
(up to 64 columns) and those that are uploaded, the smallest states, every
position of the measured qubit.  Against numpy, exactly but for the scale's one
rounding."""
import numpy as np
import pytest

from q1tsim_gb300 import Rng, VectorState, gates as G
from test_gpu_parity import rand_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["c64", "c128"])
@pytest.mark.parametrize("n,shots", [(1, 1), (1, 40), (2, 3), (5, 64), (7, 65), (8, 400), (13, 30)])
def test_basis_columns_become_dense(n, shots, precision):
    s = VectorState(n, shots, precision)
    for q in range(n):
        s.apply_gate(G.H(), [q])
    words = s.measure_all(rng=Rng(n + shots))
    s.apply_gate(G.X(), [0])                 # makes the columns dense
    got = s.states()
    cols, runs = got.shape[1], []
    for w in words:                          # neighbouring equal words share a column
        if not runs or runs[-1] != w:
            runs.append(w)
    want = np.zeros((1 << n, cols), dtype=np.complex128)
    for c, w in enumerate(runs):
        idx = sum(((int(w) >> q) & 1) << (n - 1 - q) for q in range(n))
        want[idx ^ (1 << (n - 1)), c] = 1.0
    assert cols == len(runs)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("precision", ["c64", "c128"])
@pytest.mark.parametrize("n,qbits", [(1, [0]), (2, [1, 0]), (6, [5, 0, 3]), (9, [8, 7, 0, 4, 1, 2, 3]), (14, [13, 12, 0])])
def test_collapse_of_every_column(n, qbits, precision):
    rng = np.random.default_rng(n)
    amps = rand_state(n, rng)
    if n > 2:                                # (not the whole state)
        amps[rng.integers(0, 1 << n, 3)] = 0.0
    amps /= np.linalg.norm(amps)
    s = VectorState.from_amplitudes(amps, 2000, precision)
    eps = 2.0 ** -22 if precision == "c64" else 2.0 ** -49
    for step, q in enumerate(qbits):
        before = s.states()
        bits = s.measure(q, rng=Rng(step))
        after = s.states()
        mask = (np.arange(1 << n) >> (n - 1 - q)) & 1
        col = 0
        for c in range(before.shape[1]):
            for keep in (0, 1):
                part = np.where(mask == keep, before[:, c], 0.0)
                norm = np.linalg.norm(part)
                if col < after.shape[1] and norm > 0 and np.allclose(after[:, col], part / norm, atol=1e-4):
                    assert np.all(after[mask != keep, col] == 0)
                    assert np.linalg.norm(after[:, col] - part / norm) <= 8 * eps * len(qbits)
                    col += 1
        assert col == after.shape[1] and set(np.unique(bits)) <= {0, 1}
