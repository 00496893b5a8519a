"""Product states (k_product_state, k_product_rows) against the Kronecker
product of the qubits' normalised pairs, on both sides of the size from which
the state is built from two tables."""
import numpy as np
import pytest

from q1tsim_gb300 import Plan, Rng, VectorState, gates as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["c128", "c64"])
@pytest.mark.parametrize("n", [1, 10, 14, 15, 16, 21])
def test_product_state_is_the_kronecker_product(prec, n):
    rng = np.random.default_rng(n)
    c = rng.normal(size=(n, 2)) + 1j * rng.normal(size=(n, 2))
    c[n // 2] = [0.0, 1.0j]
    want = np.ones(1, dtype=np.complex128)
    for q in range(n):
        want = np.kron(want, c[q] / np.linalg.norm(c[q]))
    got = VectorState.from_qubit_coefs(c.ravel(), 1, prec).states()[:, 0]
    # n + 1 roundings of 2^-53 (complex product: twice that) per amplitude in
    # FP64; one rounding to FP32 on top of it in complex64
    tol = (2 * n + 2) * 2.0 ** -52 + (2.0 ** -23 if prec == "c64" else 0.0)
    np.testing.assert_array_less(np.abs(got - want), tol * np.abs(want) + 1e-300)


@pytest.mark.parametrize("n,first", [(2, 0), (5, 3), (11, 0), (15, 6), (18, 17), (24, 0)])
def test_leading_one_qubit_gates_as_a_product_state(n, first):
    """A plan's leading one-qubit gates on a basis state become a product state;
    against the gates one by one in FP64, to 2^-48 per gate (of the ones behind,
    in double-float pairs)."""
    rng = np.random.default_rng(n)
    bits = [[q] for q in rng.permutation(n)[: max(2, n - first)]] + [[int(rng.integers(n))] for _ in range(2)]
    bits += [[0, 1]] + [[q] for q in range(n)]
    mats = [np.linalg.qr(rng.normal(size=(1 << len(b), 1 << len(b))) + 1j * rng.normal(size=(1 << len(b), 1 << len(b))))[0]
            for b in bits]
    mats[-n - 1] = np.eye(4)[[0, 1, 3, 2]]
    flat = np.concatenate([np.ascontiguousarray(m, dtype=np.complex128).ravel().view(np.float64) for m in mats])
    out = []
    for lead in (True, False):
        s = VectorState(n, 1, "c128")
        if first:                                # another basis state than |0...0>
            for q in range(first):
                s.apply_gate(G.X(), [q])
            s.measure_all(rng=Rng(1))
        if lead:
            s.profile(True)
            s.apply_plan(Plan(n, bits, 0), flat)
            assert s.profile_report()["product_state"]["launches"] == 1
        else:
            s.set_fp64_exact(True)
            for b, m in zip(bits, mats):
                s.apply_gate(m, b)
        out.append(s.states()[:, 0])
    assert np.linalg.norm(out[0] - out[1]) <= len(bits) * 2.0 ** -48
