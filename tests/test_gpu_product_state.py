"""Product states (k_product_state, k_product_rows) against the Kronecker
product of the qubits' normalised pairs, on both sides of the size from which
the state is built from two tables."""
import numpy as np
import pytest

from q1tsim_gb300 import VectorState

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
