"""Shot sampling (k_chunk_sums_dense, k_scan_small, k_sample) against FP64
prefix sums: part of a warp's 32 shots and many warps, one chunk and many, with
the chunks' group sums kept (many shots) and recomputed (few), results of 32
and 64 bits.

Tolerance: a shot with uniform u must land where u times the total lies
between the outcome's exclusive and inclusive prefix, up to the rounding of the
sums: 2^-24 per addition of a group (8), a chunk (5 levels) and the offset in
complex64, 2^-53 times the number of chunks' scan levels in FP64."""
import numpy as np
import pytest

from q1tsim_gb300 import Rng, VectorState
from test_gpu_parity import rand_state

pytestmark = pytest.mark.gpu


def _state(n, precision, rng):
    amps = rand_state(n, rng)
    if n > 4:
        amps[rng.integers(0, 1 << n, 1 << (n - 2))] = 0.0
        amps[: 1 << (n - 3)] = 0.0
    amps /= np.linalg.norm(amps)
    return amps.astype(np.complex64).astype(np.complex128) if precision == "c64" else amps


@pytest.mark.parametrize("precision", ["c64", "c128"])
@pytest.mark.parametrize("n,shots", [(1, 5), (3, 33), (7, 32), (8, 1), (8, 31), (9, 2047), (11, 2048), (13, 1000),
                                     (16, 8), (16, 7), (17, 40000), (20, 100), (20, 300000), (22, 140000)])
def test_outcomes_follow_the_prefix(n, shots, precision):
    rng = np.random.default_rng(n * 7 + shots)
    amps = _state(n, precision, rng)
    u = rng.random(shots)
    u[: min(shots, 2)] = [0.0, 1.0 - 2.0 ** -53][: min(shots, 2)]
    prob = np.abs(amps) ** 2
    incl = np.cumsum(prob)
    total = incl[-1]
    tol = (14 * 2.0 ** -24 * total) if precision == "c64" else 64 * 2.0 ** -53 * total
    for cbits in (list(range(n - 1, -1, -1)), [63 - q for q in range(n)]):      # narrow and wide words
        s = VectorState.from_amplitudes(amps, shots, precision)
        words = np.full(shots, (1 << 40) | 5 << 30, dtype=np.uint64)      # other bits stay
        s.peek_all_into(cbits, words, uniforms=u)
        again = words.copy()
        s.measure_all_into(cbits, again, uniforms=u)
        np.testing.assert_array_equal(words, again)
        own = np.bitwise_or.reduce([np.uint64(1) << np.uint64(cb) for cb in cbits])
        other = np.uint64((1 << 40) | 5 << 30) & ~own
        assert np.all((words & ~own) == other)
        idx = np.zeros(shots, dtype=np.int64)
        for q, cb in enumerate(cbits):
            idx |= ((words >> np.uint64(cb)) & np.uint64(1)).astype(np.int64) << (n - 1 - q)
        assert np.all(prob[idx] > 0)
        t = np.sort(u) * total
        assert np.all(incl[idx] - prob[idx] <= t + tol) and np.all(incl[idx] >= t - tol)


@pytest.mark.parametrize("shots", [1, 100, 2046, 2047, 2048, 30000, 140000])
def test_stream_uniforms_are_the_spacings(shots):
    """Sorted uniforms from the stream, in one launch and in several: the same
    words as with the same uniforms given.  (Both sum in FP64; a target moves by
    2^-50 at most, which no outcome of these 13 qubits notices.)"""
    n = 13
    amps = _state(n, "c128", np.random.default_rng(3))
    golden, mask = 0x9E3779B97F4A7C15, (1 << 64) - 1

    def draw(seed, k):
        z = (seed + (k + 1) * golden) & mask
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        return ((z ^ (z >> 31)) >> 11) * 2.0 ** -53

    e = np.array([-np.log1p(-draw(99, k)) for k in range(shots + 1)])
    u = np.cumsum(e)[:-1] / np.cumsum(e)[-1]
    a, b = np.zeros(shots, dtype=np.uint64), np.zeros(shots, dtype=np.uint64)
    s = VectorState.from_amplitudes(amps, shots, "c128")
    s.peek_all_into(list(range(n)), a, rng=Rng(99))
    s.peek_all_into(list(range(n)), b, uniforms=u)
    np.testing.assert_array_equal(a, b)
