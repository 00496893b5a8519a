"""Device memory that freed states leave for new ones: a state in reused
memory starts as any other, from several threads and streams at once; the memory
kept is bounded, and returned on request."""
import threading

import numpy as np
import pytest

from q1tsim_gb300 import Plan, VectorState, device_info
from q1tsim_gb300 import gates as G
from q1tsim_gb300.vectorstate import release_cached_memory

pytestmark = pytest.mark.gpu


def _check(n, precision, seed):
    s = VectorState(n, 3, precision)
    for q in range(0, n, 2):
        s.apply_gate(G.X(), [q])
    want = sum(1 << (n - 1 - q) for q in range(0, n, 2))
    got = s.states()[:, 0]
    assert got[want] == 1.0 and np.count_nonzero(got) == 1
    s.fill_random_normal(seed)                    # leaves anything but zeros behind
    s.apply_plan(Plan(n, [[0], [0, 1]], 5), np.concatenate(
        [G.H().matrix().ravel(), G.CX().matrix().ravel()]).astype(np.complex128).view(np.float64))


def test_reused_memory_from_threads_and_streams():
    import torch
    failures = []

    def work(t):
        try:
            rng = np.random.default_rng(t)
            with torch.cuda.stream(torch.cuda.Stream()):
                for i in range(12):
                    _check(int(rng.integers(3, 19)), ("c64", "c128")[(t + i) % 2], 100 * t + i)
        except Exception as e:                    # reported by the main thread
            failures.append(repr(e))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures


def test_kept_memory_is_bounded_and_returned():
    import torch
    release_cached_memory()
    free0 = torch.cuda.mem_get_info()[0]
    for n in (28, 27, 28, 26, 28, 29, 27, 28):    # 1 to 8 GiB
        s = VectorState(n, 1, "c128")
        s.apply_gate(G.H(), [0])
        del s
    kept = free0 - torch.cuda.mem_get_info()[0]
    assert 0 < kept <= (4 << 30) + (256 << 20)
    assert device_info()["free_bytes"] >= free0 - (256 << 20)
    release_cached_memory()
    assert free0 - torch.cuda.mem_get_info()[0] <= 256 << 20
