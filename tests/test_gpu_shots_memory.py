"""Shots are sampled without the group sums where the device has no room for
them: the same words."""
import numpy as np
import pytest

from q1tsim_gb300 import VectorState, gates as G
from q1tsim_gb300.vectorstate import release_cached_memory

pytestmark = pytest.mark.gpu


def test_shots_without_room_for_the_group_sums():
    import torch
    n, shots = 29, 200000                         # 256 MiB of group sums

    def words(limit):
        s = VectorState(n, shots, "c64")
        s.fill_random_normal(3)
        few = np.zeros(shots, dtype=np.uint64)
        s.synchronize()
        hold = None
        if limit:
            release_cached_memory()
            free = torch.cuda.mem_get_info()[0]
            hold = torch.empty(free - (192 << 20), dtype=torch.uint8, device="cuda")
        try:
            s.peek_all_into(list(range(n)), few, uniforms=np.random.default_rng(1).random(shots))
        finally:
            del hold
            torch.cuda.empty_cache()
        return few

    # (the sampler without groups is loaded before the memory is taken)
    s = VectorState(20, 1, "c64")
    s.apply_gate(G.H(), [0])
    s.measure_all(uniforms=np.full(1, 0.3))
    free_words = words(False)
    np.testing.assert_array_equal(words(True), free_words)
