"""What a state keeps beside its columns: the columns that a measurement has
split or a conditional gate has spread are not kept by the state; they serve
others, once nothing uses them any more, and count as free."""
import numpy as np
import pytest

from q1tsim_gb300 import VectorState, device_info, gates as G
from q1tsim_gb300.vectorstate import release_cached_memory

pytestmark = pytest.mark.gpu

SLACK = 160 << 20


@pytest.mark.parametrize("how", ["measure", "conditional"])
def test_split_columns_leave_no_memory_behind(how):
    n, column = 25, 16 << 25                      # 512 MiB a column
    s = VectorState(n, 64, "c128")
    s.apply_gate(G.H(), [0])
    s.synchronize()
    before = device_info()["free_bytes"]
    if how == "measure":
        s.measure(0, uniforms=np.full(1, 0.5))
    else:
        s.apply_conditional_gate(np.arange(64) < 32, G.X(), [3])
    assert s.ncols == 2
    s.synchronize()
    # one column more than before, and no third one
    assert before - device_info()["free_bytes"] <= column + SLACK
    release_cached_memory()
    import torch
    assert torch.cuda.mem_get_info()[0] >= before - column - SLACK

def test_released_columns_are_not_reused_while_in_use():
    """Splits of one state and new states on other streams, with nothing waited
    for between: the old columns go from one to the other."""
    import torch
    n = 20
    streams = [torch.cuda.Stream() for _ in range(3)]
    states = []
    for i, st in enumerate(streams):
        s = VectorState(n, 64, "c128")
        s.set_stream(st.cuda_stream)
        s.fill_random_normal(i)
        states.append(s)
    first = [s.states()[:, 0] for s in states]
    gates = [G.X(), G.S(), G.Y()]
    control = np.arange(64) < 32
    for rounds in range(2):
        for s in states:
            for g in gates:
                s.apply_gate(g, [4])
        for i, s in enumerate(states):
            if rounds == 0:
                s.apply_conditional_gate(control, G.X(), [0])
            else:
                s.apply_conditional_gate(np.arange(64) % 32 < 16, G.Z(), [1])
    for s, a in zip(states, first):
        def gate(m, q, v):
            v = np.moveaxis(v.reshape([2] * n), q, 0).reshape(2, -1)
            return np.moveaxis((m @ v).reshape([2] * n), 0, q).reshape(-1)
        unit = G.Y().matrix() @ G.S().matrix() @ G.X().matrix()
        a = gate(unit, 4, a)
        cols = []
        for x in (True, False):
            c = gate(unit, 4, gate(G.X().matrix(), 0, a) if x else a)
            cols += [gate(G.Z().matrix(), 1, c), c]
        np.testing.assert_array_equal(s.states(), np.stack(cols, axis=1))
    for s in states:
        s.set_stream(None)
