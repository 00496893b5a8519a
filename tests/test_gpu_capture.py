"""Device memory and stream capture: a state freed, or grown, in one thread
while another thread's stream is being captured leaves the capture intact
(synchronising the device then would be an invalid call, which ends it)."""
import threading

import numpy as np
import pytest

from q1tsim_gb300 import VectorState, gates as G

pytestmark = pytest.mark.gpu


def _in_thread(fn):
    errors = []

    def work():
        try:
            fn()
        except Exception as e:                    # reported by the main thread
            errors.append(repr(e))

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert not errors, errors


def _capture(fn):
    """fn in another thread while this one captures; the graph must replay."""
    import torch
    x = torch.zeros(1000, device="cuda")
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode="thread_local")
        try:
            x.add_(1.0)
            _in_thread(fn)
            x.add_(2.0)
        finally:
            graph.capture_end()
    graph.replay()
    torch.cuda.synchronize()
    assert bool((x == 3.0).all())


@pytest.mark.parametrize("n", [4, 20, 24])
def test_state_freed_during_a_capture(n):
    states = [VectorState(n, 4, "c128")]
    states[0].apply_gate(G.H(), [0])
    states[0].synchronize()
    _capture(states.clear)
    assert not states


def test_lent_memory_and_plans_freed_during_a_capture():
    """Memory that more streams than the state's may use, and plans'."""
    from q1tsim_gb300 import Plan
    from q1tsim_gb300.sharded import EngineShard
    shard = EngineShard(16, 1, "c128")
    shard.amplitudes().zero_()
    bits = [[q] for q in range(16)]
    plan = Plan(16, bits, 0)
    shard.state.apply_plan(plan, np.tile(np.asarray(G.H().matrix()).ravel(), 16).view(np.float64))
    shard.state.synchronize()
    kept = [shard.state, plan]
    del shard, plan
    _capture(kept.clear)
    assert not kept


def test_state_grown_during_a_capture():
    s = VectorState(16, 64, "c128")
    for q in range(4):
        s.apply_gate(G.H(), [q])
    s.measure(0, uniforms=np.full(1, 0.5))
    assert s.ncols == 2

    def grow():                                   # the old columns go to the kept memory
        for q in range(1, 4):
            s.measure(q, uniforms=np.full(s.ncols, 0.5))

    _capture(grow)
    assert s.ncols == 16
    np.testing.assert_allclose(np.linalg.norm(s.states(), axis=0), 1.0, rtol=0, atol=1e-12)


def test_lent_memory_waits_for_the_callers_stream():
    """A state freed while another stream still reads its amplitudes: a new
    state does not get the memory before the reader is done."""
    import torch
    from q1tsim_gb300.sharded import EngineShard
    n = 22
    for _ in range(4):
        shard = EngineShard(n, 1, "c128")
        a = shard.amplitudes()
        a.copy_(torch.full_like(a, 2.0))
        torch.cuda.synchronize()
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            torch.cuda._sleep(20_000_000)         # some 10 ms
            b = a.clone()
        del a, shard
        s = VectorState(n, 1, "c128")
        s.apply_gate(G.H(), [0])
        s.synchronize()
        stream.synchronize()
        assert bool((b == 2.0).all())
