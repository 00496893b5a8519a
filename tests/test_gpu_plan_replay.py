"""One plan run again and again: its kept launches serve only a state of the
same shape with the same matrices, and what they read is neither read before it
is uploaded nor overwritten while it is read, whatever streams the states are
on.  Every result must equal a fresh plan's, bit for bit."""
import numpy as np
import pytest

from q1tsim_gb300 import Plan, VectorState
from q1tsim_gb300 import gates as G

pytestmark = pytest.mark.gpu


def _circuit(n, seed, layers=3):
    rng = np.random.default_rng(seed)
    bits, mats = [], []
    for layer in range(layers):
        for q in range(n):
            bits.append([q])
            mats.append(G.U3(*rng.uniform(0, 6.28, 3)).matrix())
        for q in range(layer % 2, n - 1, 2):
            bits.append([q, q + 1])
            mats.append(G.CU1(float(rng.uniform(0, 6))).matrix())
    return bits, np.concatenate([m.ravel() for m in mats]).view(np.float64)


def _state(n, precision, exact=False, columns=1, dense=True):
    s = VectorState(n, 64, precision)
    s.set_fp64_exact(exact)
    if dense:
        s.fill_random_normal(n)
    if columns > 1:
        s.measure(1, uniforms=np.full(1, 0.5))
        s.measure(2, uniforms=np.full(s.ncols, 0.5))
        assert s.ncols == columns
    return s


def _bits(s):
    return np.ascontiguousarray(s.states()).view(np.uint64)


@pytest.mark.parametrize("width", [0, 3, 5])
@pytest.mark.parametrize("n", [6, 13, 16])
def test_one_plan_on_states_of_any_shape(n, width):
    bits, a = _circuit(n, 1)
    b = _circuit(n, 2)[1]
    plan = Plan(n, bits, width)
    shapes = [("c128", False, 1, True), ("c64", False, 1, True), ("c128", True, 1, True), ("c128", False, 4, True),
              ("c64", False, 4, True), ("c128", False, 1, False), ("c64", False, 1, False)]
    for shape in shapes + shapes[::-1]:
        for mats in (a, a, b, a):
            got, want = _state(n, *shape), _state(n, *shape)
            got.apply_plan(plan, mats)
            want.apply_plan(Plan(n, bits, width), mats)
            np.testing.assert_array_equal(_bits(got), _bits(want))


@pytest.mark.parametrize("precision", ["c64", "c128"])
@pytest.mark.parametrize("n", [10, 18])
def test_one_plan_on_two_streams(n, precision):
    """Tile passes only: nothing in plan_run waits for the device."""
    import torch
    sets = [_circuit(n, seed, 8)[1] for seed in range(3)]
    bits = _circuit(n, 0, 8)[0]
    want = []
    for order in ((0, 1, 2, 0), (0, 0, 1, 2)):
        s = _state(n, precision)
        for k in order:
            s.apply_plan(Plan(n, bits, 0, tensor_cores=False), sets[k])
        want.append(_bits(s))
    plan = Plan(n, bits, 0, tensor_cores=False)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(8):
        x, y = _state(n, precision), _state(n, precision)
        x.set_stream(streams[0].cuda_stream)
        y.set_stream(streams[1].cuda_stream)
        # x: 0 1 2 0, y: 0 0 1 2, no wait between
        for state, k in ((x, 0), (y, 0), (y, 0), (x, 1), (y, 1), (x, 2), (y, 2), (x, 0)):
            state.apply_plan(plan, sets[k])
        np.testing.assert_array_equal(_bits(x), want[0])
        np.testing.assert_array_equal(_bits(y), want[1])
        x.set_stream(None)
        y.set_stream(None)
