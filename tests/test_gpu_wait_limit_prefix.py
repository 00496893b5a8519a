"""A state's wait limit also holds for the passes that a plan runs on the
compact state of its leading blocks."""
import numpy as np
import pytest

from q1tsim_gb300 import DeviceTimeout, Plan, VectorState
from test_gpu_parity import rand_unitary

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["c64", "c128"])
def test_expiry_in_the_compact_prefix(precision):
    n = 24
    rng = np.random.default_rng(5)
    # blocks on the last 13 qubits: all of the plan is prefix
    bits = [[23, 22, 21, 20, 19], [18, 17, 16, 15, 14], [19, 18, 13, 12, 11]]
    mats = [rand_unitary(32, rng) for _ in bits]
    flat = np.concatenate([m.ravel() for m in mats]).view(np.float64)
    s = VectorState(n, 1, precision)
    s.set_wait_limit(1e-9)
    with pytest.raises(DeviceTimeout):
        s.apply_plan(Plan(n, bits, 5), flat)
    s.set_wait_limit(0)
    s.reset_all()
    s.apply_plan(Plan(n, bits, 5), flat)
    assert abs(float(np.linalg.norm(s.states()[:, 0])) - 1.0) <= 1e-5
