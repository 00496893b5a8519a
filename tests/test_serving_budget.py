"""The serving budget counts the group sums that measure_all keeps for many
shots (1/16 of the state, up to 1 GiB), and refuses only what does not fit
without them."""
import pytest

from q1tsim_gb300 import Circuit
from q1tsim_gb300.serving import Request, Server


def _request(n, shots, precision="c64"):
    return Request(0, Circuit(n, n, precision=precision), shots, 1)


@pytest.mark.parametrize("n,shots,precision,groups", [
    (20, 4096, "c64", 1 << 19), (20, 4096, "c128", 1 << 20), (20, 127, "c64", 0), (20, 128, "c64", 1 << 19),
    (7, 4096, "c64", 0), (8, 1, "c64", 1 << 7), (31, 1 << 20, "c64", 1 << 30), (32, 1 << 20, "c64", 0),
    (30, 1 << 20, "c128", 1 << 30)])
def test_group_sums_are_counted(n, shots, precision, groups):
    r = _request(n, shots, precision)
    assert r.state_bytes() - r.least_bytes() == groups
    assert r.least_bytes() >= (16 if precision == "c128" else 8) << n


def test_a_request_that_fits_without_them_is_admitted_alone():
    r = _request(20, 4096)
    server = Server.__new__(Server)
    server.budget = r.least_bytes() + 100
    assert r.state_bytes() > server.budget
    assert server._charge(r) == server.budget
    server.budget = r.state_bytes() + 1
    assert server._charge(r) == r.state_bytes()
