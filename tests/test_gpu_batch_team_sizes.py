"""Teams of 2, 4 and 8 CTAs (k_batch's clusters) against lone CTAs, word for
word: circuits of the fewest qubits a team takes and of more tiles than its
warps, with up to four measurements (16 columns), alone and in batches of more
circuits than teams with small ones that no team takes."""
import numpy as np
import pytest

from q1tsim_gb300 import InvalidArgument, workloads
from q1tsim_gb300.batch import Batch

pytestmark = pytest.mark.gpu


def _words(circuits, shots, size):
    b = Batch(4)
    b.set_team_size(size)
    for i, c in enumerate(circuits):
        b.add(c, shots, 50 + i)
    first, again = b.run(), b.run()
    for x, y in zip(first, again):
        np.testing.assert_array_equal(x, y)
    return first, b.teams()


def _circuit(n, nmeasure, depth=5):
    return workloads.mid_measure_circuit(n, depth, 31 * n + nmeasure, nmeasure) if nmeasure else workloads.brick(n, depth, n)


@pytest.mark.parametrize("size", [2, 4, 8])
@pytest.mark.parametrize("nmeasure", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("n", [12, 13, 17])
def test_one_circuit_on_a_team(n, nmeasure, size):
    circuits, shots = [_circuit(n, nmeasure)], 700
    lone, none = _words(circuits, shots, 1)
    team, plan = _words(circuits, shots, size)
    assert none == (0, 1, 0) and plan[:2] == (1, size) and plan[2] > 0
    np.testing.assert_array_equal(lone[0], team[0])


@pytest.mark.parametrize("size", [2, 4, 8])
def test_more_circuits_than_teams_and_lone_ones(size):
    # 170 circuits for teams (at most 76 teams of two), 60 that only lone CTAs take
    # (short: those ahead of a large one in the queue would end the teams' part)
    circuits = [_circuit(12 + i % 2, i % 5, 6) for i in range(170)] + [_circuit(6 + i % 5, 0, 2) for i in range(60)]
    lone, none = _words(circuits, 33, 1)
    team, plan = _words(circuits, 33, size)
    assert none == (0, 1, 0) and plan[1] == size and plan[2] < plan[0] <= 170
    for x, y in zip(lone, team):
        np.testing.assert_array_equal(x, y)


def test_the_estimate_puts_large_circuits_on_teams():
    lone, _ = _words([_circuit(17, 2), _circuit(9, 1)], 64, 1)
    team, plan = _words([_circuit(17, 2), _circuit(9, 1)], 64, 0)
    assert plan[0] == 1 and plan[1] > 1
    for x, y in zip(lone, team):
        np.testing.assert_array_equal(x, y)


def test_sizes_that_are_refused():
    b = Batch(4)
    for size in (-1, 3, 6, 16):
        with pytest.raises(InvalidArgument):
            b.set_team_size(size)
    b.add(_circuit(8, 0), 4, 1)
    b.run()
    with pytest.raises(InvalidArgument):
        b.set_team_size(2)
