"""Circuits that a batch runs on teams of CTAs (k_batch's clusters) give the
same words, bit for bit, as on one CTA.  A batch of a few circuits of 12 qubits
or more runs the longest on teams; in one of more than 16 circuits per SM
none is."""
import numpy as np
import pytest

from q1tsim_gb300 import Circuit, gates as G, workloads
from q1tsim_gb300.batch import Batch

pytestmark = pytest.mark.gpu


def _filler():
    c = Circuit(1, 1)
    c.add_gate(G.H(), [0])
    c.measure_all([0])
    return c


@pytest.mark.parametrize("sizes,nmeasure,shots", [([12], 1, 700), ([12, 13], 3, 33), ([14, 12, 15], 2, 1025),
                                                  ([16], 4, 3000), ([17, 9, 13], 0, 64), ([13, 8, 10, 16], 1, 1)])
def test_words_do_not_depend_on_the_team(sizes, nmeasure, shots):
    circuits = []
    for i, n in enumerate(sizes):
        if nmeasure:
            circuits.append(workloads.mid_measure_circuit(n, 5, 17 * n + nmeasure, nmeasure))
        else:
            circuits.append(workloads.brick(n, 4, 5 + n))
    few, many = Batch(4), Batch(4)
    for i, c in enumerate(circuits):
        few.add(c, shots, 100 + i)
        many.add(c, shots, 100 + i)
    filler = _filler()
    for i in range(2600):
        many.add(filler, 2, i)
    a, b = few.run(), many.run()
    for i in range(len(circuits)):
        np.testing.assert_array_equal(a[i], b[i])
    again = few.run()
    for i in range(len(circuits)):
        np.testing.assert_array_equal(a[i], again[i])
