"""Parameter-shift runs of several parameter sets (needs a GPU): each set's energy and gradient are what
the set gives alone, to the bit, and circuits that begin nowhere but at the start share their launches."""
import numpy as np
import pytest

from ruqu_b200 import workloads
from ruqu_b200.batch import VqeBatch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,n,depth,sets", [("f32", 7, 2, 50), ("f64", 6, 3, 9), ("f32", 14, 2, 5), ("f64", 13, 2, 4),
                                               ("f32", 15, 3, 5), ("f64", 14, 3, 3)])
def test_sets_do_not_depend_on_each_other(prec, n, depth, sets):
    coeffs, strings = workloads.pauli_hamiltonian(n, 12, 3)
    params = workloads.vqe_parameter_sets(sets, n * depth, 4)
    vb = VqeBatch(n, depth, coeffs, strings, prec)
    e, g = vb.run(params, gradient="shift")
    for s in range(sets):
        e1, g1 = vb.run(params[s:s + 1], gradient="shift")
        assert e1[0] == e[s] and np.array_equal(g1[0], g[s])


@pytest.mark.parametrize("prec,n", [("f32", 7), ("f32", 12), ("f64", 12)])
def test_launches_do_not_grow_with_the_sets(prec, n):
    """A state of one tile has one sweep, so there is no shared beginning; 40 sets fit one wave."""
    coeffs, strings = workloads.pauli_hamiltonian(n, 12, 3)
    nodes = []
    for sets in (2, 40):
        vb = VqeBatch(n, 2, coeffs, strings, prec)
        params = workloads.vqe_parameter_sets(sets, 2 * n, 4)
        for _ in range(3):
            vb.run(params, gradient="shift")
        assert vb.last_graph()["replayed"]
        nodes.append(vb.last_graph()["kernels"])
    assert nodes[0] == nodes[1]
