"""Prefix trees at the edges of their kernels (needs a GPU): every level of the tree of states whose
levels all fit one CTA, of one, two and more folds of three levels, with the qubits in order and
permuted, against a host fold of the same probabilities (rounded sums without FMA: equal bits)."""
import numpy as np
import pytest

import ruqu_b200 as rq
from ruqu_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("n", [1, 2, 3, 11, 12, 13, 15, 16, 18])
def test_tree_levels_equal_a_host_fold(prec, n):
    st = rq.QuantumState(n, 1, prec)
    st.apply_gates(workloads.random_layer_circuit(n, 3, n))
    p = st.probabilities()
    for order in (list(range(n)), list(range(n))[::-1], [n // 2] + [q for q in range(n) if q != n // 2]):
        st.tree_build(order)
        i = np.arange(1 << n)
        src = np.zeros(1 << n, dtype=np.int64)
        for b, q in enumerate(order):
            src |= ((i >> b) & 1) << q
        level = p[src]
        assert np.array_equal(st.tree_lookup(n, i[:257]), level[:257])
        for k in range(n - 1, -1, -1):
            level = level[:1 << k] + level[1 << k:]
            j = np.unique(np.linspace(0, (1 << k) - 1, 300).astype(np.int64))
            assert np.array_equal(st.tree_lookup(k, j), level[j]), (order[:3], k)
