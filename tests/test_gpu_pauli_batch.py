"""Batches of Pauli strings: every kernel and pass count of the expectation path (needs a GPU).

Reference: the same sums in numpy on the downloaded amplitudes (FP64).  Both sides add 2^n products
of magnitude |a_i a_j| whose total is at most 1 in FP64, in different orders: 1e-13 absolute.
"""
import numpy as np
import pytest

import ruqu_b200 as rq
from ruqu_b200 import workloads

pytestmark = pytest.mark.gpu


def _reference(a, strings):
    i = np.arange(a.size, dtype=np.uint64)
    out = []
    for s in strings:
        x = z = ny = 0
        for q, o in s:
            x ^= (1 << q) if o in (1, 2) else 0
            z ^= (1 << q) if o in (2, 3) else 0
            ny += o == 2
        j = i ^ np.uint64(x)
        p = j & np.uint64(z)
        for sh in (16, 8, 4, 2, 1):
            p ^= p >> np.uint64(sh)
        sign = 1.0 - 2.0 * (p & np.uint64(1)).astype(np.float64)
        out.append(float(np.real(1j ** ny * np.sum(np.conj(a) * sign * a[j]))))
    return np.array(out)


def _strings(n, many):
    s = [[], [(0, 3)], [(n - 1, 3)], [(0, 1)], [(n - 1, 1)], [(0, 2)], [(n - 1, 2)], [(0, 2), (n - 1, 2)],
         [(0, 2), (0, 2)], [(q, 3) for q in range(n)], [(q, 1) for q in range(n)], [(q, 2) for q in range(n)]]
    s += [[(q, 3), ((q + 1) % n, 3)] for q in range(n)] + [[(q, 1)] for q in range(n)]
    s += [[(q, 1), ((q + 2) % n, 1)] for q in range(n)]             # patterns that depend on each other
    s += [[(q % 4, 1), ((q + 5) % n, 3)] for q in range(n)]         # X only inside a contiguous run
    s += workloads.pauli_hamiltonian(n, 200 if many else 30, n)[1]
    if many:
        r = np.random.default_rng(n)
        s += [[(int(q), 3) for q in r.choice(n, 3, replace=False)] for _ in range(380)]
    return s


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("n,many", [(2, False), (9, False), (13, True), (14, True), (15, False), (18, True)])
def test_pauli_batches_match_numpy(prec, n, many):
    st = rq.QuantumState(n, 3, prec)
    st.apply_gates(workloads.random_layer_circuit(n, 4, 11))
    a = st.state_vector()
    strings = _strings(n, many) if n > 2 else [[], [(0, 3)], [(1, 1)], [(0, 2), (1, 2)], [(0, 1), (1, 3)]]
    got = st.expectation_values(strings)
    assert np.max(np.abs(got - _reference(a, strings))) < 1e-13
    again = st.expectation_values(strings)
    assert np.array_equal(got, again)
    for k in (0, len(strings) // 2, len(strings) - 1):
        assert abs(st.expectation_value(strings[k]) - got[k]) < 1e-13
