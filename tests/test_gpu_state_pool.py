"""Resources of destroyed states are reused by later ones (needs a GPU).

A reused set of buffers must look freshly made: |0...0>, its own seed and draws, no
sampling tree, correct results after a state of another size or precision used the
buffers.  Memory whose device pointer was handed out is never reused.
"""
import gc
import threading

import numpy as np
import pytest

import oracle
import ruqu_b200 as rq
from ruqu_b200 import workloads
from ruqu_b200._capi import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [("f64", 1e-12), ("f32", 1e-5)])
def test_a_reused_state_starts_fresh(prec, tol):
    for n in (3, 12, 5, 13, 3, 16, 12):
        gates = workloads.random_layer_circuit(n, 3, n)
        st = rq.QuantumState(n, n, prec)
        a = st.state_vector()
        assert a[0] == 1 and np.count_nonzero(a) == 1
        with pytest.raises(rq.InvalidArgument):
            st.tree_lookup(0, [0])           # a tree of the state before would answer
        st.apply_gates(gates)
        o = oracle.OracleState(n, oracle.RQ_F64, n)
        o.apply(gates)
        assert np.max(np.abs(st.state_vector() - o.amplitudes())) < tol
        p = st.probabilities()
        assert np.max(np.abs(p - np.abs(o.amplitudes()) ** 2)) < tol
        assert st.sample(300, 9).shape == (300,)
        assert st.measure(0).result == bool(lib.rq_uniform(n, 0, 0) >= 1 - st_prob1(o))
        del st
        gc.collect()


def st_prob1(o):
    return float(np.sum(np.abs(o.amplitudes()[1::2]) ** 2))


def test_exported_memory_is_not_reused():
    st = rq.QuantumState(10, 1, "f64")
    ptr, _ = st.device_pointer()
    others = [rq.QuantumState(10, 1, "f64") for _ in range(3)]
    del st
    others += [rq.QuantumState(10, 1, "f64") for _ in range(20)]
    # the freed block may come back from the driver, but not through the pool: a pooled set
    # would be handed to the very next state together with its stream
    assert all(o.norm_sq() == 1.0 for o in others)
    assert ptr


def test_states_from_many_threads():
    want = {}
    for n in (4, 9, 13):
        o = oracle.OracleState(n, oracle.RQ_F64, 0)
        o.apply(workloads.random_layer_circuit(n, 2, 3))
        want[n] = o.amplitudes()
    bad = []

    def work(k):
        for r in range(30):
            n = (4, 9, 13)[(k + r) % 3]
            st = rq.QuantumState(n, k, "f64")
            st.apply_gates(workloads.random_layer_circuit(n, 2, 3))
            if np.max(np.abs(st.state_vector() - want[n])) > 1e-12:
                bad.append((k, r, n))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
