"""Bounded waits that run out while RQ_EXEC_AUTO times its candidates (needs a GPU).

The limit of zero polls expires every wait at once, as in test_gpu_wait_expiry.py.  The tuner then
takes the CUDA-core sweep for that call, tells no other state of it and tunes again at the next call.
"""
import numpy as np
import pytest

import oracle
import ruqu_b200 as rq
from ruqu_b200 import _capi, workloads

pytestmark = pytest.mark.gpu

DEFAULT = 0xFFFFFFFF


def test_a_wait_that_expires_in_a_candidate_stays_there():
    n = 14
    # a structure that no other test has tuned: the choice is kept per process
    gates = workloads.random_layer_circuit(n, 4, 21) + [(12, 3, 11, 0.0), (12, 9, 0, 0.0), (12, 1, 12, 0.0)]
    other = rq.QuantumState(n, 0, "f32")
    rq.Plan(other, workloads.random_layer_circuit(n, 4, 7), rq.RQ_EXEC_SWEEP_TC16).execute(other)
    st = rq.QuantumState(n, 0, "f32")
    assert _capi.lib.rq_debug_set_wait_limit(0) == 0
    try:
        st.apply_gates(gates)                     # tunes on first sight of the structure
        st.synchronize()
    finally:
        assert _capi.lib.rq_debug_set_wait_limit(DEFAULT) == 0
    other.synchronize()                           # ran a tensor-core sweep of its own, which did not expire
    ref = oracle.OracleState(n, oracle.RQ_F64, 0)
    ref.apply(gates)
    assert float(np.max(np.abs(st.state_vector() - ref.amplitudes()))) < 1e-5
    st.reset()
    st.apply_gates(gates)
    assert float(np.max(np.abs(st.state_vector() - ref.amplitudes()))) < 1e-5
