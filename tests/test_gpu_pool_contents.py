"""What the pool of destroyed states' resources holds (needs a GPU; rq_debug_state_pool).

An ordinary state leaves one set; one whose device pointer was handed out leaves none, since another
stream may still use its memory; the sets stay within 16, 64 MiB each and 256 MiB in all.
"""
import contextlib
import ctypes as C
import gc

import numpy as np
import pytest

import ruqu_b200 as rq
from ruqu_b200 import _capi

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _pool():
    sets, size = C.c_uint64(), C.c_uint64()
    assert _capi.lib.rq_debug_state_pool(C.byref(sets), C.byref(size)) == _capi.RQ_OK
    return sets.value, size.value


@contextlib.contextmanager
def little_memory(leave=64 * MIB):
    """The rest of the device's memory taken, but for less than `leave` bytes."""
    from cuda.bindings import runtime as rt
    taken = []
    try:
        for chunk in (1 << 30, leave // 2):
            while rt.cudaMemGetInfo()[1] >= chunk + leave // 2:
                err, ptr = rt.cudaMalloc(chunk)
                if int(err) != 0:
                    break
                taken.append(ptr)
        yield rt.cudaMemGetInfo()[1]
    finally:
        for ptr in taken:
            rt.cudaFree(ptr)


def _empty():
    with little_memory():
        with pytest.raises(rq.MemoryAllocationFailed):
            rq.QuantumState(26, 1, "f64")                              # 1 GiB
    assert _pool() == (0, 0)


def test_only_memory_that_was_not_handed_out_is_kept():
    _empty()
    st = rq.QuantumState(10, 1, "f64")
    before = _pool()[0]
    st.device_pointer()
    del st
    gc.collect()
    assert _pool()[0] == before
    st = rq.QuantumState(10, 1, "f64")
    before = _pool()[0]
    del st
    gc.collect()
    assert _pool()[0] == before + 1


def test_limits():
    states = [rq.QuantumState(20, 1, "f64") for _ in range(18)]        # 16 MiB each
    del states
    gc.collect()
    sets, size = _pool()
    assert 0 < sets <= 16 and size <= 256 * MIB
    states = [rq.QuantumState(4, 1, "f64") for _ in range(40)]
    del states
    gc.collect()
    sets, size = _pool()
    assert sets == 16 and size <= 256 * MIB
    before = _pool()
    big = rq.QuantumState(23, 1, "f64")                                # 128 MiB: its amplitudes are not kept
    big.norm_sq()
    del big
    gc.collect()
    assert _pool()[1] <= before[1] + MIB


def test_pinned_staging_counts():
    """2^20 + 1 Pauli strings need 8 MiB of pinned results."""
    _empty()
    st = rq.QuantumState(1, 1, "f64")
    count = (1 << 20) + 1
    off = np.zeros(count + 1, dtype=np.uint32)
    out = np.zeros(count)
    ops = (_capi.RqPauliOp * 1)()
    rc = _capi.lib.rq_state_expectation_batch(st.handle, ops, off.ctypes.data_as(C.POINTER(C.c_uint32)), count,
                                              out.ctypes.data_as(C.POINTER(C.c_double)))
    assert rc == 0 and np.all(out == 1.0)
    del st
    gc.collect()
    assert _pool()[1] >= 8 * MIB


def test_a_failed_allocation_empties_the_pool():
    _empty()
    held = [rq.QuantumState(14, 1, "f64") for _ in range(4)]
    del held
    gc.collect()
    assert _pool()[0] >= 4
    with little_memory() as free:
        assert free < 128 * MIB
        with pytest.raises(rq.MemoryAllocationFailed):
            rq.QuantumState(26, 1, "f64")                              # 1 GiB
        assert _pool()[0] == 0
    assert rq.QuantumState(26, 1, "f64").norm_sq() == 1.0


def test_calls_that_need_memory_get_what_the_pool_holds():
    """Scratch above 64 MiB (stream-ordered), the tuner's scratch state and a plan's tables: 128 MiB are
    free only with the pool's 192 MiB."""
    from ruqu_b200 import workloads
    _empty()
    n = 24
    st = rq.QuantumState(n, 1, "f64")
    f32 = rq.QuantumState(n, 1, "f32")
    pooled = [rq.QuantumState(21, 1, "f64") for _ in range(6)]
    with little_memory() as free:
        assert free < 128 * MIB
        del pooled
        gc.collect()
        assert _pool()[0] >= 6
        assert st.probabilities()[0] == 1.0                # 128 MiB
        assert _pool()[0] == 0
    pooled = [rq.QuantumState(21, 1, "f64") for _ in range(6)]
    with little_memory() as free:
        assert free < 128 * MIB
        del pooled
        gc.collect()
        assert _pool()[0] >= 6
        plan = rq.Plan(f32, workloads.random_layer_circuit(n, 13, 5))
        assert plan.stats()["dense_ops"] > 0               # tuned: the tensor-core sweep
        assert _pool()[0] == 0


def test_a_choice_made_without_memory_is_made_again():
    """No room for the tuner's scratch state: the CUDA-core sweep, for that call only."""
    from ruqu_b200 import workloads
    n = 24
    f32 = rq.QuantumState(n, 1, "f32")
    gates = workloads.random_layer_circuit(n, 14, 5)
    with little_memory() as free:
        assert free < 128 * MIB
        with pytest.raises(rq.MemoryAllocationFailed):     # and none in the pool
            rq.QuantumState(26, 1, "f64")
        assert rq.Plan(f32, gates).stats()["dense_ops"] == 0
    assert rq.Plan(f32, gates).stats()["dense_ops"] > 0


def test_calls_without_memory_do_not_plan_every_candidate_again():
    """The second call of a structure that found no memory takes the CUDA-core sweep without planning the
    candidates (0.1 s and more for 24 qubits, 15 layers); it is a small part of the first."""
    import time

    from ruqu_b200 import workloads
    n = 24
    f32 = rq.QuantumState(n, 1, "f32")
    gates = workloads.random_layer_circuit(n, 15, 5)
    times = []
    with little_memory() as free:
        assert free < 128 * MIB
        for _ in range(3):
            t = time.perf_counter()
            assert rq.Plan(f32, gates).stats()["dense_ops"] == 0
            times.append(time.perf_counter() - t)
    assert max(times[1:]) < 0.5 * times[0], times
    assert rq.Plan(f32, gates).stats()["dense_ops"] > 0
