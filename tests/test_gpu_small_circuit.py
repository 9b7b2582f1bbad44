"""Circuits below the sweeps' 12 qubits run as one kernel (needs a GPU).

The same arithmetic per amplitude as the per-gate kernels (RQ_EXEC_PER_GATE), so the amplitudes
must be equal bit for bit, for every gate kind, list lengths around one launch's 96 and 384 gates and
its 400 and 1600 matrix entries, and 1 to 11 qubits; and within 1e-12 / 1e-5 of the oracle.
"""
import numpy as np
import pytest

import oracle
import ruqu_b200 as rq

pytestmark = pytest.mark.gpu


def _gates(n, count, seed):
    r = np.random.default_rng(seed)
    out = []
    while len(out) < count:
        kind = int(r.integers(0, 20))
        q0, q1 = int(r.integers(n)), int(r.integers(n))
        if kind in (16, 17) or (kind in (12, 13, 14, 15) and q0 == q1):
            continue
        if kind == 19:
            a = r.normal(size=(2, 2)) + 1j * r.normal(size=(2, 2))
            u = np.linalg.qr(a)[0].reshape(-1)
            out.append((19, q0, 0, 0.0, np.stack([u.real, u.imag], 1).reshape(-1).tolist()))
        else:
            out.append((kind, q0, q1, float(r.uniform(-4, 4))))
    return out


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("n,count", [(1, 7), (2, 95), (3, 96), (5, 97), (7, 383), (8, 385), (11, 1000), (10, 0)])
def test_small_circuits_equal_per_gate_kernels(prec, n, count):
    gates = _gates(n, count, 7 * n + count)
    a, b = rq.QuantumState(n, 1, prec), rq.QuantumState(n, 1, prec)
    a.apply_gates(gates)
    b.apply_gates(gates, mode=rq.RQ_EXEC_PER_GATE)
    x, y = a.state_vector(), b.state_vector()
    assert np.array_equal(x, y)
    o = oracle.OracleState(n, oracle.RQ_F64, 1)
    o.apply([g for g in gates if g[0] != 18])
    assert np.max(np.abs(x - o.amplitudes())) < (1e-12 if prec == "f64" else 1e-5 * max(1, count / 100))
