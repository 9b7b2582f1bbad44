"""Ansätze deeper than one sweep's tables hold (needs a GPU).

The state of 14 qubits f32 (13 f64) is one tile, so its sweep is cut where the phase descriptors fill
the shared memory.  Reference: the oracle's FP64 state and its exact energies.  An f32 rotation rounds each
amplitude to 2^-24 relative twice; over D = 14 * layers rotations the errors add like sqrt(D), which the
energy carries twice, scaled by the sum of |coefficients|: 2 * 2 * 6e-8 * sqrt(8400) = 2.2e-5 of it.
The f64 bound is the same with 2^-53, rounded up to 1e-12.
"""
import numpy as np
import pytest

import oracle
from ruqu_b200 import workloads
from ruqu_b200.batch import VqeBatch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,n,depth", [("f32", 14, 570), ("f32", 14, 600), ("f64", 13, 450)])
def test_energies_past_one_sweep(prec, n, depth):
    coeffs, strings = workloads.pauli_hamiltonian(n, 24, 3)
    params = workloads.vqe_parameter_sets(2, n * depth, 11)
    got = VqeBatch(n, depth, coeffs, strings, prec).run(params)
    tol = {"f32": 2.2e-5, "f64": 1e-12}[prec] * np.sum(np.abs(coeffs))
    for s in range(2):
        want = oracle.circuit_energy(n, workloads.hea_ry_cz(n, depth, params[s]), coeffs, strings)
        assert abs(got[s] - want) < tol
