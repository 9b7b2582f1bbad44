"""Batched VQE engine vs the oracle (needs a GPU).

Energies: the oracle's expectation_hamiltonian (state.rs:403-408) on the same
Ry + CZ-ladder ansatz run gate by gate; tolerance 1e-10 absolute for f64
states, 1e-5 relative (to sum |coeff|) for f32 states.  Gradients: the
parameter-shift difference of oracle energies (vqe.rs:186-198).
"""
import math

import numpy as np
import pytest

import oracle
from ruqu_b200 import workloads
from ruqu_b200.batch import VqeBatch

pytestmark = pytest.mark.gpu


def _energy(n, depth, params, coeffs, strings):
    return oracle.circuit_energy(n, workloads.hea_ry_cz(n, depth, params), coeffs, strings)


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_vqe_batch_energies_and_gradients(prec):
    n, depth = (8, 3) if prec == "f64" else (9, 2)
    coeffs, strings = workloads.pauli_hamiltonian(n, 24, 5)
    strings = strings + [[(0, 2), (0, 2)], [(1, 1), (1, 1), (3, 3)], []]   # repeated qubits, identity
    coeffs = np.concatenate([coeffs, [0.3, -0.7, 1.1]])
    P = n * depth
    r = np.random.default_rng(1)
    params = r.uniform(-math.pi, math.pi, size=(3, P))
    vb = VqeBatch(n, depth, coeffs, strings, prec)
    e, g = vb.run(params, gradient=True)
    scale = float(np.sum(np.abs(coeffs)))
    tol = 1e-10 if prec == "f64" else 1e-5 * scale
    for s in range(3):
        assert abs(e[s] - _energy(n, depth, params[s], coeffs, strings)) < tol
        for k in range(0, P, max(1, P // 6)):
            pp, pm = params[s].copy(), params[s].copy()
            pp[k] += math.pi / 2
            pm[k] -= math.pi / 2
            want = (_energy(n, depth, pp, coeffs, strings) - _energy(n, depth, pm, coeffs, strings)) / 2
            assert abs(g[s, k] - want) < tol, (s, k, g[s, k], want)
    e2 = vb.run(params)
    assert np.max(np.abs(e2 - e)) == 0.0


def test_vqe_batch_config_shape_16q():
    """16 qubits, 200 random Pauli strings (seed 3), depth 8 Ry + CZ ladder, f32 states."""
    n, depth = 16, 8
    coeffs, strings = workloads.pauli_hamiltonian(n, 200, 3)
    params = workloads.vqe_parameter_sets(2, n * depth, 4)
    vb = VqeBatch(n, depth, coeffs, strings, "f32")
    e, g = vb.run(params, gradient=True)
    scale = float(np.sum(np.abs(coeffs)))
    for s in range(2):
        want = _energy(n, depth, params[s], coeffs, strings)
        assert abs(e[s] - want) < 1e-5 * scale, (e[s], want)
    k = 37
    pp, pm = params[0].copy(), params[0].copy()
    pp[k] += math.pi / 2
    pm[k] -= math.pi / 2
    want = (_energy(n, depth, pp, coeffs, strings) - _energy(n, depth, pm, coeffs, strings)) / 2
    assert abs(g[0, k] - want) < 1e-5 * scale


def test_vqe_batch_f64_two_energy_tiles():
    """f64 states above 12 qubits: the energy kernel pairs 2^12-amplitude tiles."""
    n, depth = 14, 2
    coeffs, strings = workloads.pauli_hamiltonian(n, 12, 8)
    params = workloads.vqe_parameter_sets(2, n * depth, 9)
    vb = VqeBatch(n, depth, coeffs, strings, "f64")
    e = vb.run(params)
    for s in range(2):
        want = _energy(n, depth, params[s], coeffs, strings)
        assert abs(e[s] - want) < 1e-10, (e[s], want)


@pytest.mark.parametrize("gradient", [False, "shift", "adjoint"])
def test_vqe_runs_replay_one_graph_with_identical_results(gradient):
    """rq_vqe_batch_run as a CUDA graph: results equal a batch
    that never uses graphs, for new parameters every run; the first run of a shape is plain,
    later ones launch the captured graph."""
    n, depth = 12, 3
    coeffs, strings = workloads.pauli_hamiltonian(n, 40, 7)
    P = n * depth
    r = np.random.default_rng(8)
    a = VqeBatch(n, depth, coeffs, strings, "f32")
    b = VqeBatch(n, depth, coeffs, strings, "f32")
    b.set_graphs(False)
    flags = []
    for it in range(3):
        params = r.uniform(-math.pi, math.pi, size=(5, P))
        x = a.run(params, gradient=gradient)
        flags.append(a.last_graph()["replayed"])
        y = b.run(params, gradient=gradient)
        if gradient:
            assert np.array_equal(x[0], y[0]) and np.array_equal(x[1], y[1])
        else:
            assert np.array_equal(x, y)
    assert flags == [False, True, True]


@pytest.mark.parametrize("prec,n", [("f32", 7), ("f32", 10), ("f32", 11), ("f32", 14), ("f32", 15), ("f64", 6),
                                    ("f64", 12), ("f64", 13), ("f64", 15)])
def test_vqe_batch_tile_edges(prec, n):
    """States of one partly filled block, of one tile, of a tile without and with one register
    bit, and of several tiles; strings whose X pattern is empty, only qubit 0, only inside a warp,
    on a register bit, and across tiles, each with and without Z on qubit 0, and strings with one
    and two Y factors.  Tolerances as above."""
    top = n - 1
    strings = [[], [(0, 3)], [(0, 1)], [(0, 1), (2, 3)], [(1, 1)], [(1, 1), (0, 3)], [(0, 1), (3, 1)],
               [(0, 2), (3, 2)], [(0, 2), (4, 1)], [(top, 1)], [(top, 1), (0, 1)], [(top, 2), (0, 2), (1, 3)],
               [(top - 1, 1), (2, 3)], [(top - 1, 2), (top, 2)], [(top - 2, 1), (top, 3), (0, 1)],
               [(q, 3) for q in range(n)], [(q, 1) for q in range(n)], [(0, 2), (1, 2), (top, 2)]]
    coeffs = np.linspace(-1.0, 1.3, len(strings))
    depth = 2
    params = np.random.default_rng(n).uniform(-math.pi, math.pi, size=(3, n * depth))
    vb = VqeBatch(n, depth, coeffs, strings, prec)
    e, g = vb.run(params, gradient="adjoint")
    tol = 1e-10 if prec == "f64" else 1e-5 * float(np.sum(np.abs(coeffs)))
    for s in range(3):
        assert abs(e[s] - _energy(n, depth, params[s], coeffs, strings)) < tol
    for k in (0, 1, n - 1, n, 2 * n - 1):
        pp, pm = params[0].copy(), params[0].copy()
        pp[k] += math.pi / 2
        pm[k] -= math.pi / 2
        want = (_energy(n, depth, pp, coeffs, strings) - _energy(n, depth, pm, coeffs, strings)) / 2
        assert abs(g[0, k] - want) < tol, (k, g[0, k], want)


def test_vqe_batch_non_finite_inputs_stay_non_finite():
    """NaN or infinite coefficients and angles give NaN energies, also through a string with one
    Y factor, which adds nothing otherwise."""
    p = np.full((2, 14), 0.3)
    e, g = VqeBatch(7, 2, [1.0, np.inf], [[(0, 3)], [(1, 2)]], "f32").run(p, gradient="adjoint")
    assert np.all(np.isnan(e)) and np.all(np.isnan(g))
    p[1, 3] = np.nan
    e = VqeBatch(7, 2, [1.0], [[(1, 2)]], "f32").run(p)
    assert e[0] == 0.0 and np.isnan(e[1])


@pytest.mark.parametrize("prec,n,depth", [("f32", 14, 42), ("f32", 14, 102), ("f64", 13, 42), ("f64", 13, 82)])
def test_many_layers_with_tables_in_and_out_of_shared_memory(prec, n, depth):
    """Two layers of angle 0 are two CZ ladders, an exact identity, so a deep batch equals the two-layer
    one up to the order of the sums (f64 1e-12; f32: 32 terms a thread of at most sum |c| in all); the
    depths lie on both sides of what fits beside a tile."""
    coeffs, strings = workloads.pauli_hamiltonian(n, 20, 7)
    params = np.zeros((2, n * depth))
    params[:, :2 * n] = np.random.default_rng(n).uniform(-math.pi, math.pi, size=(2, 2 * n))
    want, wgrad = VqeBatch(n, 2, coeffs, strings, prec).run(params[:, :2 * n], gradient="adjoint")
    vb = VqeBatch(n, depth, coeffs, strings, prec)
    tol = (1e-12 if prec == "f64" else 2 * 32 * 2.0 ** -24) * float(np.sum(np.abs(coeffs)))
    assert np.max(np.abs(vb.run(params) - want)) <= tol
    if n * depth <= 600:   # the adjoint kernel refuses the deeper ones
        _, grad = vb.run(params, gradient="adjoint")
        assert np.max(np.abs(grad[:, :2 * n] - wgrad)) <= tol


@pytest.mark.parametrize("prec,n,depth,sets", [("f32", 8, 3, 3), ("f32", 14, 2, 5), ("f32", 16, 8, 3), ("f32", 20, 2, 8),
                                               ("f32", 24, 2, 1), ("f64", 12, 3, 2), ("f64", 13, 3, 4), ("f64", 16, 3, 40)])
def test_shift_rule_equals_explicitly_shifted_runs(prec, n, depth, sets):
    """A shifted circuit begins with the sweep of its parameter, on the unshifted circuit's state: to the bit
    what running it from the start gives.  One sweep and several; one wave and several; one group of sets
    and several (20 qubits); a state too large to keep between the sweeps (24 qubits)."""
    coeffs, strings = workloads.pauli_hamiltonian(n, 12, 3)
    params = np.random.default_rng(n).uniform(-math.pi, math.pi, size=(sets, n * depth))
    vb = VqeBatch(n, depth, coeffs, strings, prec)
    e, g = vb.run(params, gradient="shift")
    assert np.array_equal(e, vb.run(params))
    for k in sorted({0, 1, n - 1, n, n * depth // 2, n * depth - n, n * depth - 1}):
        up, dn = params.copy(), params.copy()
        up[:, k] += math.pi / 2
        dn[:, k] -= math.pi / 2
        assert np.array_equal(g[:, k], (vb.run(up) - vb.run(dn)) / 2.0), k
