"""The work that users of ruqu_b200 have it do, as cases that can be timed and compared.

Nine kinds of call, each through the entry points a program uses:

* ``vqe_energy``   -- one ``evaluate_energy`` of a small VQE problem (the reference's own use:
                      a fresh state per evaluation, complex f64): the smallest calls, where
                      launches, allocations and synchronisations count;
* ``maxcut``       -- one ``qaoa_maxcut``: the QAOA circuit of a graph, all probabilities and
                      the expected cut on the host (complex f64);
* ``circuit``      -- a gate list with new angles applied to a state, every <Z_i> read back and
                      the amplitudes left on the device: the random-layer circuits of bench.py,
                      complex f64 and f32, up to its 30 qubits;
* ``observables``  -- many Pauli strings on one state (random strings, or the ZZ couplings and
                      X fields of a transverse-field Ising model);
* ``shots``        -- shot sampling of every qubit of a state;
* ``qaoa_batch``   -- energies and best sampled cuts of many graphs (QaoaBatch.run);
* ``qaoa_grad``    -- energies and exact gradients of many graphs (QaoaBatch.gradient);
* ``vqe_batch``    -- many parameter sets of one ansatz: energies with the parameter-shift
                      gradients of the reference, or with the adjoint gradients (VqeBatch.run);
* ``mlp``          -- training steps of the warm-start network (Mlp.train).

What a complex-f32 state gives is handed on in single precision, as a program that chose f32
states holds it; complex-f64 results stay in double precision, and so do the expectations of a
given state, which are accumulated in FP64 whatever its type.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from ruqu_b200 import workloads
from ruqu_b200.rng import Stream


def listed():
    return [
        # a few-qubit VQE energy, as run_vqe asks for by the thousand
        {"name": "vqe_energy_8q", "kind": "vqe_energy", "n": 8, "depth": 3, "terms": 32},
        # an ordinary MaxCut evaluation of one graph, with its probabilities
        {"name": "maxcut_16q", "kind": "maxcut", "n": 16, "p": 4},
        # the mid-size simulation in the default precision
        {"name": "circuit_f64_22q", "kind": "circuit", "n": 22, "layers": 20, "precision": "f64"},
        # the headline circuit: 30 qubits, 20 layers, complex f32 (8 GiB of amplitudes)
        {"name": "circuit_f32_30q", "kind": "circuit", "n": 30, "layers": 20, "precision": "f32"},
        # a molecular-style Hamiltonian (random strings) measured on one state
        {"name": "observables_f32_24q", "kind": "observables", "n": 24, "strings": 64, "family": "pauli",
         "precision": "f32"},
        # the read-out of a run_shots call
        {"name": "shots_f64_23q", "kind": "shots", "n": 23, "shots": 8192, "precision": "f64"},
        # many small to mid-size graphs with shots: the batched MaxCut leg of bench.py, scaled
        {"name": "qaoa_batch_12_22q", "kind": "qaoa_batch", "graphs": 192, "n_min": 12, "n_max": 22, "p": 4,
         "shots": 1024, "precision": "f32"},
        # one optimizer step's gradients over a set of graphs
        {"name": "qaoa_grad_12_20q", "kind": "qaoa_grad", "graphs": 256, "n_min": 12, "n_max": 20, "p": 4,
         "precision": "f32"},
        # the reference's parameter-shift rule (257 circuits per parameter set)
        {"name": "vqe_shift_16q", "kind": "vqe_batch", "n": 16, "depth": 8, "terms": 200, "sets": 8,
         "gradient": "shift", "precision": "f32"},
        # the same problem's exact gradients over many parameter sets
        {"name": "vqe_adjoint_16q", "kind": "vqe_batch", "n": 16, "depth": 8, "terms": 200, "sets": 512,
         "gradient": "adjoint", "precision": "f32"},
        # a depth and size that fit no tile, in double precision, energies only (a parameter scan)
        {"name": "vqe_scan_f64_13q", "kind": "vqe_batch", "n": 13, "depth": 5, "terms": 60, "sets": 300,
         "gradient": "none", "precision": "f64"},
        # training steps of the warm-start network (its default widths, minibatch 256)
        {"name": "mlp_train_64", "kind": "mlp", "rows": 4000, "batch": 256, "steps": 64, "hidden": 256},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["vqe_energy", "maxcut", "circuit", "circuit", "observables", "shots", "qaoa_batch",
                       "qaoa_grad", "vqe_batch", "mlp"])
    if kind == "vqe_energy":
        return {"kind": kind, "n": rng.randint(2, 13), "depth": rng.randint(1, 4), "terms": _log_int(rng, 4, 128)}
    if kind == "maxcut":
        return {"kind": kind, "n": rng.randint(4, 20), "p": rng.randint(1, 6)}
    if kind == "circuit":
        precision = rng.choice(["f64", "f32"])
        return {"kind": kind, "n": rng.randint(9, 24 if precision == "f64" else 27), "layers": rng.randint(3, 24),
                "precision": precision}
    if kind == "observables":
        return {"kind": kind, "n": rng.randint(12, 25), "strings": _log_int(rng, 4, 100),
                "family": rng.choice(["pauli", "ising"]), "precision": rng.choice(["f32", "f64"])}
    if kind == "shots":
        return {"kind": kind, "n": rng.randint(9, 25), "shots": _log_int(rng, 100, 60000),
                "precision": rng.choice(["f32", "f64"])}
    if kind == "qaoa_batch" or kind == "qaoa_grad":
        lo = rng.choice([8, 10, 12, 14, 16])
        c = {"kind": kind, "graphs": _log_int(rng, 6, 200), "n_min": lo, "n_max": rng.choice([lo, 18, 20]),
             "p": rng.randint(1, 6), "precision": rng.choice(["f32", "f32", "f64"])}
        if c["n_max"] == 20:
            c["graphs"] = min(c["graphs"], 64)
        if kind == "qaoa_batch":
            c["shots"] = rng.choice([0, 256, 1000, 1024])
        return c
    if kind == "vqe_batch":
        gradient = rng.choice(["shift", "adjoint", "none"])
        return {"kind": kind, "n": rng.randint(8, 16), "depth": rng.randint(2, 8), "terms": _log_int(rng, 10, 200),
                "sets": _log_int(rng, 1, 4 if gradient == "shift" else 300), "gradient": gradient,
                "precision": rng.choice(["f32", "f32", "f64"])}
    return {"kind": kind, "rows": rng.randint(300, 8000), "batch": rng.choice([64, 200, 256, 512]),
            "steps": _log_int(rng, 4, 100), "hidden": rng.choice([64, 128, 256])}


# ---- inputs ------------------------------------------------------------------------------

def _graph(n, st):
    """A random 3-regular graph for an even n, a random graph of as many edges otherwise."""
    if n % 2 == 0:
        return workloads.random_3regular_graph(n, st)
    edges = set()
    while len(edges) < min((3 * n) // 2, n * (n - 1) // 2):
        a, b = st.randint(n), st.randint(n)
        if a != b:
            edges.add((min(a, b), max(a, b)))
    return sorted(edges)


def _sizes(case):
    """Graph sizes of a batch: the even sizes of its range in turn (bench.py's 12, 14, .. 24)."""
    vals = list(range(case["n_min"], case["n_max"] + 1, 2))
    return [vals[k % len(vals)] for k in range(case["graphs"])]


def _qaoa_inputs(case, seed):
    st, ang = Stream(seed, 2), Stream(seed, 3)
    graphs = [(n, _graph(n, st)) for n in _sizes(case)]
    u = ang.take(2 * case["p"] * len(graphs)).reshape(len(graphs), 2, case["p"])
    # angles around the annealing-style ramp that the optimizers start from
    ramp = (np.arange(1, case["p"] + 1) - 0.5) / case["p"]
    return graphs, -0.75 * ramp + 0.3 * (u[:, 0] - 0.5), 0.75 * (1 - ramp) + 0.3 * (u[:, 1] - 0.5)


def _strings(case, seed):
    """Pauli strings as [(qubit, op)] lists (ops 1 X, 2 Y, 3 Z)."""
    n, count = case["n"], case["strings"]
    if case["family"] == "pauli":
        return workloads.pauli_hamiltonian(n, count, seed)[1]
    st = Stream(seed, 2)
    pairs = set()
    while len(pairs) < max(1, min(count - n, n * (n - 1) // 2)):
        a, b = st.randint(n), st.randint(n)
        if a != b:
            pairs.add((min(a, b), max(a, b)))
    return ([[(a, 3), (b, 3)] for a, b in sorted(pairs)] + [[(q, 1)] for q in range(n)])[:count]


def _amplitudes(n, precision, seed):
    """A normalised Gaussian vector, the amplitudes a deep random circuit leaves, as complex128
    values that the state's own type holds exactly."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randn(1 << n, 2, generator=g, device="cuda", dtype=torch.float64)
    a /= a.norm()
    if precision == "f32":
        a = a.to(torch.float32).to(torch.float64)
    return torch.view_as_complex(a)


def _mlp_inputs(case, seed):
    """Standardised features and targets, and He-uniform weights, in the network's flat layout."""
    n_in, h, n_out = 325, case["hidden"], 8
    r = np.random.default_rng(seed)
    x = (r.random((case["rows"], n_in)) < 0.12).astype(np.float32)     # adjacency features
    t = r.standard_normal((case["rows"], n_out)).astype(np.float32)
    parts = []
    for rows, cols in ((h, n_in), (h, h), (n_out, h)):
        parts += [(r.random(rows * cols) * 2 - 1) * math.sqrt(6.0 / cols), np.zeros(rows)]
    return x, t, np.concatenate(parts).astype(np.float32)


class _DeviceAmplitudes:
    """The amplitudes of a QuantumState as a device array (its documented zero-copy interop)."""

    def __init__(self, state):
        self.state = state
        ptr, _ = state.device_pointer()
        self.__cuda_array_interface__ = {"shape": (state.num_amplitudes(),), "data": (ptr, False), "version": 3,
                                         "typestr": "<c8" if state.precision == "f32" else "<c16"}


def _held(values, precision):
    return np.asarray(values, dtype=np.float32 if precision == "f32" else np.float64)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "vqe_energy":
        from ruqu_b200.types import Hamiltonian, PauliOp, PauliString
        from ruqu_b200.vqe import VqeConfig, num_parameters
        n = case["n"]
        coeffs, strings = workloads.pauli_hamiltonian(n, case["terms"], seed)
        h = Hamiltonian([(float(c), PauliString([(q, PauliOp(o)) for q, o in s])) for c, s in zip(coeffs, strings)], n)
        params = workloads.vqe_parameter_sets(1, num_parameters(n, case["depth"]), seed)[0].tolist()
        return {"kind": kind, "config": VqeConfig(h, n, case["depth"], 1, 1e-6, 0.1, seed=7), "params": params}
    if kind == "maxcut":
        edges = _graph(case["n"], Stream(seed, 2))
        u = Stream(seed, 3).take(2 * case["p"])
        return {"kind": kind, "n": case["n"], "edges": [v for e in edges for v in e], "p": case["p"],
                "gammas": (-u[:case["p"]]).tolist(), "betas": u[case["p"]:].tolist()}
    if kind == "circuit":
        from ruqu_b200 import QuantumState
        from ruqu_b200.circuit import gates_to_array
        state = QuantumState(case["n"], 1, case["precision"])
        return {"kind": kind, "state": state, "precision": case["precision"],
                "gates": gates_to_array(workloads.random_layer_circuit(case["n"], case["layers"], seed)),
                "zs": [[(q, 3)] for q in range(case["n"])], "amps": torch.as_tensor(_DeviceAmplitudes(state), device="cuda")}
    if kind in ("observables", "shots"):
        from ruqu_b200 import QuantumState
        state = QuantumState.from_amplitudes(_amplitudes(case["n"], case["precision"], seed).cpu().numpy(), case["n"],
                                             case["precision"])
        if kind == "observables":
            return {"kind": kind, "state": state, "strings": _strings(case, seed)}
        return {"kind": kind, "state": state, "shots": case["shots"], "seed": seed}
    if kind in ("qaoa_batch", "qaoa_grad"):
        from ruqu_b200.batch import QaoaBatch
        graphs, g, b = _qaoa_inputs(case, seed)
        return {"kind": kind, "batch": QaoaBatch(graphs, case["p"], case["precision"]), "gammas": g, "betas": b,
                "shots": case.get("shots", 0), "seed": seed, "precision": case["precision"]}
    if kind == "vqe_batch":
        from ruqu_b200.batch import VqeBatch
        n, depth = case["n"], case["depth"]
        coeffs, strings = workloads.pauli_hamiltonian(n, case["terms"], seed)
        return {"kind": kind, "batch": VqeBatch(n, depth, coeffs, strings, case["precision"]),
                "params": workloads.vqe_parameter_sets(case["sets"], n * depth, seed),
                "gradient": None if case["gradient"] == "none" else case["gradient"], "precision": case["precision"]}
    from ruqu_b200.warmstart import Mlp
    x, t, w = _mlp_inputs(case, seed)
    return {"kind": kind, "net": Mlp(h1=case["hidden"], h2=case["hidden"]), "x": x, "t": t, "w": w,
            "batch": case["batch"], "steps": case["steps"]}


def run(state):
    kind = state["kind"]
    if kind == "vqe_energy":
        from ruqu_b200.vqe import evaluate_energy
        return evaluate_energy(state["config"], state["params"])
    if kind == "maxcut":
        from ruqu_b200.qaoa import qaoa_maxcut
        return qaoa_maxcut(state["n"], state["edges"], state["p"], state["gammas"], state["betas"], seed=7)
    if kind == "circuit":
        q = state["state"]
        q.reset()
        q.apply_gates(state["gates"])
        return {"z": _held(q.expectation_values(state["zs"]), state["precision"]), "amplitudes": state["amps"]}
    if kind == "observables":
        return state["state"].expectation_values(state["strings"])
    if kind == "shots":
        return state["state"].sample(state["shots"], state["seed"]).astype(np.int64)
    if kind == "qaoa_batch":
        r = state["batch"].run(state["gammas"], state["betas"], shots=state["shots"], seed=state["seed"])
        out = {"energies": _held(r["energies"], state["precision"])}
        if state["shots"]:
            out["best_bits"] = r["best_bits"].astype(np.int64)
            out["best_cut"] = r["best_cut"].astype(np.int64)
        return out
    if kind == "qaoa_grad":
        e, g = state["batch"].gradient(state["gammas"], state["betas"])
        return {"energies": _held(e, state["precision"]), "gradients": _held(g, state["precision"])}
    if kind == "vqe_batch":
        r = state["batch"].run(state["params"], gradient=state["gradient"])
        if state["gradient"] is None:
            return {"energies": _held(r, state["precision"])}
        return {"energies": _held(r[0], state["precision"]), "gradients": _held(r[1], state["precision"])}
    net = state["net"]
    net.set_params(state["w"])
    loss = net.train(state["x"], state["t"], batch=state["batch"], steps=state["steps"], lr=1e-3)
    return {"loss": loss, "params": net.get_params()}


# ---- the work of one pass -------------------------------------------------------------------

def work(case):
    kind = case["kind"]
    pair = 14.0          # a 2x2 complex matrix on a pair of amplitudes, per amplitude
    rot = 6.0            # a real rotation of a complex pair, per amplitude
    if kind == "vqe_energy":
        n, N = case["n"], 2.0 ** case["n"]
        # Ry and Rz of a qubit as one matrix; every string's pair products
        return {"bytes": 16.0 * n * case["depth"] + 16.0 * case["terms"],
                "flops": N * (case["depth"] * n * pair + 4.0 * case["terms"])}
    if kind == "maxcut":
        N = 2.0 ** case["n"]
        return {"bytes": 8.0 * N, "flops": N * (case["p"] * (case["n"] * rot + 6) + 3)}
    if kind == "circuit":
        N, elem = 2.0 ** case["n"], 8 if case["precision"] == "f32" else 16
        return {"bytes": N * elem, "flops": N * (case["layers"] * case["n"] * pair + 3)}
    if kind == "observables":
        N, elem = 2.0 ** case["n"], 8 if case["precision"] == "f32" else 16
        return {"bytes": N * elem, "flops": 4.0 * N * case["strings"]}
    if kind == "shots":
        N, elem = 2.0 ** case["n"], 8 if case["precision"] == "f32" else 16
        return {"bytes": N * elem + 8.0 * case["shots"], "flops": 4.0 * N}
    if kind in ("qaoa_batch", "qaoa_grad"):
        flops = 0.0
        for n in _sizes(case):
            evolve = case["p"] * (n * rot + 6) + 4
            flops += 2.0 ** n * (evolve if kind == "qaoa_batch" else evolve + case["p"] * (2 * n * rot + 4 * n + 16))
            flops += 2.0 ** n * 4 if case.get("shots") else 0.0
        return {"bytes": 16.0 * case["graphs"] * case["p"], "flops": flops}
    if kind == "vqe_batch":
        n, N, P = case["n"], 2.0 ** case["n"], case["n"] * case["depth"]
        evolve, energy = P * rot, 4.0 * case["terms"]
        per = {"none": evolve + energy, "shift": (1 + 2 * P) * (evolve + energy),
               "adjoint": evolve + energy + 8.0 * case["terms"] + P * (2 * rot + 4)}[case["gradient"]]
        return {"bytes": 8.0 * case["sets"] * (P + 1 + (P if case["gradient"] != "none" else 0)),
                "flops": case["sets"] * N * per}
    h = case["hidden"]
    weights = 325 * h + h * h + h * 8
    return {"bytes": 4.0 * case["rows"] * (325 + 8) + 8.0 * weights,
            "flops": case["steps"] * 6.0 * min(case["batch"], case["rows"]) * weights}


# ---- the same results in 64 bits, from plain torch and numpy ---------------------------------

def _on_pair(psi, q):
    """View of psi (.., 2^n) as (.., high, 2, low) around qubit q."""
    return psi.view(*psi.shape[:-1], -1, 2, 1 << q)


def _apply(psi, q, m):
    v = _on_pair(psi, q)
    a, b = v[..., 0, :].clone(), v[..., 1, :].clone()
    v[..., 0, :] = m[0][0] * a + m[0][1] * b
    v[..., 1, :] = m[1][0] * a + m[1][1] * b


def _cnot(psi, c, t):
    hi, lo = max(c, t), min(c, t)
    v = psi.view(-1, 2, 1 << (hi - lo - 1), 2, 1 << lo)
    a, b = (v[:, 1, :, 0], v[:, 1, :, 1]) if c == hi else (v[:, 0, :, 1], v[:, 1, :, 1])
    x = a.clone()
    a.copy_(b)
    b.copy_(x)


def _parity(i, mask):
    p = i & mask
    for s in (32, 16, 8, 4, 2, 1):
        p = p ^ (p >> s)
    return p & 1


def _string_masks(ops):
    x = z = ny = 0
    for q, o in ops:
        x |= (1 << q) if o in (1, 2) else 0
        z |= (1 << q) if o in (2, 3) else 0
        ny += o == 2
    return x, z, ny


def _times_string(psi, i, ops):
    """P psi for a Pauli string P, psi of shape (.., 2^n) and i = arange(2^n): entry j ^ x of the
    result is i^ny (-1)^(z.j) psi_j."""
    x, z, ny = _string_masks(ops)
    j = i ^ x
    sign = (1 - 2 * _parity(j, z)).to(torch.float64)
    return psi[..., j] * sign * (1, 1j, -1, -1j)[ny % 4]


def _new_state(n):
    psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    psi[0] = 1
    return psi


def _cuts(n, edges):
    i = torch.arange(1 << n, device="cuda")
    c = torch.zeros(1 << n, dtype=torch.float64, device="cuda")
    for a, b in edges:
        c += ((i >> a) ^ (i >> b)) & 1
    return c


def _rx_all(psi, n, beta):
    c, s = math.cos(beta), math.sin(beta)
    for q in range(n):
        _apply(psi, q, ((c, -1j * s), (-1j * s, c)))


def _qaoa_state(n, edges, gammas, betas):
    cut = _cuts(n, edges)
    psi = torch.full((1 << n,), 2.0 ** (-n / 2), dtype=torch.complex128, device="cuda")
    for g, b in zip(gammas, betas):
        psi *= torch.exp(-1j * float(g) * (len(edges) - 2 * cut))
        _rx_all(psi, n, float(b))
    return psi, cut


def _exact_circuit(case, seed):
    n = case["n"]
    psi = _new_state(n)
    k, layer = 0, workloads.random_layer_circuit(n, case["layers"], seed)
    per_qubit = {}
    for kind, q0, q1, angle in layer:
        h = angle / 2
        if kind == 10:                                   # Rz
            per_qubit[q0] = np.diag([np.exp(-1j * h), np.exp(1j * h)])
        elif kind == 8:                                  # Rx
            rx = np.array([[math.cos(h), -1j * math.sin(h)], [-1j * math.sin(h), math.cos(h)]])
            per_qubit[q0] = rx @ per_qubit[q0]
            k += 1
            if k % n == 0:                               # the layer's 2x2 matrices, up to five qubits at a time
                for lo in range(0, n, 5):
                    qs = range(lo, min(lo + 5, n))
                    u = np.eye(1)
                    for q in qs:
                        u = np.kron(per_qubit[q], u)
                    ut = torch.from_numpy(u).cuda()
                    v = psi.view(-1, 1 << len(qs), 1 << lo)
                    psi = (v.view(-1, 1 << len(qs)) @ ut.T if lo == 0 else torch.matmul(ut, v)).reshape(-1)
                    del v
        else:                                            # CNOT
            _cnot(psi, q0, q1)
    p = torch.view_as_real(psi).square().sum(-1)
    z = [float(_on_pair(p, q)[:, 0].sum() - _on_pair(p, q)[:, 1].sum()) for q in range(n)]
    return {"z": np.array(z), "amplitudes": psi}


def _exact_vqe_energy(case, seed):
    n = case["n"]
    coeffs, strings = workloads.pauli_hamiltonian(n, case["terms"], seed)
    params = workloads.vqe_parameter_sets(1, 2 * n * case["depth"], seed)[0]
    psi = _new_state(n)
    for layer in params.reshape(case["depth"], 2, n):
        for q in range(n):
            c, s = math.cos(layer[0, q] / 2), math.sin(layer[0, q] / 2)
            _apply(psi, q, ((c, -s), (s, c)))
        for q in range(n):
            e = complex(math.cos(layer[1, q] / 2), math.sin(layer[1, q] / 2))
            _apply(psi, q, ((e.conjugate(), 0), (0, e)))
        for q in range(n - 1):
            _cnot(psi, q, q + 1)
    i = torch.arange(1 << n, device="cuda")
    return sum(float(c) * float(torch.vdot(psi, _times_string(psi, i, s)).real) for c, s in zip(coeffs, strings))


def _exact_qaoa_grad(n, edges, gammas, betas):
    psi, cut = _qaoa_state(n, edges, gammas, betas)
    energy = float((torch.view_as_real(psi).square().sum(-1) * cut).sum())
    lam = psi * cut
    p = len(gammas)
    grad = np.zeros(2 * p)
    diag = len(edges) - 2 * cut
    for l in range(p - 1, -1, -1):
        for q in range(n):                               # X_q commutes with the layer's mixers
            v, w = _on_pair(lam, q), _on_pair(psi, q)
            grad[p + l] += 2 * float((torch.sum(v[:, 0].conj() * w[:, 1]) + torch.sum(v[:, 1].conj() * w[:, 0])).imag)
        for s in (psi, lam):
            _rx_all(s, n, -float(betas[l]))
        grad[l] = 2 * float(torch.sum(lam.conj() * diag * psi).imag)
        phase = torch.exp(1j * float(gammas[l]) * diag)
        psi *= phase
        lam *= phase
    return energy, grad


def _ry_cz_layers(psi, theta, n, inverse=False):
    """One layer of Ry(theta[:, q]) on every qubit, then CZ(q, q+1), on real vectors (sets, 2^n)."""
    i = torch.arange(1 << n, device="cuda")
    sign = 1.0 - 2.0 * (torch.stack([(i >> q) & (i >> (q + 1)) & 1 for q in range(n - 1)]).sum(0) & 1)
    if inverse:
        psi *= sign
    for q in range(n):
        t = theta[:, q, None, None] / 2
        c, s = torch.cos(t), torch.sin(t) * (-1 if inverse else 1)
        v = _on_pair(psi, q)
        a, b = v[..., 0, :].clone(), v[..., 1, :].clone()
        v[..., 0, :] = c * a - s * b
        v[..., 1, :] = s * a + c * b
    if not inverse:
        psi *= sign


def _exact_vqe_batch(case, seed):
    n, depth, sets = case["n"], case["depth"], case["sets"]
    coeffs, strings = workloads.pauli_hamiltonian(n, case["terms"], seed)
    params = torch.from_numpy(workloads.vqe_parameter_sets(sets, n * depth, seed)).cuda().view(sets, depth, n)
    i = torch.arange(1 << n, device="cuda")
    energies, grads = [], []
    for lo in range(0, sets, 64):
        th = params[lo:lo + 64]
        psi = torch.zeros(len(th), 1 << n, dtype=torch.float64, device="cuda")
        psi[:, 0] = 1
        for l in range(depth):
            _ry_cz_layers(psi, th[:, l], n)
        hpsi = torch.zeros_like(psi)
        for c, s in zip(coeffs, strings):
            x, z, ny = _string_masks(s)
            if ny % 2 == 0:          # the state is real: odd strings are imaginary and add nothing
                j = i ^ x
                hpsi += psi[:, j] * ((1 - 2 * _parity(j, z)) * (float(c) * (1 if ny % 4 == 0 else -1)))
        energies.append((psi * hpsi).sum(1))
        if case["gradient"] != "none":
            g = torch.zeros_like(th)
            for l in range(depth - 1, -1, -1):
                for v in (psi, hpsi):
                    _ry_cz_layers(v, th[:, l], n, inverse=True)
                # Ry rotations of one layer commute: dE/dtheta_q = <lambda| -i Y_q |psi>
                for q in range(n):
                    a, b = _on_pair(hpsi, q), _on_pair(psi, q)
                    g[:, l, q] = (a[:, :, 1] * b[:, :, 0] - a[:, :, 0] * b[:, :, 1]).sum((1, 2))
            grads.append(g.reshape(len(th), -1))
    out = {"energies": torch.cat(energies)}
    if case["gradient"] != "none":
        out["gradients"] = torch.cat(grads)
    return out


def _exact_mlp(case, seed):
    x, t, w = (torch.from_numpy(v).cuda().double() for v in _mlp_inputs(case, seed))
    h, shapes = case["hidden"], []
    for rows, cols in ((h, 325), (h, h), (8, h)):
        shapes += [(rows, cols), (rows,)]
    m, v, loss = torch.zeros_like(w), torch.zeros_like(w), 0.0
    for step in range(1, case["steps"] + 1):
        r0 = (step - 1) * case["batch"] % case["rows"]
        xb, tb = x[r0:r0 + case["batch"]], t[r0:r0 + case["batch"]]
        w.requires_grad_(True)
        parts = [p.view(s) for p, s in zip(torch.split(w, [int(np.prod(s)) for s in shapes]), shapes)]
        y = torch.relu(xb @ parts[0].T + parts[1])
        y = torch.relu(y @ parts[2].T + parts[3]) @ parts[4].T + parts[5]
        e = (y - tb).square().mean()
        (g,) = torch.autograd.grad(e, w)
        loss, w = float(e.detach()), w.detach()
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        w = w - 1e-3 * (m / (1 - 0.9 ** step)) / (torch.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
    return {"loss": loss, "params": w}


def exact(case, seed):
    kind = case["kind"]
    if kind == "vqe_energy":
        return _exact_vqe_energy(case, seed)
    if kind == "maxcut":
        edges = _graph(case["n"], Stream(seed, 2))
        u = Stream(seed, 3).take(2 * case["p"])
        psi, cut = _qaoa_state(case["n"], edges, -u[:case["p"]], u[case["p"]:])
        prob = torch.view_as_real(psi).square().sum(-1)
        return {"probabilities": prob, "expected_cut": float((prob * cut).sum())}
    if kind == "circuit":
        return _exact_circuit(case, seed)
    if kind == "observables":
        psi = _amplitudes(case["n"], case["precision"], seed)
        i = torch.arange(1 << case["n"], device="cuda")
        return np.array([float(torch.vdot(psi, _times_string(psi, i, s)).real) for s in _strings(case, seed)])
    if kind == "qaoa_batch":
        graphs, g, b = _qaoa_inputs(case, seed)
        energies = []
        for k, (n, edges) in enumerate(graphs):
            psi, cut = _qaoa_state(n, edges, g[k], b[k])
            energies.append(float((torch.view_as_real(psi).square().sum(-1) * cut).sum()))
        return {"energies": np.array(energies)}          # the sampled cuts are whole numbers
    if kind == "qaoa_grad":
        graphs, g, b = _qaoa_inputs(case, seed)
        got = [_exact_qaoa_grad(n, e, g[k], b[k]) for k, (n, e) in enumerate(graphs)]
        return {"energies": np.array([e for e, _ in got]), "gradients": np.stack([x for _, x in got])}
    if kind == "vqe_batch":
        return _exact_vqe_batch(case, seed)
    if kind == "mlp":
        return _exact_mlp(case, seed)
    return None                                          # shots: whole numbers
