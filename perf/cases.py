"""The work that the performance of the engine is judged by: user-level calls over the range of
sizes, precisions and circuit shapes the framework is used at.

A case is a dict of plain values.  ``prepare`` makes what a user's program holds before the call
(a state handle, a bound circuit, a batch, a Hamiltonian), ``run`` is one pass through the public
entry points, ``exact`` the same result in 64 bits from plain torch, ``work`` the bytes and
operations a pass cannot do without.  The circuit's structure (which gate on which qubits) comes
from the case, the angles, matrices and amplitudes from the seed: one program run again with
other parameters.
"""
import math

import numpy as np
import torch

from snuqs_b200 import adjoint, capi, circuits
from snuqs_b200.simulation import StateVectorSimulation

C128, C64 = "complex128", "complex64"


def listed():
    return [
        # One task of a plugin user at the small end: a new simulation, 100 gates on 10 qubits,
        # state vector and probabilities back on the host.  Latency and launches.
        {"name": "simulate 10q", "kind": "simulate", "shape": "mix", "n": 10, "gates": 100, "dtype": C128,
         "circuit": 11},
        # A circuit of ordinary width in the cheaper precision, on a state that is kept.
        {"name": "mix 17q complex64", "kind": "circuit", "shape": "mix", "n": 17, "gates": 240, "dtype": C64,
         "circuit": 5},
        # A hardware-efficient ansatz with the full probability vector: the usual variational task.
        {"name": "ansatz 20q probabilities", "kind": "simulate", "shape": "ansatz", "n": 20, "gates": 4,
         "dtype": C128, "circuit": 0},
        # The benchmark's random gate mix: 400 gates on a 16 GiB state.
        {"name": "mix 30q", "kind": "circuit", "shape": "mix", "n": 30, "gates": 400, "dtype": C128,
         "circuit": 1234},
        # Quantum-volume circuits (dense two-qubit gates) in both precisions; an odd width leaves one
        # qubit idle in every layer.
        {"name": "volume 26q", "kind": "circuit", "shape": "volume", "n": 26, "gates": 26, "dtype": C128,
         "circuit": 7},
        {"name": "volume 27q complex64", "kind": "circuit", "shape": "volume", "n": 27, "gates": 27, "dtype": C64,
         "circuit": 8},
        # Energies of a prepared state: a Hamiltonian of random Pauli strings and a diagonal one.
        {"name": "energies 25q", "kind": "energies", "n": 25, "terms": 64, "dtype": C128, "circuit": 3},
        # Outcome distributions of some qubits of a large state.
        {"name": "marginals 26q", "kind": "marginals", "n": 26, "targets": "1,5,11", "dtype": C128, "circuit": 4},
        # A million shots of a large state.
        {"name": "shots 28q", "kind": "shots", "n": 28, "shots": 1000000, "dtype": C128},
        # One training step's gradient: QAOA MaxCut, 16 parameters.
        {"name": "gradient 24q", "kind": "gradient", "n": 24, "layers": 8, "dtype": C128, "circuit": 1234},
        # A VQE iteration over many small circuits of uneven size, all angles new.
        {"name": "batch energies", "kind": "batch_energies", "low": 8, "n": 20, "sets": 512, "terms": 64,
         "layers": 6, "dtype": C128, "circuit": 1234},
        # Gradients of many parameter sets of one circuit.
        {"name": "batch gradients 16q", "kind": "batch_gradients", "n": 16, "sets": 64, "layers": 8,
         "dtype": C128, "circuit": 1234},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["simulate", "circuit", "circuit", "circuit", "energies", "marginals", "shots", "gradient",
                       "batch_energies", "batch_gradients"])
    case = {"kind": kind, "dtype": rng.choice([C128, C128, C64])}
    if kind != "shots":
        case["circuit"] = rng.randrange(1, 1 << 20)
    if kind == "simulate":
        case["shape"] = rng.choice(["mix", "ansatz"])
        case["n"] = rng.randint(6, 21)
        case["gates"] = log(40, 240) if case["shape"] == "mix" else rng.randint(2, 6)
    elif kind == "circuit":
        case["shape"] = rng.choice(["mix", "mix", "volume"])
        case["n"] = rng.randint(13, 29) if case["shape"] == "mix" else rng.randint(19, 27)
        case["gates"] = log(60, 400) if case["shape"] == "mix" else rng.randint(6, case["n"])
    elif kind == "energies":
        case["n"] = rng.randint(15, 26)
        case["terms"] = log(12, 96)
    elif kind == "marginals":
        case["n"] = rng.randint(17, 27)
        k = sorted(rng.sample(range(1, case["n"] - 2), 3))
        case["targets"] = ",".join(str(x) for x in k)
    elif kind == "shots":
        case["n"] = rng.randint(14, 28)
        case["shots"] = log(500, 1000000)
    elif kind == "gradient":
        case["n"] = 2 * rng.randint(7, 12)
        case["layers"] = rng.randint(2, 8)
    elif kind == "batch_energies":
        case["low"], case["n"] = rng.randint(6, 10), rng.randint(14, 20)
        case["sets"], case["terms"], case["layers"] = log(64, 400), log(12, 64), rng.randint(2, 6)
    else:
        case["n"] = 2 * rng.randint(5, 8)
        case["sets"], case["layers"] = log(16, 64), rng.randint(2, 8)
    return case


# ---- inputs ----------------------------------------------------------------------------------


def _sq(case):
    return capi.SQ_C64 if case["dtype"] == C64 else capi.SQ_C128


class _Amplitudes:
    """A state's device memory, for torch (holds the state while a tensor of it lives)."""

    def __init__(self, state):
        self.state = state
        self.__cuda_array_interface__ = {
            "shape": (1 << state.n,), "typestr": "<c8" if state.dtype == capi.SQ_C64 else "<c16",
            "data": (state.data_ptr(), False), "strides": None, "version": 3}


def _tensor(state):
    return torch.as_tensor(_Amplitudes(state), device="cuda")


def _random_state(case, seed):
    """Normalised complex Gaussian amplitudes: the statistics of a deep random circuit's output."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)
    psi = torch.randn(1 << case["n"], dtype=torch.complex64 if case["dtype"] == C64 else torch.complex128,
                      device="cuda", generator=gen)
    psi /= torch.linalg.vector_norm(psi)
    return psi


def _ops(case, seed):
    rng = np.random.default_rng([int(seed), 1])
    n = case["n"]
    if case["shape"] == "ansatz":
        return circuits.vqe_ansatz(n, rng.uniform(0, 2 * np.pi, 2 * n * case["gates"]), layers=case["gates"])
    if case["shape"] == "mix":
        return [(name, qubits, tuple(float(x) for x in rng.uniform(0, 2 * np.pi, len(angles))))
                for name, qubits, angles in circuits.random_mix(n, case["gates"], seed=case["circuit"])]
    pairs = np.random.default_rng(case["circuit"])
    ops = []
    for _ in range(case["gates"]):
        perm = pairs.permutation(n)
        ops += [("Unitary", (int(perm[2 * w]), int(perm[2 * w + 1])), (), circuits.haar_unitary(4, rng))
                for w in range(n // 2)]
    return ops


def _qaoa(case):
    edges = circuits.random_regular_graph(case["n"], 3, seed=case["circuit"])
    p = case["layers"]
    ops = [("Hadamard", (q,), ()) for q in range(case["n"])]
    for l in range(p):
        ops += [("ZZ", (i, j), (0.0,), (l,)) for i, j in edges]
        ops += [("RotX", (q,), (0.0,), (p + l,)) for q in range(case["n"])]
    return ops, circuits.maxcut_hamiltonian(case["n"], edges), edges


def _hamiltonians(case):
    """Random Pauli strings, and the diagonal coupling sum of a ring."""
    n = case["n"]
    ring = [(1.0, "".join("Z" if q in (i, (i + 1) % n) else "I" for q in range(n))) for i in range(n)]
    return [circuits.random_pauli_hamiltonian(n, case["terms"], seed=case["circuit"]), ring]


def _targets(case):
    rng = np.random.default_rng(case["circuit"])
    return [[int(q) for q in rng.choice(case["n"], size=int(k), replace=False)] for k in case["targets"].split(",")]


def _batch_sizes(case):
    return [int(x) for x in np.random.default_rng(case["circuit"]).integers(case["low"], case["n"] + 1, case["sets"])]


def _batch_angles(case, seed):
    rng = np.random.default_rng([int(seed), 2])
    return [rng.uniform(0, 2 * np.pi, 2 * n * case["layers"]) for n in _batch_sizes(case)]


def _batch_terms(case, n):
    return circuits.random_pauli_hamiltonian(n, case["terms"], seed=case["circuit"] + n)


def _thetas(case, seed, sets):
    return np.random.default_rng([int(seed), 3]).uniform(0, np.pi, (sets, 2 * case["layers"]))


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "simulate":
        s["ops"] = _ops(case, seed)
    elif kind == "circuit":
        s["ops"] = _ops(case, seed)
        s["state"] = capi.State(case["n"], _sq(case))
    elif kind in ("energies", "marginals", "shots"):
        s["state"] = capi.State(case["n"], _sq(case))
        _tensor(s["state"]).copy_(_random_state(case, seed))
        if kind == "energies":
            s["hams"] = _hamiltonians(case)
        elif kind == "marginals":
            s["targets"] = _targets(case)
        else:
            s["uniforms"] = np.random.default_rng([int(seed), 4]).random(case["shots"])
    elif kind == "gradient":
        s["ops"], s["terms"], _ = _qaoa(case)
        s["theta"] = _thetas(case, seed, 1)[0]
        s["ws"] = adjoint.Workspace(case["n"], _sq(case))
    elif kind == "batch_energies":
        b = s["batch"] = capi.Batch(_sq(case))
        s["angles"] = _batch_angles(case, seed)
        ham = {}
        for n, a in zip(_batch_sizes(case), s["angles"]):
            if n not in ham:
                ham[n] = b.add_hamiltonian(n, _batch_terms(case, n))
            b.add_circuit(n, circuits.vqe_ansatz(n, a, layers=case["layers"]), ham[n])
    else:
        ops, terms, _ = _qaoa(case)
        b = s["batch"] = capi.Batch(_sq(case))
        ham = b.add_hamiltonian(case["n"], terms)
        for theta in _thetas(case, seed, case["sets"]):
            b.add_circuit(case["n"], adjoint.bind(ops, theta), ham)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "simulate":
        sim = StateVectorSimulation(case["n"], precision=case["dtype"])
        sim.evolve(s["ops"])
        out = [sim.probabilities, sim.state_vector]
        sim.close()
        return out
    if kind == "circuit":
        state = s["state"]
        state.init_basis(0)
        state.apply_ops(s["ops"])
        state.flush()
        return _tensor(state)
    if kind == "energies":
        return np.array([s["state"].expectation(h) for h in s["hams"]])
    if kind == "marginals":
        return [s["state"].marginal_probabilities(t) for t in s["targets"]]
    if kind == "shots":
        return s["state"].sample(s["uniforms"])
    if kind == "gradient":
        e, g = adjoint.adjoint_gradient(s["ws"], s["ops"], s["theta"], s["terms"], 2 * case["layers"])
        return [np.float64(e), g]
    if kind == "batch_energies":
        for i, a in enumerate(s["angles"]):
            s["batch"].set_angles(i, a)
        return s["batch"].run()
    return list(s["batch"].run_gradients(2 * case["layers"]))


# ---- 64-bit results from plain torch ---------------------------------------------------------


def _matrix(name, a):
    """Gate matrices of the mix; the first target is the most significant bit of the index."""
    if name in ("RotX", "RotY", "RotZ", "XX", "YY", "ZZ"):
        pauli = {"X": np.array([[0, 1], [1, 0]], complex), "Y": np.array([[0, -1j], [1j, 0]]),
                 "Z": np.diag([1.0 + 0j, -1])}[name[-1]]
        g = pauli if name.startswith("Rot") else np.kron(pauli, pauli)
        return math.cos(a[0] / 2) * np.eye(len(g)) - 1j * math.sin(a[0] / 2) * g
    if name == "U":
        c, s = math.cos(a[0] / 2), math.sin(a[0] / 2)
        return np.array([[c, -np.exp(1j * a[2]) * s], [np.exp(1j * a[1]) * s, np.exp(1j * (a[1] + a[2])) * c]])
    if name == "PhaseShift":
        return np.diag([1, np.exp(1j * a[0])])
    if name == "CZ":
        return np.diag([1.0 + 0j, 1, 1, -1])
    order = {"CX": [0, 1, 3, 2], "Swap": [0, 2, 1, 3], "ISwap": [0, 2, 1, 3],
             "CCNot": [0, 1, 2, 3, 4, 5, 7, 6], "CSwap": [0, 1, 2, 3, 4, 6, 5, 7]}[name]
    m = np.eye(len(order), dtype=complex)[order]
    if name == "ISwap":
        m[1, 2] = m[2, 1] = 1j
    return m


def _apply(psi, n, mat, qubits):
    """psi [K, 2^n]; mat [d, d] or one of its own for each of the K states."""
    k = len(qubits)
    order = sorted(range(k), key=lambda j: qubits[j])
    mat = torch.as_tensor(mat, dtype=torch.complex128, device=psi.device)
    lead = list(range(mat.dim() - 2))
    axes = [len(lead) + j for j in order]
    mat = mat.reshape(list(mat.shape[:-2]) + [2] * (2 * k)).permute(lead + axes + [x + k for x in axes])
    mat = mat.reshape(list(mat.shape[: len(lead)]) + [1 << k, 1 << k])
    shape, last = [psi.shape[0]], -1
    for q in sorted(qubits):
        shape += [1 << (q - last - 1), 2]
        last = q
    shape.append(1 << (n - 1 - last))
    front = [2 + 2 * j for j in range(k)]
    rest = [1 + 2 * j for j in range(k + 1)]
    x = psi.reshape(shape).permute([0] + front + rest)
    full = list(x.shape)
    x = torch.matmul(mat, x.reshape(shape[0], 1 << k, -1)).reshape(full)
    back = [0] * len(full)
    for i, d in enumerate([0] + front + rest):
        back[d] = i
    return x.permute(back).reshape(psi.shape)


def _zero(count, n):
    psi = torch.zeros(count, 1 << n, dtype=torch.complex128, device="cuda")
    psi[:, 0] = 1
    return psi


def _pauli(psi, n, string):
    """P psi for one Pauli string over the last axis."""
    i = torch.arange(1 << n, device=psi.device)
    x = sum(1 << (n - 1 - q) for q, c in enumerate(string) if c in "XY")
    z = [n - 1 - q for q, c in enumerate(string) if c in "YZ"]
    j = i ^ x
    par = torch.zeros_like(i)
    for b in z:
        par ^= (j >> b) & 1
    return psi[..., j] * (1 - 2 * par).double() * (1j ** string.count("Y"))


def _energy(psi, n, terms):
    return sum(w * (psi.conj() * _pauli(psi, n, p)).sum(-1).real for w, p in terms)


def _rotations(name, angles):
    """One rotation matrix for each of the angles."""
    return np.array([_matrix(name, [x]) for x in angles])


def _qaoa_exact(case, thetas):
    """Energies and gradients of the parameter sets: an adjoint pass in plain torch."""
    n, p = case["n"], case["layers"]
    _, terms, edges = _qaoa(case)
    i = torch.arange(1 << n, device="cuda")
    zz = [(1 - 2 * (((i >> (n - 1 - a)) ^ (i >> (n - 1 - b))) & 1)).double() for a, b in edges]
    cost = sum(zz)
    t = torch.as_tensor(thetas, device="cuda")
    psi = torch.full((len(thetas), 1 << n), 2.0 ** (-n / 2), dtype=torch.complex128, device="cuda")
    for l in range(p):
        psi = psi * torch.exp(-0.5j * t[:, l, None] * cost)
        for q in range(n):
            psi = _apply(psi, n, _rotations("RotX", thetas[:, p + l]), (q,))
    lam = psi * cost
    energy = (psi.conj() * lam).sum(-1).real
    grad = torch.zeros(len(thetas), 2 * p, dtype=torch.float64, device="cuda")
    for l in reversed(range(p)):
        for q in range(n):
            flipped = psi.reshape(len(thetas), 1 << q, 2, -1).flip(2).reshape(psi.shape)
            grad[:, p + l] += (lam.conj() * flipped).sum(-1).imag
        for q in range(n):
            m = _rotations("RotX", -thetas[:, p + l])
            psi, lam = _apply(psi, n, m, (q,)), _apply(lam, n, m, (q,))
        grad[:, l] = (lam.conj() * (psi * cost)).sum(-1).imag
        back = torch.exp(0.5j * t[:, l, None] * cost)
        psi, lam = psi * back, lam * back
    return energy, grad


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind in ("simulate", "circuit"):
        if n > 26:
            return None  # too long for a check
        psi = _zero(1, n)
        for op in _ops(case, seed):
            psi = _apply(psi, n, op[3] if op[0] == "Unitary" else _matrix(op[0], op[2]), op[1])
        psi = psi[0]
        return psi if kind == "circuit" else [psi.abs().square().cpu().numpy(), psi.cpu().numpy()]
    if kind in ("energies", "marginals"):
        psi = _random_state(case, seed).to(torch.complex128)
        if kind == "energies":
            return np.array([float(_energy(psi, n, h)) for h in _hamiltonians(case)])
        out, prob = [], psi.abs().square()
        del psi
        for targets in _targets(case):
            # Bits of the index outside the targets are summed, highest position first.
            x, kept = prob, list(range(n))
            for q in [q for q in range(n) if q not in targets]:
                at = kept.index(q)
                x = x.reshape(1 << at, 2, -1).sum(1)
                kept.pop(at)
            x = x.reshape([2] * len(kept)).permute([kept.index(q) for q in targets]) if len(kept) < 25 else None
            out.append(None if x is None else x.reshape(-1).cpu().numpy())
        return out
    if kind == "gradient":
        e, g = _qaoa_exact(case, _thetas(case, seed, 1))
        return [np.float64(e[0].item()), g[0].cpu().numpy()]
    if kind == "batch_energies":
        sizes, angles = _batch_sizes(case), _batch_angles(case, seed)
        out = np.zeros(len(sizes))
        for m in sorted(set(sizes)):
            ids = [i for i, x in enumerate(sizes) if x == m]
            step = max(1, (1 << 24) >> m)
            for at in range(0, len(ids), step):
                part = ids[at:at + step]
                a = np.array([angles[i] for i in part]).reshape(len(part), case["layers"], 2, m)
                psi = _zero(len(part), m)
                for l in range(case["layers"]):
                    for q in range(m):
                        psi = _apply(psi, m, _rotations("RotY", a[:, l, 0, q]), (q,))
                    for q in range(m):
                        psi = _apply(psi, m, _rotations("RotZ", a[:, l, 1, q]), (q,))
                    for q in range(m - 1):
                        psi = _apply(psi, m, _matrix("CX", ()), (q, q + 1))
                out[part] = _energy(psi, m, _batch_terms(case, m)).cpu().numpy()
        return out
    if kind == "batch_gradients":
        e, g = _qaoa_exact(case, _thetas(case, seed, case["sets"]))
        return [e.cpu().numpy(), g.cpu().numpy()]
    return None  # shots are indices


# ---- bytes and operations ---------------------------------------------------------------------

# Operations an amplitude costs in one gate (a complex product is 6, a product with a real 2).
_FLOPS = {"RotX": 6, "RotY": 6, "XX": 6, "YY": 6, "RotZ": 6, "ZZ": 6, "PhaseShift": 3, "U": 14, "Unitary": 30,
          "Hadamard": 4}


def _circuit_flops(ops, n):
    return sum(_FLOPS.get(op[0], 0) for op in ops) << n


def work(case):
    kind, n = case["kind"], case["n"]
    amp = 8 if case["dtype"] == C64 else 16
    state = amp << n
    if kind == "simulate":
        return {"bytes": state + (8 << n), "flops": _circuit_flops(_ops(case, 0), n) + (3 << n)}
    if kind == "circuit":
        return {"bytes": state, "flops": _circuit_flops(_ops(case, 0), n)}
    if kind == "energies":
        # A pair of amplitudes: the real part of a product and its weight.
        return {"bytes": 2 * state, "flops": (5 * case["terms"] << (n - 1)) + (5 << n)}
    if kind == "marginals":
        ks = [int(k) for k in case["targets"].split(",")]
        return {"bytes": len(ks) * state + sum(8 << k for k in ks), "flops": len(ks) * (4 << n)}
    if kind == "shots":
        return {"bytes": state + 16 * case["shots"], "flops": 4 << n}
    if kind in ("gradient", "batch_gradients"):
        # Forward, backward on two states, and one inner product for each parameter.
        one = 3 * _circuit_flops(_qaoa(case)[0], n) + (2 * case["layers"] * 4 << n)
        sets = case.get("sets", 1)
        return {"bytes": sets * 2 * state, "flops": sets * one}
    flops = size = 0
    for m in _batch_sizes(case):
        flops += (case["layers"] * 2 * m * 6 << m) + (5 * case["terms"] << (m - 1))
        size += amp << m
    return {"bytes": size, "flops": flops}
