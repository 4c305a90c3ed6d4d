"""Gradient batches of one circuit's parameter sets (multi-state sweeps) against
the single-circuit gradient: one qubit above the tile, one set and so many
that a block crosses from state to state, more inner products per sweep than a
thread keeps in registers, every generator kind, and angles that share one
parameter with different factors."""
import numpy as np
import pytest

from snuqs_b200 import adjoint, capi, circuits

pytestmark = pytest.mark.gpu


def circuit(n, kind):
    if kind == "own parameters":
        ops, p = [], 0
        for q in range(n):
            for name in ("RotY", "RotZ", "RotX"):
                ops.append((name, (q,), (0.0,), (p,)))
                p += 1
        for q in range(n - 1):
            ops.append((("XX", "YY", "ZZ", "CPhaseShift")[q % 4], (q, q + 1), (0.0,), (p,)))
            p += 1
        return ops, p
    ops = [("Hadamard", (q,), ()) for q in range(n)]
    for q in range(n):
        ops.append(("ZZ", (q, (q + 1) % n), (0.0,), (0,), (1.0 + q % 2,)))
        ops.append(("RotX", (q,), (0.0,), (1,), (0.5,)))
        ops.append(("PhaseShift", (q,), (0.0,), (0,)))
    return ops, 2


@pytest.mark.parametrize("n,sets", [(12, 1), (12, 3), (12, 300), (13, 40), (15, 2)])
@pytest.mark.parametrize("kind", ["own parameters", "shared"])
def test_sets_match_single_gradients(n, sets, kind):
    ops, params = circuit(n, kind)
    terms = circuits.random_pauli_hamiltonian(n, 9, seed=n) + [(0.7, "Z" * n), (0.3, "I" * n)]
    thetas = np.random.default_rng(n + sets).uniform(0, 2 * np.pi, (sets, params))
    b = capi.Batch(capi.SQ_C128)
    ham = b.add_hamiltonian(n, terms)
    for th in thetas:
        b.add_circuit(n, adjoint.bind(ops, th), ham)
    e, g = b.run_gradients(params)
    ws = adjoint.Workspace(n)
    # Energies and inner products are FP64 sums of 2^n products of size at most
    # the Hamiltonian's weight (and two angles share at most 3 n gates).
    tol = 1e-12 * sum(abs(w) for w, _ in terms) * 3 * n
    for i in sorted({0, sets // 2, sets - 1}):
        es, gs = adjoint.adjoint_gradient(ws, ops, thetas[i], terms, params)
        assert abs(e[i] - es) <= tol
        np.testing.assert_allclose(g[i], gs, rtol=0, atol=tol)
    e2, g2 = b.run_gradients(params)
    assert np.array_equal(e, e2) and np.array_equal(g, g2)
    ws.close()
    b.close()
