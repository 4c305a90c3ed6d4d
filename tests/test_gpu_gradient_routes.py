"""Gradient batches of one width by every route against single gradients: the
multi-state sweeps, the generated and the generic kernel of one CTA per
circuit, and batches that only look like parameter sets of one program."""
import numpy as np
import pytest

from snuqs_b200 import adjoint, capi, circuits

pytestmark = pytest.mark.gpu


def program(n, layers):
    ops, p = [("Hadamard", (q,), ()) for q in range(n)], 0
    for l in range(layers):
        ops += [(("ZZ", "XX", "YY")[(q + l) % 3], (q, (q + 1) % n), (0.0,), (p,)) for q in range(n)]
        ops += [(("RotX", "RotY", "PhaseShift")[(q + l) % 3], (q,), (0.0,), (p + 1,)) for q in range(n)]
        p += 2
    return ops, p


def check(n, dtype, programs, thetas, params, tile=0):
    """Gradients of every circuit; (blocks of the launch, generated kernels ran)."""
    terms = circuits.random_pauli_hamiltonian(n, 7, seed=n) + [(0.5, "Z" * n)]
    b = capi.Batch(dtype)
    b.set_option(capi.SQ_BOPT_TILE_BITS, tile)
    ham = b.add_hamiltonian(n, terms)
    for ops, th in zip(programs, thetas):
        b.add_circuit(n, adjoint.bind(ops, th), ham)
    before = capi.jit_info()[1]
    e, g = b.run_gradients(params)
    route = b.last_timing()[1], capi.jit_info()[1] > before
    b.close()
    ws = adjoint.Workspace(n)
    # FP64 sums of 2^n products of size at most the Hamiltonian's weight, over
    # at most 6 n angles; complex64 amplitudes carry the roundings of its gates.
    tol = (1e-12 if dtype == capi.SQ_C128 else 1e-4) * sum(abs(w) for w, _ in terms) * 6 * n
    for i in range(0, len(programs), max(1, len(programs) // 6)):
        es, gs = adjoint.adjoint_gradient(ws, programs[i], thetas[i], terms, params)
        assert abs(e[i] - es) <= tol
        np.testing.assert_allclose(g[i], gs, rtol=0, atol=tol)
    ws.close()
    return route


@pytest.mark.parametrize("route", ["multi", "generated", "generic"])
@pytest.mark.parametrize("n,tile", [(11, 10), (12, 0), (14, 0)])
def test_sets_of_one_program(n, tile, route, monkeypatch):
    monkeypatch.setenv("SQ_BATCH_MULTI", "1" if route == "multi" else "0")
    monkeypatch.setenv("SQ_JIT", "0" if route == "generic" else "1")
    ops, params = program(n, 2)
    sets = 10
    thetas = np.random.default_rng(n).uniform(0, 2 * np.pi, (sets, params))
    blocks, jit = check(n, capi.SQ_C128, [ops] * sets, thetas, params, tile)
    assert (blocks > sets) == (route == "multi" and n >= 12)
    if route == "generic":
        assert blocks <= sets


@pytest.mark.parametrize("dtype", [capi.SQ_C128, capi.SQ_C64])
@pytest.mark.parametrize("kind", ["different circuits", "a dropped gate", "a gate less"])
def test_circuits_of_one_width(kind, dtype):
    n, sets = 13, 12
    ops, params = program(n, 2)
    thetas = np.random.default_rng(5).uniform(0.1, 3.0, (sets, params))
    programs = [ops] * sets
    if kind == "different circuits":
        programs = [[(o[0], tuple((q * (1 + 2 * (k % 3)) + k) % n for q in o[1])) + tuple(o[2:]) for o in ops]
                    for k in range(sets)]
    elif kind == "a dropped gate":
        thetas[7, 1] = 0.0
    else:
        programs = programs[:-1] + [ops[:-1]]
    blocks, _ = check(n, dtype, programs, thetas, params)
    assert blocks <= sets  # one CTA per circuit
