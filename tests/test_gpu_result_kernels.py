"""Sampling and marginal kernels at the edges of their splits: fewer qubits
than a warp's lane bits, one node of the stored tree, blocks and chunks just
reached, and trees whose stored nodes hold several runs of 128 amplitudes."""
import numpy as np
import pytest

import oracle
from snuqs_b200 import capi

pytestmark = pytest.mark.gpu
DTYPES = [capi.SQ_C128, capi.SQ_C64]


def random_state(n, dtype, seed):
    rng = np.random.default_rng(seed)
    psi = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    psi = (psi / np.linalg.norm(psi)).astype(np.complex64 if dtype == capi.SQ_C64 else np.complex128)
    st = capi.State(n, dtype)
    st.from_host(psi)
    return st, psi


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n", [1, 3, 5, 6, 8, 9, 13, 17, 20])
def test_marginals(n, dtype):
    st, psi = random_state(n, dtype, n)
    rng = np.random.default_rng(100 + n)
    sets = [list(range(n)), [], [0], [n - 1], list(range(n))[::-1]]
    sets += [[int(q) for q in rng.permutation(n)[:k]] for k in range(1, n, 3)]
    sets += [list(range(max(0, n - 6), n)), list(range(0, max(0, n - 5)))]
    for qubits in sets:
        want = oracle.marginal_probabilities(psi, n, qubits) if qubits else \
            np.array([np.sum(np.abs(psi.astype(np.complex128)) ** 2)])
        got = st.marginal_probabilities(qubits)
        # Both sides add at most 2^n positive terms, in blocks of at most 2^8
        # sequential additions: 2^9 roundings of 1.2e-16 at worst.
        np.testing.assert_allclose(got, want, rtol=6e-14, atol=0, err_msg=str(qubits))
    st.close()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n", [1, 2, 6, 7, 8, 11, 12, 13, 17, 23, 24])
def test_shots_are_the_oracle_walk(n, dtype):
    st, psi = random_state(n, dtype, 7 * n)
    for shots in (1, 31, 33, 5000):
        u = np.random.default_rng(n + shots).random(shots)
        u[0] = 0.0
        u[-1] = np.nextafter(1.0, 0.0)
        assert np.array_equal(st.sample(u), oracle.sample_inverse_cdf(psi, u)), shots
    st.close()


def test_many_shots_per_warp():
    st, psi = random_state(15, capi.SQ_C128, 3)
    u = np.random.default_rng(5).random(700001)
    assert np.array_equal(st.sample(u), oracle.sample_inverse_cdf(psi, u))
    st.close()


@pytest.mark.parametrize("n", [31, 33])
def test_nodes_of_several_runs(n):
    """Equal weights on the eight settings of three index bits (one inside a
    run of 128 amplitudes, one inside a stored node, one above): shot s lands
    on the setting floor(8 u_s)."""
    bits = (2, 7, n - 2)
    st = capi.State(n, capi.SQ_C64)
    st.init_basis(0)
    for b in bits:
        st.apply_gate("Hadamard", (n - 1 - b,))
    u = np.random.default_rng(n).random(4099)
    e = np.floor(8 * u).astype(np.uint64)
    want = sum(((e >> np.uint64(i)) & np.uint64(1)) << np.uint64(b) for i, b in enumerate(bits))
    assert np.array_equal(st.sample(u), want)
    st.close()
