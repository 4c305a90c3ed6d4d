"""The marginal kernel at the edges of its splits: fewer qubits than a warp's
lane bits, chunks just reached, every target and none."""
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
