"""Shots on both sides of the rule for the sampler's node size, against the
oracle's walk of the same tree (equal indices)."""
import numpy as np
import pytest

import oracle
from snuqs_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [capi.SQ_C128, capi.SQ_C64])
@pytest.mark.parametrize("n", [1, 4, 5, 6, 7, 8, 11, 12, 13, 18, 23])
def test_node_sizes(n, dtype):
    rng = np.random.default_rng(n)
    psi = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    psi[rng.integers(0, 1 << n, max(1, (1 << n) // 3))] = 0  # empty runs
    psi[-1] = 0
    psi[0] += 1
    psi = (psi / np.linalg.norm(psi)).astype(np.complex64 if dtype == capi.SQ_C64 else np.complex128)
    st = capi.State(n, dtype)
    st.from_host(psi)
    rule = max(1 << 14, (1 << n) >> 7)
    u = np.concatenate([[0.0, np.nextafter(1.0, 0.0)], rng.random(rule)])
    want = oracle.sample_inverse_cdf(psi, u)
    for shots in (1, rule - 1, rule, rule + 2):
        assert np.array_equal(st.sample(u[:shots]), want[:shots]), shots
    st.close()
