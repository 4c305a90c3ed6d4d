"""The tiled Pauli-sum expectation against the oracle: states below, at and
above one tile, groups of one and of many terms, both Y parities, masks inside
the low bits, and sums of more groups than one plan holds."""
import numpy as np
import pytest

import oracle
from snuqs_b200 import capi

pytestmark = pytest.mark.gpu


def terms_of(n, count, kind, rng):
    letters = np.array(list("IXYZ"))
    out = []
    for t in range(count):
        if kind == "random":
            s = letters[rng.integers(4, size=n)]
        elif kind == "diagonal":
            s = np.where(rng.integers(2, size=n) == 1, "Z", "I")
        elif kind == "few masks":  # many terms share a flip mask, with both Y parities
            flip = (np.arange(n) * 7 + t % 3) % 3 == 0
            s = np.where(flip, np.where(rng.integers(2, size=n) == 1, "Y", "X"),
                         np.where(rng.integers(2, size=n) == 1, "Z", "I"))
        else:  # flips on the last (lowest) three qubits only
            s = np.where(rng.integers(2, size=n) == 1, "Z", "I").astype(object)
            s[max(0, n - 3):] = letters[rng.integers(4, size=min(n, 3))]
        out.append((float(rng.standard_normal()), "".join(s)))
    return out


@pytest.mark.parametrize("dtype", [capi.SQ_C128, capi.SQ_C64])
@pytest.mark.parametrize("n", [1, 2, 4, 8, 9, 10, 11, 12, 14, 17])
def test_expectation(n, dtype):
    rng = np.random.default_rng(n)
    psi = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    psi = (psi / np.linalg.norm(psi)).astype(np.complex64 if dtype == capi.SQ_C64 else np.complex128)
    st = capi.State(n, dtype)
    st.from_host(psi)
    for kind, count in (("random", 1), ("random", 40), ("diagonal", 25), ("few masks", 60), ("low", 30),
                        ("random", 300)):
        terms = terms_of(n, count, kind, rng)
        got, want = st.expectation(terms), oracle.expectation_indexed(psi, n, terms)
        # Every term is a sum of 2^n products of total size at most |w|; both
        # sides add them in FP64 (rounding far below 1e-13 of that).
        tol = 1e-13 * sum(abs(w) for w, _ in terms)
        assert abs(got - want) <= tol, (kind, count, got, want)
    assert abs(st.norm2() - np.sum(np.abs(psi.astype(np.complex128)) ** 2)) <= 1e-13
    assert st.expectation([]) == 0.0
    st.close()
