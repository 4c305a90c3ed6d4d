"""Rounding of sums of Pauli strings over whole states."""
import numpy as np
import pytest

import oracle
from snuqs_b200 import capi

pytestmark = pytest.mark.gpu


def ring(n):
    return [(1.0, "".join("Z" if q in (i, (i + 1) % n) else "I" for q in range(n))) for i in range(n)]


def exact_ring(psi, n):
    """The same sum with x87 extended products and a compensated total."""
    idx = np.arange(1 << n, dtype=np.uint64)
    w = np.zeros(1 << n, dtype=np.int64)
    for i in range(n):
        a, b = np.uint64(n - 1 - i), np.uint64(n - 1 - (i + 1) % n)
        w += 1 - 2 * (((idx >> a) ^ (idx >> b)) & np.uint64(1)).astype(np.int64)
    re, im = psi.real.astype(np.longdouble), psi.imag.astype(np.longdouble)
    return np.sum((re * re + im * im) * w)


@pytest.mark.parametrize("n", [18, 19, 20, 21])
def test_ring_sum_rounding(n):
    """The ring sum of Z Z strings on random states cancels to about 2^-(n/2)
    of its weights.  What a sum that carries its additions' errors leaves is
    the rounding of the products: about a dozen roundings (eight rows, their
    signed sums, the weights) of size 2^-53 * n * 2^-n for each of the 2^n
    amplitudes, independent of each other, so 2^-53 * n * 2^-(n/2) times the
    root of a dozen over the states; partial sums added plainly leave about
    ten times that."""
    rng = np.random.default_rng(n)
    errors = []
    for _ in range(12):
        psi = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
        psi /= np.linalg.norm(psi)
        st = capi.State(n, capi.SQ_C128)
        st.from_host(psi)
        errors.append(float(np.longdouble(st.expectation(ring(n))) - exact_ring(psi, n)))
        st.close()
    rms = float(np.sqrt(np.mean(np.square(errors))))
    assert rms <= 4.0 * 2.0 ** -53 * n * 2.0 ** (-n / 2), rms


@pytest.mark.parametrize("string", ["XXXXXXXXXXXX", "IIIIIIIIIIIX", "ZIIIIIIIIIII", "XIIIIIIIIIIY"])
def test_weight_near_the_range_end(string):
    """A finite weight times an expectation of at most 1 is finite: <P> = 1 on
    the +1 eigenstate of the string's letters, every other product smaller."""
    n, w = 12, 1.5e308
    eig = {"I": [1, 0], "X": [1, 1], "Y": [1, 1j], "Z": [1, 0]}
    psi = np.ones(1, dtype=np.complex128)
    for c in string:
        v = np.array(eig[c], dtype=np.complex128)
        psi = np.kron(psi, v / np.linalg.norm(v))
    st = capi.State(n, capi.SQ_C128)
    st.from_host(psi)
    got = st.expectation([(w, string)])
    st.close()
    assert np.isfinite(got) and abs(got - w) <= 1e-13 * w, got


@pytest.mark.parametrize("dtype", [capi.SQ_C128, capi.SQ_C64])
@pytest.mark.parametrize("n", [10, 11, 12, 13, 16, 21])
def test_flips_of_the_last_qubits(n, dtype):
    """Strings of one flip within the last three qubits, alone (their own
    kernel from a tile's size up), with several signs, and with others."""
    rng = np.random.default_rng(n)
    psi = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    psi = (psi / np.linalg.norm(psi)).astype(np.complex64 if dtype == capi.SQ_C64 else np.complex128)
    st = capi.State(n, dtype)
    st.from_host(psi)
    for tail in ("IIX", "IIY", "IXI", "XIY", "YXX", "YYZ", "ZIX", "XXI"):
        heads = ["".join(rng.choice(list("IZ"), n - 3)) for _ in range(3)]
        one = [(float(rng.standard_normal()), h + tail) for h in heads]
        other = [(0.7, "X" + "I" * (n - 1)), (-0.3, "I" * (n - 2) + "XX"), (0.2, "Z" * n)]
        for terms in (one[:1], one, one + other):
            got, want = st.expectation(terms), oracle.expectation_indexed(psi, n, terms)
            assert abs(got - want) <= 1e-13 * sum(abs(w) for w, _ in terms), (tail, got, want)
    st.close()
