"""Marginals of states where a warp's item takes several steps, a block several
rounds and a bin many chunks (25 qubits and more), against torch's FP64 sums."""
import numpy as np
import pytest

from snuqs_b200 import capi

pytestmark = pytest.mark.gpu


class Amplitudes:
    def __init__(self, st):
        self.__cuda_array_interface__ = {
            "shape": (1 << st.n,), "typestr": "<c8" if st.dtype == capi.SQ_C64 else "<c16",
            "data": (st.data_ptr(), False), "strides": None, "version": 3}


@pytest.mark.parametrize("n,dtype", [(25, capi.SQ_C128), (26, capi.SQ_C128), (27, capi.SQ_C64), (28, capi.SQ_C64)])
def test_marginals(n, dtype):
    import torch

    st = capi.State(n, dtype)
    psi = torch.as_tensor(Amplitudes(st), device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(n)
    psi.copy_(torch.randn(1 << n, dtype=psi.dtype, device="cuda", generator=gen))
    psi /= torch.linalg.vector_norm(psi)
    p = (psi.real.double() ** 2 + psi.imag.double() ** 2).reshape([2] * n)
    rng = np.random.default_rng(n)
    sets = [[], [0], [n - 1], list(range(5)), list(range(n - 5, n)), list(range(11)), list(range(n - 11, n)),
            [2, n - 2], [int(q) for q in rng.permutation(n)[:5]], [int(q) for q in rng.permutation(n)[:11]],
            [int(q) for q in rng.permutation(n)[:15]], [int(q) for q in rng.permutation(n)[:20]]]
    for qubits in sets:
        rest = [q for q in range(n) if q not in qubits]
        m = p.sum(dim=rest) if rest else p
        order = sorted(qubits)
        if len(qubits) > 1:
            m = m.permute([order.index(q) for q in qubits])
        # Positive terms on both sides, at most some five hundred additions
        # one after the other: 2^9 roundings of 1.2e-16 at worst.
        np.testing.assert_allclose(st.marginal_probabilities(qubits), m.reshape(-1).cpu().numpy(), rtol=6e-14, atol=0,
                                   err_msg=str(qubits))
    del p, psi
    st.close()
