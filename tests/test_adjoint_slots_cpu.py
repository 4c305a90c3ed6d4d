"""Angles that follow one parameter share an inner-product slot only when
their factors are the same number, not-a-number among them."""
import numpy as np

from tests.native import emulator

OPS = [("RotX", (0,), (0.3,), (0,), (1.0,)), ("RotY", (1,), (0.4,), (1,), (1.0,)), ("CX", (0, 1), ()),
       ("RotX", (2,), (0.5,), (0,), (2.0,)), ("RotX", (1,), (0.7,), (0,), (1.0,)), ("CX", (1, 2), ()),
       ("RotY", (3,), (0.2,), (1,), (1.0,))]
TERMS = [(1.0, "ZZII"), (0.5, "IXZI"), (0.25, "IIIZ")]


def test_a_factor_that_is_not_a_number_keeps_to_its_parameter():
    _, want, _ = emulator.adjoint(4, OPS, TERMS, 2, tile_bits=4)
    for where in (0, 3, 4):  # the first, a different and the last factor of parameter 0
        ops = list(OPS)
        ops[where] = ops[where][:4] + ((float("nan"),),)
        _, got, _ = emulator.adjoint(4, ops, TERMS, 2, tile_bits=4)
        assert np.isnan(got[0]), (where, got)
        assert got[1] == want[1], (where, got, want)
