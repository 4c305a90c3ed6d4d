"""Which kernels a gradient batch takes: parameter sets of one program the
multi-state sweeps (whose source NVRTC compiles here), everything else one CTA
per circuit.  The engine's host code over pretended devices
(tests/native/fake_cudart.cc), where two blocks fit an SM: the multi-state
sweeps fill the device, the other kernel has a block per circuit."""
import os
import subprocess
import sys

import pytest

from tests.native.build import build_fake

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import sys
from snuqs_b200 import capi

capi.LIB_PATH = sys.argv[1]
n, sets = 13, 40


def program(k, first=0.1):
    ops = [("RotX", (q,), (first + 0.01 * k + q,), (q % 2,)) for q in range(n)]
    return ops + [("ZZ", (q, (q + 1) % n), (0.2 + q,), (q % 2,)) for q in range(n)]


def blocks(dtype, circuits, tile=0):
    b = capi.Batch(dtype)
    b.set_option(capi.SQ_BOPT_TILE_BITS, tile)
    h = b.add_hamiltonian(n, [(1.0, "Z" * 2 + "I" * (n - 2)), (0.5, "I" * (n - 1) + "X")])
    for ops in circuits:
        b.add_circuit(n, ops, h)
    out = []
    for _ in range(2):
        b.run_gradients(2)
        out.append(b.last_timing()[1])
    b.close()
    assert out[0] == out[1]
    return out[0]


same = [program(k) for k in range(sets)]
turned = [[(g, tuple((q + k) % n for q in t), a, p) for g, t, a, p in program(k)] for k in range(sets)]
dropped = same[:-1] + [[(g, t, (0.0,) if i == 3 else a, p) for i, (g, t, a, p) in enumerate(same[-1])]]
shorter = same[:-1] + [same[-1][:-1]]
multi = sys.argv[2] == "multi"
assert (blocks(capi.SQ_C128, same) > sets) == multi
assert (blocks(capi.SQ_C128, same[:1]) > 1) == multi
for mixed in (turned, dropped, shorter):
    assert blocks(capi.SQ_C128, mixed) == sets
assert blocks(capi.SQ_C64, same) == sets
"""


@pytest.mark.parametrize("env,expect", [({}, "multi"), ({"SQ_BATCH_MULTI": "0"}, "single"), ({"SQ_JIT": "0"}, "single")])
def test_gradient_routes(tmp_path, env, expect):
    r = subprocess.run([sys.executable, "-c", SCRIPT, build_fake(str(tmp_path)), expect], cwd=ROOT,
                       env=dict(os.environ, HOME=str(tmp_path), **env), capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
