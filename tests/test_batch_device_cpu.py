"""A batch made on one device and run from a thread whose current device is
another: every call that acts on the current device (kernel attributes,
occupancy, allocations, launches) is made on the batch's own.  The engine's
host code runs here over pretended devices (tests/native/fake_cudart.cc)."""
import os
import subprocess
import sys

import pytest

from tests.native.build import build_fake

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import sys
import numpy as np
from snuqs_b200 import capi, circuits

capi.LIB_PATH = sys.argv[1]
lib = capi.lib()
dtype = capi.SQ_C64 if sys.argv[2] == "complex64" else capi.SQ_C128
n = 13
ops = [("RotX", (q,), (0.1 + q,), (q % 2,)) for q in range(n)]
ops += [("ZZ", (q, q + 1), (0.2 + q,), (q % 2,)) for q in range(n - 1)]
terms = [(1.0, "Z" * 2 + "I" * (n - 2)), (0.5, "I" * (n - 1) + "X")]
for call in ("run", "run_gradients", "run"):
    assert lib.sq_set_device(1) == 0
    b = capi.Batch(dtype)
    h = b.add_hamiltonian(n, terms)
    for k in range(200):
        b.add_circuit(n, [(g, q, (a[0] + 0.01 * k,), p) for g, q, a, p in ops], h)
    assert lib.sq_set_device(0) == 0
    lib.fake_expect(1)
    b.run() if call == "run" else b.run_gradients(2)
    assert lib.fake_launches() > 0
    assert lib.fake_wrong() == 0, (call, lib.fake_wrong())
"""


@pytest.mark.parametrize("jit", ["1", "0"])
@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
def test_batch_runs_on_its_own_device(tmp_path, dtype, jit):
    env = dict(os.environ, SQ_JIT=jit, HOME=str(tmp_path))
    r = subprocess.run([sys.executable, "-c", SCRIPT, build_fake(str(tmp_path)), dtype], cwd=ROOT, env=env,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
