"""The table of H0 and H1 (csrc/helm_bessel.cuh) goes to the device on the
stream of the call that needs it first and is waited for: not on the legacy
stream, which the library's streams do not order with.  Seen from outside: a
process's first call with a real wavenumber does not wait for work queued on
the legacy stream, and gives what later calls give."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import numpy as np
import torch
import wrappers as W
import fmm2d_c_translation_b200 as fm

L = fm.lib()
rng = np.random.default_rng(1)
n = 3000
src = rng.random((2, n))
q = rng.standard_normal(n) + 1j * rng.standard_normal(n)


def call(zk):
    got, ier = W.call(L, "h", "s_c_g", 1e-8, src, q, zk=zk)
    assert ier == 0, fm.last_error()
    return got


call(30.0 + 0.1j)  # (everything but the real wavenumber's table)
torch.cuda.synchronize()
done = torch.cuda.Event()
torch.cuda._sleep(4_000_000_000)  # about two seconds on the legacy stream
done.record()
first = call(30.0)
assert not done.query(), "the call waited for the legacy stream"
torch.cuda.synchronize()
again = call(30.0)
for k in first:
    assert np.array_equal(first[k], again[k]), k
"""


def test_first_real_call_leaves_the_legacy_stream_alone():
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, CUDA_MODULE_LOADING="EAGER",
               PYTHONPATH=os.pathsep.join([os.path.dirname(here), here]))
    r = subprocess.run([sys.executable, "-c", CHILD], env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr
