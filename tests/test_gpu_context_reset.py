"""A context opened after the process's CUDA context was torn down works, although an
older handle was never closed: nothing on the host side outlives the CUDA context that
it belongs to.  In a child process, so that the other tests keep theirs."""
import os
import subprocess
import sys

import pytest

from conftest import PKG, ROOT

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes, sys
sys.path[:0] = [%r, %r, %r]
import numpy as np
import haplo_gb300 as hx
from conftest import small_cohort
from haplo_gb300.admix import random_init
c = small_cohort(60, 20, 3, seed=3)
q, p = random_init(60, 20, 3, np.random.default_rng(1))
def opened():
    return hx.GB300Admix(c["bed"], 60, 20, 3, bytes_per_snp=c["bed"].shape[1], n_snp=c["bed"].shape[0])
a = opened()
first = a.loglikelihood(q, p)
a._h = None                                   # never closed
cu = ctypes.CDLL("libcuda.so.1")
dev = ctypes.c_int()
assert cu.cuDeviceGet(ctypes.byref(dev), 0) == 0 and cu.cuDevicePrimaryCtxReset_v2(dev) == 0
ds = [opened() for _ in range(3)]
for d in ds:
    assert d.loglikelihood(q, p) == first
    d.set_qp(q, p)
    assert np.isfinite(d.fit(n_iter=2, rtol=0.0, em_iters=1)["ll"])
for d in ds:
    d.close()
print("reopened")
"""


def test_context_opened_after_a_reset(hx, O):
    r = subprocess.run([sys.executable, "-c", CHILD % (ROOT, PKG, os.path.join(ROOT, "tests"))],
                       capture_output=True, text=True, timeout=300)
    assert "reopened" in r.stdout, r.stdout + r.stderr
