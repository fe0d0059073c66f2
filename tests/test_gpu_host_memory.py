"""A host allocation that fails is an error code, not an exception through the
C interface: a moments call in a process whose address space may not grow."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = """
import resource, sys
sys.path.insert(0, %r)
import pevsl_b200 as pv
from pevsl_b200.problems import laplacian
M = pv.Matrix.from_csr(*laplacian(3, 2, 2))
mdeg = 2000000  # 64 MB of moments on the host
with pv.Instance(M) as ev:
    assert ev.kpmdos(mdeg, 0, 2, [0.5, 6.0, 0.0, 12.0])[0] == 0
    size = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
    import numpy as np, ctypes as C
    mu, ec, iv = np.zeros(mdeg + 1), C.c_double(), np.array([0.5, 6.0, 0.0, 12.0])
    size += mu.nbytes
    resource.setrlimit(resource.RLIMIT_AS, (size + (32 << 20), size + (32 << 20)))
    st = ev.lib.pEVSL_Kpmdos(ev.p, mdeg, 0, 2, pv._ptr(iv), 1, 0, 0, pv._ptr(mu), C.byref(ec))
print("status", st)
"""


def test_moments_without_host_memory(gpu):
    r = subprocess.run([sys.executable, "-c", CHILD % ROOT], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "status -1002" in r.stdout, r.stderr[-500:]
