"""The bounded wait between the blocks of a cluster launch.

With a value withheld and a limit of 200 microseconds every wait runs out: the
launch ends by itself, the call returns PEVSL_ERR_CUDA, and the next call
without the fault gives the bits of the launch-per-degree recurrence.
"""
import ctypes as C

import numpy as np
import pytest

import pevsl_b200 as pv
from pevsl_b200.problems import laplacian, random_sparse_symmetric

pytestmark = pytest.mark.gpu

# symmetric structure and more than one block, so that blocks wait for each
# other: entries in registers (one and two rows per thread) and in shared memory
MATRICES = {
    "registers": lambda: laplacian(19, 20, 21), "two_rows": lambda: laplacian(26, 25, 24),
    "shared": lambda: random_sparse_symmetric(6007, 10, 900, 6),
}


def poly(deg):
    k = np.arange(deg + 1)
    return pv.Filter(1, deg, 0.0, 0.5, 6.0, 7.5, np.cos(0.7 * k) / (1.0 + 0.1 * k))


@pytest.fixture
def wait():
    lib = pv.load()

    def fault(on):
        lib.pEVSL_B200_SetClusterWait(200 if on else -1)
        lib.pEVSL_B200_WithholdClusterValues(on)

    yield fault
    fault(0)
    lib.pEVSL_B200_LastError()


@pytest.mark.parametrize("name", sorted(MATRICES))
def test_filter_wait_runs_out(gpu, wait, name):
    n, ia, ja, a = MATRICES[name]()
    M = pv.Matrix.from_csr(n, ia, ja, a)
    v = np.random.default_rng(3).standard_normal(n)
    pol, keep = pv._polparams(poly(37))
    with pv.Instance(M) as ev:
        want = ev.chebav(poly(37), v)
        x, y = pv.Vector(n, v), pv.Vector(n)
        wait(1)
        assert ev.lib.pEVSL_B200_ChebAv(ev.p, C.byref(pol), x.pv.data, y.pv.data) == pv.ERR_CUDA
        assert np.all(np.isnan(y.get()))
        wait(0)
        assert ev.lib.pEVSL_B200_ChebAv(ev.p, C.byref(pol), x.pv.data, y.pv.data) == 0
        assert np.array_equal(y.get(), want)
    M.free()


def test_lockstep_solve_reports_it(gpu, wait):
    n, ia, ja, a = laplacian(14, 13, 12)
    M = pv.Matrix.from_csr(n, ia, ja, a)
    intvs = [[0.5 + 0.2 * i, 0.7 + 0.2 * i, 0.0, 12.0] for i in range(4)]
    fl = [pv.findpol(iv)[1] for iv in intvs]
    v = np.cos(np.arange(n) * 0.37)
    outs = []
    for on in (0, 1, 0):
        wait(on)
        with pv.Instance(M) as ev:
            outs.append(pv.cheblannr_batch(ev, intvs, [150] * 4, 1e-8, v, fl))
    M.free()
    assert outs[0][0] == outs[2][0] == 0 and outs[1][0] == pv.ERR_CUDA
    for p, q in zip(outs[0][1], outs[2][1]):
        assert p["its"] == q["its"] and np.array_equal(p["lam"], q["lam"])
