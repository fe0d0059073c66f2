"""Lanczos breakdowns behind a user operator.

The bounds and the Lanczos DOS queue the built-in operator's steps ahead of
their breakdown tests; a user operator is called once per step that counts,
on that step's normalised vector.  Diagonal matrices of few distinct values
break down after as many steps.
"""
import ctypes as C

import numpy as np
import pytest

import pevsl_b200 as pv

pytestmark = pytest.mark.gpu


def diagonal(n, distinct):
    ia = np.arange(n + 1, dtype=np.int32)
    return n, ia, np.arange(n, dtype=np.int32), 1.0 + (np.arange(n) % distinct)


class Operator:
    """M behind a callback that looks at every vector it is given."""

    def __init__(self, M):
        lib = pv.load()
        self.norms = []

        def call(x, y, data):
            h = np.empty(M.n)
            assert lib.pEVSL_B200_Memcpy(h.ctypes.data, x, h.nbytes) == 0
            self.norms.append(float(np.linalg.norm(h)))
            lib.pEVSL_ParcsrMatvec0(x, y, C.cast(C.byref(M.A), C.c_void_p))

        self.cb = pv.MVFUNC(call)

    def install(self, ev):
        ev.lib.pEVSL_SetAMatvec(ev.p, self.cb, None)


def products(ev):
    """the statistic n_mvA: 17 doubles come before it"""
    return C.cast(ev.p.contents.stats + 17 * 8, C.POINTER(C.c_size_t))[0]


def unit(norms):
    return all(np.isfinite(v) and abs(v - 1.0) < 1e-8 for v in norms)


@pytest.mark.parametrize("n,distinct,msteps,nvec", [(600, 3, 12, 5), (40, 7, 60, 18), (1000, 200, 20, 4)])
def test_lanczos_dos(gpu, n, distinct, msteps, nvec):
    M = pv.Matrix.from_csr(*diagonal(n, distinct))
    intv = [0.5, distinct + 0.5, 0.0, distinct + 1.0]
    outs, counts = [], []
    op = Operator(M)
    for user in (False, True):
        with pv.Instance(M) as ev:
            if user:
                op.install(ev)
            ev.lib.pEVSL_StatsReset(ev.p)
            pv.set_rng(pv.RNG_GAUSS, 7)
            outs.append(ev.landos(nvec, msteps, 51, intv))
            counts.append(products(ev))
    M.free()
    assert outs[0][0] == outs[1][0] == 0
    assert unit(op.norms) and len(op.norms) == nvec * min(msteps, n)
    assert counts == [nvec * min(msteps, n)] * 2
    assert np.array_equal(outs[0][2], outs[1][2]) and outs[0][3] == outs[1][3]


def test_lanczos_dos_of_a_tiny_problem_runs_once(gpu):
    """As many steps as rows: every run breaks down at the last, so none is
    queued ahead only to be repeated."""
    M = pv.Matrix.from_csr(*diagonal(30, 30))
    op, launches = Operator(M), []
    lib = pv.load()
    for user in (False, True):
        with pv.Instance(M) as ev:
            if user:
                op.install(ev)
            pv.set_rng(pv.RNG_GAUSS, 7)
            first = lib.pEVSL_B200_LaunchCount()
            assert ev.landos(18, 40, 51, [0.5, 30.5, 0.0, 31.0])[0] == 0
            launches.append(lib.pEVSL_B200_LaunchCount() - first)
    M.free()
    assert launches[0] <= launches[1]


@pytest.mark.parametrize("n,distinct,lanm,maxit", [(600, 3, 20, 40), (30, 30, 30, 60), (500, 5, 4, 30)])
def test_bounds(gpu, n, distinct, lanm, maxit):
    M = pv.Matrix.from_csr(*diagonal(n, distinct))
    x0 = np.random.default_rng(1).standard_normal(n)
    outs, counts = [], []
    op = Operator(M)
    for user in (False, True):
        with pv.Instance(M) as ev:
            if user:
                op.install(ev)
            ev.lib.pEVSL_StatsReset(ev.p)
            pv.set_rng(pv.RNG_GAUSS, 3)
            outs.append(ev.lantrbounds(lanm, maxit, 1e-8, x0))
            counts.append(products(ev))
    M.free()
    assert outs[0] == outs[1]  # the status too: four basis vectors are reported as too few
    assert unit(op.norms)
    assert counts[0] == counts[1] == len(op.norms) <= maxit
