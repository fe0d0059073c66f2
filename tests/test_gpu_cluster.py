"""The one-launch filter of small problems (a thread-block cluster per vector)
against the launch-per-degree recurrence: the same bits, since both form a
row's products unfused, add them in entry order and share the recurrence's
rounding.  The other side is the same matrix behind a user matvec, which
takes the SpMV and the vector update as separate launches.
"""
import ctypes as C

import numpy as np
import pytest

import pevsl_b200 as pv
from pevsl_b200.problems import laplacian, random_sparse_symmetric

pytestmark = pytest.mark.gpu


def arrow(n):
    """Diagonal, first row and last column dense: every window spans all."""
    rows, cols = np.arange(n), np.arange(n)
    i = np.concatenate([rows, np.zeros(n - 1, int), np.arange(1, n)])
    j = np.concatenate([cols, np.arange(1, n), np.zeros(n - 1, int)])
    v = np.concatenate([2.0 + rows % 3, np.full(2 * (n - 1), 0.01)])
    o = np.lexsort((j, i))
    ia = np.concatenate([[0], np.cumsum(np.bincount(i, minlength=n))]).astype(np.int32)
    return n, ia, j[o].astype(np.int32), v[o]


def empty_rows(n):
    """Every third row without entries (and so no diagonal there)."""
    keep = np.arange(n) % 3 != 1
    ia = np.concatenate([[0], np.cumsum(keep)]).astype(np.int32)
    r = np.arange(n)[keep]
    return n, ia, ((r * 7 + 3) % n).astype(np.int32), 1.0 + 0.25 * (r % 5)


MATRICES = {
    "n1": lambda: laplacian(1, 1, 1), "n31": lambda: laplacian(31, 1, 1), "n33": lambda: laplacian(33, 1, 1),
    "n511": lambda: laplacian(73, 7, 1), "n513": lambda: laplacian(27, 19, 1), "n1025": lambda: laplacian(41, 25, 1),
    "n8191": lambda: laplacian(8191, 1, 1), "n8193": lambda: laplacian(2731, 3, 1),
    "3d": lambda: laplacian(19, 20, 21), "3d_two_rows": lambda: laplacian(26, 25, 24),
    "3d_largest": lambda: laplacian(31, 32, 33), "2d": lambda: laplacian(180, 181, 1),
    "above": lambda: laplacian(32769, 1, 1),
    "random": lambda: random_sparse_symmetric(3001, 16, 200, 5), "random_wide": lambda: random_sparse_symmetric(6007, 10, 900, 6),
    "arrow": lambda: arrow(301), "empty": lambda: empty_rows(1000),
}


def poly(deg, cc, dd):
    k = np.arange(deg + 1)
    return pv.Filter(1, deg, 0.0, 0.5, cc, dd, np.cos(0.7 * k) / (1.0 + 0.1 * k))


def both(M, apply):
    """apply(instance) with the built-in matrix and behind a user matvec."""
    lib = pv.load()
    cb = pv.MVFUNC(lambda x, y, data: lib.pEVSL_ParcsrMatvec0(x, y, C.cast(C.byref(M.A), C.c_void_p)))
    with pv.Instance(M) as ev:
        a = apply(ev)
    with pv.Instance(M) as ev:
        lib.pEVSL_SetAMatvec(ev.p, cb, None)
        b = apply(ev)
    return a, b


@pytest.mark.parametrize("name", sorted(MATRICES))
@pytest.mark.parametrize("deg", [1, 2, 37])
def test_filter_equals_launch_per_degree(gpu, name, deg):
    n, ia, ja, a = MATRICES[name]()
    M = pv.Matrix.from_csr(n, ia, ja, a)
    v = np.random.default_rng(3).standard_normal(n)
    got, want = both(M, lambda ev: ev.chebav(poly(deg, 5.0, 7.5), v))
    M.free()
    assert np.array_equal(got, want)


@pytest.mark.parametrize("grid", [(5, 4, 3), (13, 11, 1), (20, 19, 21), (26, 25, 27)])
@pytest.mark.parametrize("deg", [1, 9])
def test_generalized_filter_equals_launch_per_degree(gpu, grid, deg):
    n, ia, ja, a = laplacian(*grid)
    M = pv.Matrix.from_csr(n, ia, ja, a)
    B = pv.Matrix.from_csr(*laplacian(n, 1, 1)[:3], np.where(laplacian(n, 1, 1)[3] > 0, 4.0, -1.0))
    S = pv.BSolver(B, "lsrec", 2.0, 6.0, 40, 1e-8)
    v = np.random.default_rng(4).standard_normal(n)

    def apply(ev):
        lib = ev.lib
        lib.pEVSL_SetBParcsr(ev.p, C.byref(B.A))
        lib.pEVSL_SetBSol(ev.p, S.func, S.h)
        lib.pEVSL_SetGenEig(ev.p)
        pol, keep = pv._polparams(poly(deg, 3.0, 3.5))
        x, y = pv.Vector(n, v), pv.Vector(n)
        assert lib.pEVSL_B200_ChebAvGen(ev.p, C.byref(pol), x.pv.data, y.pv.data) == 0
        return y.get()

    got, want = both(M, apply)
    S.free()
    B.free()
    M.free()
    assert np.array_equal(got, want)


def test_one_vector_in_place(gpu):
    """y may be x: every block has read x before any block writes y."""
    n, ia, ja, a = laplacian(20, 21, 22)
    M = pv.Matrix.from_csr(n, ia, ja, a)
    v = np.random.default_rng(5).standard_normal(n)
    with pv.Instance(M) as ev:
        for deg in (1, 2, 11):
            pol, keep = pv._polparams(poly(deg, 6.0, 6.0))
            x = pv.Vector(n, v)
            assert ev.lib.pEVSL_B200_ChebAv(ev.p, C.byref(pol), x.pv.data, x.pv.data) == 0
            assert np.array_equal(x.get(), ev.chebav(poly(deg, 6.0, 6.0), v))
    M.free()


def test_many_slices_of_several_matrices_fp32_and_fp64(gpu):
    """More jobs than clusters run at a time, on matrices of different shapes,
    against the persistent form (which shares no code with the cluster's)."""
    grids = [(9, 10, 11), (40, 41, 1), (20, 19, 18)]
    mats = [pv.Matrix.from_csr(*laplacian(*g)) for g in grids]
    lib = pv.load()
    for precision in (pv.PREC_FP64, pv.PREC_MIXED):
        outs = []
        for form in (2, 1):
            lib.pEVSL_B200_SetFilterForm(form)
            evs, probs = [], []
            for M, g in zip(mats, grids):
                top = 12.0 if g[2] > 1 else 8.0
                edges = np.linspace(0.3, 0.3 + 0.02 * top, 7)
                ev = pv.Instance(M)
                ev.set_precision(precision)
                ivs = [[edges[i], edges[i + 1], 0.0, top] for i in range(6)]
                evs.append(ev)
                probs.append((ev, ivs, [60] * 6, 1e-8, np.cos(0.3 * np.arange(M.n)),
                              [pv.findpol(iv)[1] for iv in ivs]))
            st, out = pv.cheblannr_multi(probs)
            outs.append((st, out))
            for ev in evs:
                ev.close()
        lib.pEVSL_B200_SetFilterForm(-1)
        assert outs[0][0] == outs[1][0] == 0
        for p, q in zip(outs[0][1], outs[1][1]):
            for s, t in zip(p, q):
                assert s["its"] == t["its"] and np.array_equal(s["lam"], t["lam"])
    for M in mats:
        M.free()
