"""The Lanczos steps queued without host synchronisation (bounds, Lanczos DOS)
and the kernels under them.

* A Lanczos DOS of several vectors runs them in lockstep; its sum equals the
  sum of one-vector calls on the same random stream.  Each vector's
  contribution is the same bits, so the sums differ by the rounding of
  scaling and of at most nvec additions: nvec eps of the sum.  With msteps
  above the number of distinct eigenvalues a run breaks down and restarts
  from the next random vector, which shifts the later vectors' draws.
* Projections and narrow products against numpy: sums of n (k) products of
  values below 6, error below n (k) eps times the sum of magnitudes.
"""
import ctypes as C

import numpy as np
import pytest

import pevsl_b200 as pv
from pevsl_b200.problems import laplacian, random_sparse_symmetric

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


@pytest.mark.parametrize("rng", [pv.RNG_GAUSS, pv.RNG_GLIBC])
@pytest.mark.parametrize("matrix,msteps,nvec", [
    ((20, 19, 18), 30, 1), ((20, 19, 18), 30, 2), ((33, 31, 1), 25, 16), ((33, 31, 1), 25, 17), ("random", 20, 5),
    ((3, 3, 1), 9, 5), ((2, 2, 2), 8, 18), ((4, 4, 4), 40, 7)])
def test_lanczos_dos_in_lockstep_equals_one_by_one(gpu, matrix, msteps, nvec, rng):
    L = random_sparse_symmetric(2003, 12, 100, 2) if matrix == "random" else laplacian(*matrix)
    intv = [0.5, 6.0, -20.0, 30.0] if matrix == "random" else [0.5, 6.0, 0.0, 12.0]
    M = pv.Matrix.from_csr(*L)
    with pv.Instance(M) as ev:
        pv.set_rng(rng, 5)
        st, xd, yd, count = ev.landos(nvec, msteps, 101, intv)
        draws = ev.lib.pEVSL_B200_RngDraws()
        pv.set_rng(rng, 5)
        y, c = np.zeros(101), 0.0
        for _ in range(nvec):
            s1, _, y1, c1 = ev.landos(1, msteps, 101, intv)
            assert s1 == 0
            y, c = y + y1, c + c1
        assert ev.lib.pEVSL_B200_RngDraws() == draws
    M.free()
    assert st == 0
    assert np.max(np.abs(yd - y / nvec)) <= 2 * (nvec + 2) * EPS * max(np.max(np.abs(yd)), 1e-300)
    assert abs(count - c / nvec) <= 2 * (nvec + 2) * EPS * 101 * max(abs(count), 1e-300)


@pytest.mark.parametrize("grid,lanm,maxit", [((5, 4, 3), 60, 200), ((3, 3, 1), 9, 50), ((2, 2, 2), 8, 8), ((30, 31, 29), 30, 150)])
def test_bounds_enclose_the_spectrum(gpu, grid, lanm, maxit):
    """Small problems break down inside a cycle, whose queued steps are dropped."""
    M = pv.Matrix.from_csr(*laplacian(*grid))
    ev_all = sum(np.ix_(*[4 * np.sin(np.arange(1, m + 1) * np.pi / (2 * (m + 1))) ** 2 for m in grid if m > 1]))
    with pv.Instance(M) as ev:
        pv.set_rng(pv.RNG_GAUSS, 3)
        st, lo, hi = ev.lantrbounds(lanm, maxit, 1e-8, np.random.default_rng(1).standard_normal(M.n))
    M.free()
    assert st == 0 and lo <= ev_all.min() + 1e-9 and hi >= ev_all.max() - 1e-9
    if lanm >= M.n:
        assert abs(lo - ev_all.min()) < 1e-6 and abs(hi - ev_all.max()) < 1e-6


@pytest.mark.parametrize("n", [1, 31, 255, 257, 1025, 65537])
@pytest.mark.parametrize("k", [1, 7, 8, 9, 31, 33, 65])
def test_projection_against_numpy(gpu, n, k):
    rng = np.random.default_rng(n + k)
    lib, V, x = pv.load(), rng.uniform(-1, 1, (k, n)), rng.uniform(-1, 1, n)
    P = pv.Parvecs()
    lib.pEVSL_ParvecsCreate(n, k, n, n, 0, 1, C.byref(P))
    assert lib.pEVSL_B200_Memcpy(P.data, V.ctypes.data, V.nbytes) == 0
    xv, yv = pv.Vector(n, x), pv.Vector(n, np.full(n, 0.5))
    w, c = np.zeros(k), rng.uniform(-1, 1, k)
    lib.pEVSL_ParvecsGemtv(1.0, C.byref(P), k, C.byref(xv.pv), 0.0, w.ctypes.data_as(C.POINTER(C.c_double)))
    lib.pEVSL_ParvecsGemv(-2.0, C.byref(P), k, c.ctypes.data_as(C.POINTER(C.c_double)), 3.0, C.byref(yv.pv))
    assert np.all(np.abs(w - V @ x) <= n * EPS * (np.abs(V) @ np.abs(x)) + 1e-300)
    assert np.all(np.abs(yv.get() - (1.5 - 2.0 * c @ V)) <= (k + 4) * EPS * (1.5 + 2.0 * np.abs(c) @ np.abs(V)))
    lib.pEVSL_ParvecsFree(C.byref(P))


@pytest.mark.parametrize("n,k", [(1, 1), (255, 8), (257, 15), (1000, 1024), (777, 1025), (300, 2050)])
@pytest.mark.parametrize("m", [1, 2, 3, 4, 5])
def test_narrow_product_against_numpy(gpu, n, k, m):
    import torch
    lib = pv.load()
    lib.pEVSL_B200_GemmNN.argtypes = [C.c_long, C.c_int, C.c_int] + [C.c_void_p, C.c_long] * 3
    g = torch.Generator().manual_seed(n + k + m)
    V, Y = (torch.rand(r, c, generator=g, dtype=torch.float64) - 0.5 for r, c in ((k, n + 3), (m, k + 2)))
    Vd, Yd, U = V.cuda(), Y.cuda(), torch.zeros(m, n + 1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert lib.pEVSL_B200_GemmNN(n, k, m, Vd.data_ptr(), n + 3, Yd.data_ptr(), k + 2, U.data_ptr(), n + 1) == 0
    assert lib.pEVSL_B200_Sync() == 0
    want, mag = Y[:, :k] @ V[:, :n], Y[:, :k].abs() @ V[:, :n].abs()
    assert torch.all((U.cpu()[:, :n] - want).abs() <= (k + 2) * EPS * mag) and torch.all(U[:, n] == 0)
