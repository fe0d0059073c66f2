"""The doubled KPM moments are no further off than the plain recurrence's.

Both against moments in long double with the same start vectors and the same
double constants: the library's (c_2k from <v_k, v_k>) and the plain recurrence
in numpy doubles (c_k = <v_k, v_0>).  The mean moments' errors past the tenth
(before, the rounding of the start vectors' norms shows) are averages of many
roundings, so the two sides' root mean squares are compared: the library's at
most 1.5 times the plain one's.  Rounding the rows' sums in doubled moments
gives 1.5 (general coefficients) to 7 times (powers of two).
"""
import numpy as np
import pytest

import pevsl_b200 as pv
from pevsl_b200.problems import laplacian

pytestmark = pytest.mark.gpu


def moments(grid, scale, V, mdeg, ctr, wid, dtype):
    """sum over the columns of <v_k, v_0>, k = 1..mdeg, of scale * Laplacian"""
    V = V.astype(dtype)
    shape = grid[::-1] + (V.shape[1],)
    d = dtype(scale * 2.0 * sum(g > 1 for g in grid))
    o = dtype(-scale)

    def apply(x):
        x = x.reshape(shape)
        y = d * x
        for ax in range(3):
            lo = tuple(slice(None, -1) if i == ax else slice(None) for i in range(4))
            hi = tuple(slice(1, None) if i == ax else slice(None) for i in range(4))
            y[lo] += o * x[hi]
            y[hi] += o * x[lo]
        return y.reshape(V.shape)

    out, vm, vk = [], None, V
    for k in range(mdeg):
        sc = dtype(np.float64(1.0 if k == 0 else 2.0) / np.float64(wid))
        w = (apply(vk) - dtype(ctr) * vk) * sc
        vm, vk = vk, w if vm is None else w - vm
        out.append(float((vk * V).sum(dtype=dtype)) if dtype is np.float64 else (vk * V).sum())
    return np.array(out)


@pytest.mark.parametrize("grid,scale,lmax", [((33, 32, 31), 1.0, 12.0), ((33, 32, 31), 0.37, 4.5), ((100, 101, 1), 0.7, 7.1)])
def test_error_is_not_above_the_plain_recurrence(gpu, grid, scale, lmax):
    n, ia, ja, a = laplacian(*grid)
    if grid[2] == 1:  # the library's 2D Laplacian has the diagonal 4
        assert a.max() == 4.0
    nvec, mdeg = 4, 300
    M = pv.Matrix.from_csr(n, ia, ja, scale * a)
    with pv.Instance(M) as ev:
        pv.set_rng(pv.RNG_GAUSS, 13)
        V = np.empty((n, nvec))
        for c in range(nvec):
            x = pv.Vector(n)
            ev.lib.pEVSL_ParvecRand(x.pv)
            V[:, c] = x.get()
        pv.set_rng(pv.RNG_GAUSS, 13)
        st, mu, _ = ev.kpmdos(mdeg, 0, nvec, [0.1, lmax - 0.1, 0.0, lmax])
    M.free()
    assert st == 0
    V = V * (1.0 / np.sqrt((V.astype(np.longdouble) ** 2).sum(0).astype(float)))
    ctr, wid = lmax / 2, lmax / 2
    exact = moments(grid, scale, V, mdeg, ctr, wid, np.longdouble)
    got = mu[1:].astype(np.longdouble) * (nvec * np.pi) / 2
    plain = moments(grid, scale, V, mdeg, ctr, wid, np.float64).astype(np.longdouble)
    err = [float(np.sqrt(np.mean((m - exact)[10:] ** 2))) for m in (got, plain)]
    assert err[0] <= 1.5 * err[1], err
