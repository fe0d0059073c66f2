"""KPM moments from doubled recurrences (c_{2k} = 2 <v_k, v_k> - c_0, c_{2k+1} =
2 <v_{k+1}, v_k> - c_1) against the moments of the plain recurrence in long
double on the host, for the same random vectors.  Tolerance: each of the
nvec summed moments carries the rounding of a recurrence of at most Mdeg
steps with |T_k| <= 1, below Mdeg * 4 eps in the 2-norm of unit vectors; the
mean over vectors is then within Mdeg * 4 eps / pi of the exact one.
"""
import numpy as np
import pytest

import pevsl_b200 as pv
from pevsl_b200.problems import laplacian, random_sparse_symmetric

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def apply(n, ia, ja, a, X):
    prod = a[:, None].astype(np.longdouble) * X[ja]
    out = np.zeros_like(X)
    rows = np.repeat(np.arange(n), np.diff(ia))
    np.add.at(out, rows, prod)
    return out


def plain_moments(n, ia, ja, a, V, mdeg, lmin, lmax):
    V = V.astype(np.longdouble)
    V = V / np.sqrt((V * V).sum(0))
    ctr, wid = (np.longdouble(lmax) + lmin) / 2, (np.longdouble(lmax) - lmin) / 2
    k1, q = np.arange(1, mdeg + 1), np.pi / (mdeg + 2)
    jac = np.sin((k1 + 1) * q) / ((mdeg + 2) * np.sin(q)) + (1 - (k1 + 1) / (mdeg + 2)) * np.cos(k1 * q)
    vm, vk, c = None, V, []
    for k in range(mdeg):
        w = (apply(n, ia, ja, a, vk) - ctr * vk) * ((1 if k == 0 else 2) / wid)
        vm, vk = vk, w if vm is None else w - vm
        c.append((vk * V).sum())
    return np.concatenate([[V.shape[1]], 2 * jac * np.array(c)]) / (V.shape[1] * np.pi)


CASES = {
    "grid": lambda: (laplacian(7, 6, 5), 0.0, 12.0), "plane": lambda: (laplacian(31, 17, 1), 0.0, 8.0),
    "scattered": lambda: (random_sparse_symmetric(900, 12, 60, 3), -25.0, 30.0),
    "dense_rows": lambda: (random_sparse_symmetric(300, 60, 100, 4), -70.0, 80.0),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("mdeg,nvec", [(1, 1), (2, 2), (3, 5), (40, 33), (41, 64), (12, 67)])
def test_moments_against_plain_recurrence(gpu, name, mdeg, nvec):
    (n, ia, ja, a), lmin, lmax = CASES[name]()
    M = pv.Matrix.from_csr(n, ia, ja, a)
    with pv.Instance(M) as ev:
        pv.set_rng(pv.RNG_GAUSS, 11)
        V = np.empty((n, nvec))
        for c in range(nvec):
            x = pv.Vector(n)
            ev.lib.pEVSL_ParvecRand(x.pv)
            V[:, c] = x.get()
        pv.set_rng(pv.RNG_GAUSS, 11)
        st, mu, count = ev.kpmdos(mdeg, 1, nvec, [lmin + 0.1, lmax - 0.1, lmin, lmax])
    M.free()
    assert st == 0 and np.isfinite(count)
    want = plain_moments(n, ia, ja, a, V, mdeg, lmin, lmax)
    assert np.max(np.abs(mu - want)) <= mdeg * 4 * EPS / np.pi + 4 * EPS
