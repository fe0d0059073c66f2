"""Groups of slices of several problems as parallel branches of one captured
filter application: each slice has the bits of its own run.
"""
import numpy as np
import pytest

import pevsl_b200 as pv
from pevsl_b200.problems import laplacian

pytestmark = pytest.mark.gpu

SETS = {
    "two": [((31, 30, 29), 2), ((181, 183, 1), 3)],
    "more_than_branches": [((27, 26, 25), 2), ((28, 27, 26), 3), ((131, 133, 1), 2), ((29, 27, 26), 5), ((30, 28, 27), 2)],
    "cluster_and_single": [((12, 11, 10), 2), ((31, 30, 29), 1), ((28, 29, 30), 2), ((33, 31, 17), 4)],
    "groups_of_one_matrix": [((31, 30, 29), 19), ((27, 29, 28), 2)],
}


@pytest.mark.parametrize("name", sorted(SETS))
def test_branches_equal_one_by_one(gpu, name):
    probs, mats = [], []
    for p, (grid, slices) in enumerate(SETS[name]):
        M = pv.Matrix.from_csr(*laplacian(*grid))
        top = 12.0 if grid[2] > 1 else 8.0
        edges = np.linspace(1.0, 1.0 + 0.4 * slices, slices + 1)
        ivs = [[edges[i], edges[i + 1], 0.0, top] for i in range(slices)]
        fl = [pv.findpol(iv, deg_in=18 + 2 * i + p)[1] for i, iv in enumerate(ivs)]
        mats.append(M)
        # slices of different lengths, so that the set of live ones changes
        its = [20 + 7 * ((i + p) % 3) for i in range(slices)]
        probs.append((pv.Instance(M), ivs, its, 1e3, np.cos(0.3 * np.arange(M.n) + p), fl))
    st, out = pv.cheblannr_multi(probs)
    assert st == 0
    for p, (ev, ivs, its, tol, v, fl) in enumerate(probs):
        for s in sorted({0, 1, len(ivs) - 1} & set(range(len(ivs)))):
            one = ev.cheblannr(ivs[s], its[s], tol, v, fl[s])
            assert one["nev"] == out[p][s]["nev"] and np.array_equal(one["lam"], out[p][s]["lam"])
    for p in probs:
        p[0].close()
    for M in mats:
        M.free()
