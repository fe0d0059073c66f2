"""Thick-restart bounds over the dimensions of the projected matrix on both
sides of the ones that its device eigensolver takes (16 to 112, odd and even).
"""
import numpy as np
import pytest

import pevsl_b200 as pv
from pevsl_b200.problems import laplacian

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bndtype", [1, 2])
@pytest.mark.parametrize("lanm", [15, 16, 17, 33, 50, 111, 112, 113])
def test_bounds_enclose_the_spectrum(gpu, lanm, bndtype):
    """Rayleigh-Ritz: the outer Ritz value lies inside the spectrum and an end
    of it within the residual t, so that lam_1 - t <= lmin = theta - t <= lam_1,
    with t below tol (|lmin| + |lmax|) at the stop; rounding of a projected
    matrix of norm 12 and dimension lanm: 12 lanm eps."""
    grid, tol = (13, 12, 11), 1e-8
    M = pv.Matrix.from_csr(*laplacian(*grid))
    ends = [4.0 * sum(np.sin(k * np.pi / (2 * (g + 1))) ** 2 for g, k in zip(grid, ks))
            for ks in ((1, 1, 1), grid)]
    with pv.Instance(M) as ev:
        st, lo, hi = ev.lantrbounds(lanm, 2000, tol, np.random.default_rng(3).standard_normal(M.n), bndtype)
    M.free()
    assert st == 0
    t, eps = tol * (abs(lo) + abs(hi)), 12.0 * lanm * np.finfo(float).eps
    assert ends[0] - t - eps <= lo <= ends[0] + eps
    assert ends[1] - eps <= hi <= ends[1] + t + eps
