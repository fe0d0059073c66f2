"""The bounds of a matrix times a power of two are the bounds times it, to the
bit, also where the squares of the projected matrix would overflow or vanish
(the Lanczos vectors' own sums of squares stay inside the range)."""
import numpy as np
import pytest

import pevsl_b200 as pv
from pevsl_b200.problems import laplacian

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exponent", [509, 200, -200, -505])
@pytest.mark.parametrize("lanm", [15, 50, 51])
def test_bounds_scale(gpu, exponent, lanm):
    n, ia, ja, a = laplacian(13, 12, 11)
    x0 = np.random.default_rng(3).standard_normal(n)
    out = []
    for s in (1.0, 2.0 ** exponent):
        M = pv.Matrix.from_csr(n, ia, ja, a * s)
        with pv.Instance(M) as ev:
            st, lo, hi = ev.lantrbounds(lanm, 400, 1e-8, x0)
        M.free()
        out.append((st, lo / s, hi / s))
    assert out[0] == out[1] and out[0][0] == 0
