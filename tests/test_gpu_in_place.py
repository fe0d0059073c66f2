"""A filter application whose result replaces its input, in each launch form:
one cluster launch, a launch per degree on a small and on a large stencil, on a
general matrix, and behind a user operator.  Repeated, since a form that wrote
rows which others still read would show only now and then."""
import ctypes as C

import numpy as np
import pytest

import pevsl_b200 as pv
from pevsl_b200.problems import laplacian, random_sparse_symmetric

pytestmark = pytest.mark.gpu

MATRICES = {"small": lambda: laplacian(20, 21, 22), "large": lambda: laplacian(64, 65, 63),
            "general": lambda: random_sparse_symmetric(70001, 12, 3000, 2), "rows": lambda: random_sparse_symmetric(20001, 40, 900, 3)}


@pytest.mark.parametrize("user", [False, True])
@pytest.mark.parametrize("name", sorted(MATRICES))
def test_result_over_input(gpu, name, user):
    n, ia, ja, a = MATRICES[name]()
    M = pv.Matrix.from_csr(n, ia, ja, a)
    lib = pv.load()
    cb = pv.MVFUNC(lambda x, y, data: lib.pEVSL_ParcsrMatvec0(x, y, C.cast(C.byref(M.A), C.c_void_p)))
    v = np.random.default_rng(5).standard_normal(n)
    with pv.Instance(M) as ev:
        if user:
            lib.pEVSL_SetAMatvec(ev.p, cb, None)
        for deg in (0, 1, 2, 3, 11):
            k = np.arange(deg + 1)
            f = pv.Filter(1, deg, 0.0, 0.5, 6.0, 30.0, np.cos(0.7 * k) / (1.0 + 0.1 * k))
            pol, keep = pv._polparams(f)
            want = ev.chebav(f, v)
            for _ in range(5):
                x = pv.Vector(n, v)
                assert lib.pEVSL_B200_ChebAv(ev.p, C.byref(pol), x.pv.data, x.pv.data) == 0
                assert np.array_equal(x.get(), want)
    M.free()
