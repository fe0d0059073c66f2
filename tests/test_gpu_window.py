"""The CSR product with the gathered vector's window in shared memory against
the CSR-stream kernel (the form forced through PEVSL_B200_STREAM_R, which is
read when a matrix is first used): the same bits."""
import numpy as np
import pytest

import pevsl_b200 as pv
from pevsl_b200.problems import random_coef_laplacian, random_sparse_symmetric

pytestmark = pytest.mark.gpu


def skewed(n):
    """The first rows long, some empty, the last ones short; not symmetric."""
    rng = np.random.default_rng(2)
    cnt = np.where(np.arange(n) < n // 50, 90, rng.integers(0, 6, n))
    ia = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int32)
    r = np.repeat(np.arange(n), cnt)
    ja = np.clip(r + rng.integers(-700, 1500, r.size), 0, n - 1)
    o = np.lexsort((ja, r))
    return n, ia, ja[o].astype(np.int32), rng.standard_normal(r.size)


MATRICES = {
    "smallest": lambda: random_sparse_symmetric(9473, 12, 40, 1), "diagonal": lambda: (20001, np.arange(20002, dtype=np.int32), np.arange(20001, dtype=np.int32), np.cos(np.arange(20001.0))),
    "band31": lambda: random_sparse_symmetric(15013, 10, 31, 2), "band5000": lambda: random_sparse_symmetric(40009, 16, 5000, 3),
    "two_blocks": lambda: random_sparse_symmetric(300007, 6, 11500, 4), "too_wide": lambda: random_sparse_symmetric(40011, 6, 20000, 5),
    "skewed": lambda: skewed(60000), "grid": lambda: random_coef_laplacian(41, 39, 37, 6),
}


@pytest.mark.parametrize("name", sorted(MATRICES))
def test_windowed_product_equals_stream(gpu, name, monkeypatch):
    n, ia, ja, a = MATRICES[name]()
    v = np.random.default_rng(7).standard_normal(n)
    k = np.arange(8)
    p = pv.Filter(1, 7, 0.0, 0.5, 3.0, 40.0, np.cos(0.7 * k) / (1.0 + 0.1 * k))
    out = []
    for form in ("1", "3"):
        monkeypatch.setenv("PEVSL_B200_STREAM_R", form)
        M = pv.Matrix.from_csr(n, ia, ja, a)
        with pv.Instance(M) as ev:
            out.append((M.matvec(v), ev.chebav(p, v)))
        M.free()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
