"""The CSR product with the entries loaded ahead of the wait for the degree
before, against the CSR-stream kernel (forms 4 and 1 of PEVSL_B200_STREAM_R,
which is read when a matrix is first used): the same bits.
"""
import numpy as np
import pytest

import pevsl_b200 as pv
from pevsl_b200.problems import random_sparse_symmetric

pytestmark = pytest.mark.gpu


def uneven(n, seed=3):
    """Rows of 0 to 60 entries, so that 32 of them need one or two passes of 640; values of any size."""
    rng = np.random.default_rng(seed)
    cnt = np.where(np.arange(n) % 97 < 40, rng.integers(0, 61, n), rng.integers(0, 12, n))
    ia = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int32)
    r = np.repeat(np.arange(n), cnt)
    ja = np.clip(r + rng.integers(-3000, 3001, r.size), 0, n - 1)
    o = np.lexsort((ja, r))
    return n, ia, ja[o].astype(np.int32), rng.standard_normal(r.size) * 10.0 ** rng.integers(-3, 4, r.size)


MATRICES = {
    "smallest": lambda: random_sparse_symmetric(4097, 12, 40, 1), "tail": lambda: random_sparse_symmetric(20031, 16, 5000, 2),
    "rule": lambda: random_sparse_symmetric(40009, 16, 9000, 3), "uneven": lambda: uneven(30001),
    "large": lambda: random_sparse_symmetric(150001, 16, 5000, 4),
}


@pytest.mark.parametrize("name", sorted(MATRICES))
def test_entries_ahead_equal_stream(gpu, name, monkeypatch):
    n, ia, ja, a = MATRICES[name]()
    v = np.random.default_rng(7).standard_normal(n)
    k = np.arange(10)
    p = pv.Filter(1, 9, 0.0, 0.5, 3.0, 40.0, np.cos(0.7 * k) / (1.0 + 0.1 * k))
    out = []
    for form in ("1", "4", None):
        if form:
            monkeypatch.setenv("PEVSL_B200_STREAM_R", form)
        else:
            monkeypatch.delenv("PEVSL_B200_STREAM_R")
        M = pv.Matrix.from_csr(n, ia, ja, a)
        with pv.Instance(M) as ev:
            out.append((M.matvec(v), ev.chebav(p, v)))
        M.free()
    for got in out[1:]:
        assert np.array_equal(out[0][0], got[0]) and np.array_equal(out[0][1], got[1])
