"""The form that a product runs in is the one that was forced, or that the
rules choose: without this the comparisons of forms could compare one with
itself."""
import pytest

import pevsl_b200 as pv
import test_gpu_ahead
import test_gpu_stencil
import test_gpu_window
from pevsl_b200.problems import laplacian, random_sparse_symmetric

pytestmark = pytest.mark.gpu


def form_of(matrix):
    import numpy as np
    M = pv.Matrix.from_csr(*matrix)
    M.matvec(np.ones(M.n))
    form = pv.load().pEVSL_B200_ProductForm(M.A)
    M.free()
    return form


@pytest.mark.parametrize("name", sorted(test_gpu_window.MATRICES))
def test_windowed_form_runs(gpu, name, monkeypatch):
    monkeypatch.setenv("PEVSL_B200_STREAM_R", "3")
    assert form_of(test_gpu_window.MATRICES[name]()) == (1 if name == "too_wide" else 3)


@pytest.mark.parametrize("name", sorted(test_gpu_ahead.MATRICES))
def test_entries_ahead_run(gpu, name, monkeypatch):
    matrix = test_gpu_ahead.MATRICES[name]()
    monkeypatch.setenv("PEVSL_B200_STREAM_R", "4")
    assert form_of(matrix) == 4
    monkeypatch.delenv("PEVSL_B200_STREAM_R")
    # by the rule below 2^16 rows with 8 entries per row, 8 10^5 in all
    n, nnz = matrix[0], int(matrix[1][-1])
    if n < 65536 and 8 * n <= nnz <= 800000:
        assert form_of(matrix) == 4
    else:
        assert form_of(matrix) in (1, 2, 3)


@pytest.mark.parametrize("name", sorted(test_gpu_stencil.MATRICES))
def test_stencil_form_runs(gpu, name):
    matrix = test_gpu_stencil.MATRICES[name]()
    wide = name == "box27"  # more than 24 entries per row on average: several threads per row
    assert form_of(matrix) == (0 if wide else 6)


def test_other_forms(gpu):
    n, ia, ja, a = laplacian(30, 29, 28)
    assert form_of(test_gpu_stencil.with_extra_rows(n, ia, ja, a)) == 5
    assert form_of(random_sparse_symmetric(5003, 60, 300, 1)) == 0


@pytest.mark.parametrize("deg", [1, 2, 7, 8, 30])
def test_small_problems_by_degree(gpu, deg):
    """One cluster launch from degree 8 on, a launch per degree below."""
    import numpy as np
    lib = pv.load()
    M = pv.Matrix.from_csr(*laplacian(19, 20, 21))
    k = np.arange(deg + 1)
    p = pv.Filter(1, deg, 0.0, 0.5, 6.0, 7.5, np.cos(0.7 * k) / (1.0 + 0.1 * k))
    with pv.Instance(M) as ev:
        ev.chebav(p, np.ones(M.n))
        first = lib.pEVSL_B200_LaunchCount()
        ev.chebav(p, np.ones(M.n))
        assert lib.pEVSL_B200_LaunchCount() - first == (1 if deg >= 8 else deg)
    M.free()
