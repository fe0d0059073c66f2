"""The stencil form (a mask of constant (offset, value) pairs per row) against
the general CSR kernels: the same bits.  The general side is the same matrix
with decoupled diagonal rows of 40 further values appended, which leaves the
first n rows' arithmetic alone and has too many pairs for the form.
"""
import numpy as np
import pytest

import pevsl_b200 as pv
from pevsl_b200.problems import laplacian

pytestmark = pytest.mark.gpu


def banded(n, offsets, values):
    """Row i has the entries of column i + offsets[j] that exist, offsets ascending."""
    cols = np.arange(n)[:, None] + np.array(offsets)[None, :]
    keep = (cols >= 0) & (cols < n)
    ia = np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.int32)
    return n, ia, cols[keep].astype(np.int32), np.broadcast_to(np.array(values, float), cols.shape)[keep]


def with_extra_rows(n, ia, ja, a, m=40):
    return (n + m, np.concatenate([ia, ia[-1] + 1 + np.arange(m)]).astype(np.int32),
            np.concatenate([ja, n + np.arange(m)]).astype(np.int32), np.concatenate([a, 1.0 + np.arange(m) / 64.0]))


def box27(s):
    o = [dz * s * s + dy * s + dx for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1)]
    return banded(s ** 3, o, [8.0 if x == 0 else -0.25 for x in o])


MATRICES = {
    "1d": lambda: laplacian(33001, 1, 1), "2d": lambda: laplacian(129, 131, 1), "3d": lambda: laplacian(26, 25, 27),
    "3d_large": lambda: laplacian(41, 43, 42), "3d_two_rows": lambda: laplacian(97, 98, 97),
    "2d_large": lambda: laplacian(301, 299, 1), "box27": lambda: box27(33),
    "nine": lambda: banded(20011, [-144, -143, -142, -1, 0, 1, 142, 143, 144], [.5, 1, .5, 1, -6, 1, .5, 1, .25]),
    "no_diagonal": lambda: banded(20011, [-9, -5, -2, 1, 3, 4, 11], [1, 2, 3, .5, .25, 1, 2]),
    "three": lambda: banded(17003, [-3, 0, 3], [1, 2, 3]), "small": lambda: laplacian(5, 4, 3),
}


@pytest.mark.parametrize("name", sorted(MATRICES))
def test_filter_and_product_equal_the_csr_kernels(gpu, name):
    n, ia, ja, a = MATRICES[name]()
    M, G = pv.Matrix.from_csr(n, ia, ja, a), pv.Matrix.from_csr(*with_extra_rows(n, ia, ja, a))
    v = np.random.default_rng(7).standard_normal(n + 40)
    assert np.array_equal(M.matvec(v[:n]), G.matvec(v)[:n])
    with pv.Instance(M) as e, pv.Instance(G) as f:
        for deg in (1, 2, 3, 4, 5, 38):
            k = np.arange(deg + 1)
            p = pv.Filter(1, deg, 0.0, 0.5, 5.0, 7.5, np.cos(0.7 * k) / (1.0 + 0.1 * k))
            assert np.array_equal(e.chebav(p, v[:n]), f.chebav(p, v)[:n])
    M.free()
    G.free()


@pytest.mark.parametrize("kind", ["cheb1", "cheb2", "lsrec"])
def test_b_solves_equal_the_csr_kernels(gpu, kind):
    n, ia, ja, a = laplacian(35003, 1, 1)
    a = np.where(a > 0, 4.0, -1.0)
    M, G = pv.Matrix.from_csr(n, ia, ja, a), pv.Matrix.from_csr(*with_extra_rows(n, ia, ja, a))
    v = np.random.default_rng(8).standard_normal(n + 40)
    S, T = pv.BSolver(M, kind, 2.0, 6.0, 12), pv.BSolver(G, kind, 2.0, 6.0, 12)
    assert np.array_equal(S.solve(v[:n]), T.solve(v)[:n])
    for x in (S, T, M, G):
        x.free()


@pytest.mark.parametrize("grid", [(27, 26, 25), (181, 183, 1), (42, 41, 43)])
@pytest.mark.parametrize("slices", [2, 3, 7, 13])
def test_lockstep_slices_equal_one_by_one(gpu, grid, slices):
    M = pv.Matrix.from_csr(*laplacian(*grid))
    edges = np.linspace(1.0, 3.0, slices + 1)
    ivs = [[edges[i], edges[i + 1], 0.0, 12.0] for i in range(slices)]
    fl = [pv.findpol(iv, deg_in=20 + i)[1] for i, iv in enumerate(ivs)]
    v = np.cos(0.3 * np.arange(M.n))
    with pv.Instance(M) as ev:
        st, outs = pv.cheblannr_batch(ev, ivs, [40] * slices, 1e3, v, fl)
        assert st == 0
        for s in (0, slices - 1):
            one = ev.cheblannr(ivs[s], 40, 1e3, v, fl[s])
            assert one["nev"] == outs[s]["nev"] and np.array_equal(one["lam"], outs[s]["lam"])
    M.free()


def test_generalized_lockstep_equals_one_by_one(gpu):
    """Too large for a cluster: the interleaved kernel with its SpMV on B^{-1} X."""
    n, ia, ja, a = laplacian(32, 33, 34)
    M, B = pv.Matrix.from_csr(n, ia, ja, a), pv.Matrix.from_csr(n, ia, ja, np.where(a > 0, 12.0 / 18, 1.0 / 18))
    S = pv.BSolver(B, "lsrec", 1.0 / 3.0, 1.0, 30, 1e-6)
    ivs = [[1.0, 2.0, 0.0, 36.0], [2.0, 3.0, 0.0, 36.0], [3.0, 4.5, 0.0, 36.0]]
    fl = [pv.findpol(iv, deg_in=15 + i)[1] for i, iv in enumerate(ivs)]
    v = np.cos(0.3 * np.arange(n))
    with pv.Instance(M) as ev:
        ev.set_generalized(B, S)
        st, outs = pv.cheblannr_batch(ev, ivs, [35] * 3, 1e3, v, fl)
        assert st == 0
        for s in range(3):
            one = ev.cheblannr(ivs[s], 35, 1e3, v, fl[s])
            assert one["nev"] == outs[s]["nev"] and np.array_equal(one["lam"], outs[s]["lam"])
    for x in (S, B, M):
        x.free()


@pytest.mark.parametrize("grid", [(107, 108, 106), (1103, 1101, 1), (129, 130, 128), (1461, 1463, 1)])
def test_two_rows_per_thread(gpu, grid):
    """Past seven waves of blocks the degrees between the sum's first and last update take two rows per thread."""
    n, ia, ja, a = laplacian(*grid)
    M, G = pv.Matrix.from_csr(n, ia, ja, a), pv.Matrix.from_csr(*with_extra_rows(n, ia, ja, a))
    v = np.random.default_rng(9).standard_normal(n + 40)
    with pv.Instance(M) as e, pv.Instance(G) as f:
        for deg in (4, 23):
            k = np.arange(deg + 1)
            p = pv.Filter(1, deg, 0.0, 0.5, 6.0, 7.5, np.cos(0.7 * k) / (1.0 + 0.1 * k))
            assert np.array_equal(e.chebav(p, v[:n]), f.chebav(p, v)[:n])
    M.free()
    G.free()


@pytest.mark.parametrize("grid", [(68, 67, 69), (561, 563, 1)])
@pytest.mark.parametrize("slices", [2, 3])
def test_lockstep_past_one_wave(gpu, grid, slices):
    M = pv.Matrix.from_csr(*laplacian(*grid))
    edges = np.linspace(1.0, 3.0, slices + 1)
    ivs = [[edges[i], edges[i + 1], 0.0, 12.0] for i in range(slices)]
    fl = [pv.findpol(iv, deg_in=20 + i)[1] for i, iv in enumerate(ivs)]
    v = np.cos(0.3 * np.arange(M.n))
    with pv.Instance(M) as ev:
        st, outs = pv.cheblannr_batch(ev, ivs, [30] * slices, 1e3, v, fl)
        assert st == 0
        for s in range(slices):
            one = ev.cheblannr(ivs[s], 30, 1e3, v, fl[s])
            assert one["nev"] == outs[s]["nev"] and np.array_equal(one["lam"], outs[s]["lam"])
    M.free()


def without(n, ia, ja, a, drop):
    rows = np.repeat(np.arange(n), np.diff(ia))
    keep = ~drop(rows, ja)
    return n, np.concatenate([[0], np.cumsum(np.bincount(rows[keep], minlength=n))]).astype(np.int32), ja[keep], a[keep]


@pytest.mark.parametrize("name", ["no_diagonal_in_some_rows", "empty_rows", "infinite_value"])
def test_rows_that_lack_pairs(gpu, name):
    """A pair that a row lacks adds nothing: not where it is the diagonal, not
    in an empty row, and not where its value is infinite."""
    n, ia, ja, a = laplacian(41, 43, 42)
    if name == "no_diagonal_in_some_rows":
        n, ia, ja, a = without(n, ia, ja, a, lambda r, c: (r == c) & (r % 7 == 0))
    elif name == "empty_rows":
        n, ia, ja, a = without(n, ia, ja, a, lambda r, c: r % 11 == 3)
    else:
        rows = np.repeat(np.arange(n), np.diff(ia))
        a = np.where(ja == rows + 41, np.inf, a)
    M, G = pv.Matrix.from_csr(n, ia, ja, a), pv.Matrix.from_csr(*with_extra_rows(n, ia, ja, a))
    v = np.random.default_rng(10).standard_normal(n + 40)
    v[5] = -0.0
    got, want = M.matvec(v[:n]), G.matvec(v)[:n]
    assert np.array_equal(got, want, equal_nan=True) and np.array_equal(np.signbit(got), np.signbit(want))
    with pv.Instance(M) as e, pv.Instance(G) as f:
        k = np.arange(12)
        p = pv.Filter(1, 11, 0.0, 0.5, 6.0, 7.5, np.cos(0.7 * k) / (1.0 + 0.1 * k))
        assert np.array_equal(e.chebav(p, v[:n]), f.chebav(p, v)[:n], equal_nan=True)
    M.free()
    G.free()
