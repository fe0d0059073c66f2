"""Two and four lockstep slices on stencil matrices of other widths than the
compiled ones, whose pairs the interleaved kernel takes a few at a time: the
bits of one slice alone.  32 pairs are the most the form has."""
import numpy as np
import pytest

import pevsl_b200 as pv

pytestmark = pytest.mark.gpu


def banded(n, offsets, values, diagonals=1):
    """Constant bands; the diagonal cycles through `diagonals` values."""
    cols = np.arange(n)[:, None] + np.array(offsets)[None, :]
    val = np.broadcast_to(np.array(values, float), cols.shape).copy()
    if diagonals > 1:
        val[:, offsets.index(0)] += (np.arange(n) % diagonals) / 64.0
    keep = (cols >= 0) & (cols < n)
    ia = np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.int32)
    return n, ia, cols[keep].astype(np.int32), val[keep]


MATRICES = {
    "three": lambda: banded(33001, [-3, 0, 3], [-1, 4, -1]),
    "six": lambda: banded(33001, [-7, -1, 0, 1, 7], [-1, -1, 4, -1, -1], 2),
    "nine": lambda: banded(40011, [-201, -200, -199, -1, 0, 1, 199, 200, 201], [-.5, -1, -.5, -1, 6, -1, -.5, -1, -.5]),
    "thirty_one": lambda: banded(33001, [-3, 0, 3], [-1, 4, -1], 29),
    "thirty_two": lambda: banded(33001, [-3, 0, 3], [-1, 4, -1], 30),
}


@pytest.mark.parametrize("name", sorted(MATRICES))
@pytest.mark.parametrize("slices", [2, 4])
def test_lockstep_equals_one_by_one(gpu, name, slices):
    M = pv.Matrix.from_csr(*MATRICES[name]())
    edges = np.linspace(1.0, 3.0, slices + 1)
    ivs = [[edges[i], edges[i + 1], 0.0, 13.0] for i in range(slices)]
    fl = [pv.findpol(iv, deg_in=20 + i)[1] for i, iv in enumerate(ivs)]
    v = np.cos(0.3 * np.arange(M.n))
    with pv.Instance(M) as ev:
        st, outs = pv.cheblannr_batch(ev, ivs, [40] * slices, 1e3, v, fl)
        assert st == 0
        for s in (0, slices - 1):
            one = ev.cheblannr(ivs[s], 40, 1e3, v, fl[s])
            assert one["nev"] == outs[s]["nev"] and np.array_equal(one["lam"], outs[s]["lam"])
    M.free()
