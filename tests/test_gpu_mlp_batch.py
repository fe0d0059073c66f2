"""Batches beyond 65535 tiles of 32 rows: the last rows of a forward pass have
the bits that they have alone."""
import numpy as np
import pytest

import pevsl_b200 as pv

pytestmark = pytest.mark.gpu


def test_batch_of_more_than_65535_row_tiles(gpu):
    B, nin, nout = 65535 * 32 + 37, 5, 3
    net = pv.Mlp(nin, 16, nout, 2)
    rng = np.random.default_rng(2)
    net.set_params(rng.normal(size=net.np).astype(np.float32) * 0.3)
    X = rng.normal(size=(B, nin)).astype(np.float32)
    Xm, Ym = pv.ManagedArray((B, nin)).set(X), pv.ManagedArray((B, nout))
    net.forward(Xm, Ym, B)
    m = 1000
    Xt, Yt = pv.ManagedArray((m, nin)).set(X[-m:]), pv.ManagedArray((m, nout))
    net.forward(Xt, Yt, m)
    assert np.array_equal(Ym.get()[-m:], Yt.get()) and np.all(np.isfinite(Yt.get()))
    net.close()
