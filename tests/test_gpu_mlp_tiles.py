"""The network's products at the edges of their 32 x 32 tiles and of the 320
k values staged at once (batches and layer sizes just below, at and above),
against the CPU oracle.  Tolerances as in test_gpu_learned.py: the loss to
1e-4, outputs and gradients per layer to 1e-2 in relative 2-norm."""
import os
import sys

import numpy as np
import pytest

import pevsl_b200 as pv

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "oracle"))
import mlp_oracle as mo  # noqa: E402

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-30))


@pytest.mark.parametrize("nin,width,nout,layers", [(1, 1, 1, 2), (16, 32, 17, 2), (33, 320, 30, 3), (320, 47, 321, 2), (336, 330, 9, 3)])
@pytest.mark.parametrize("B", [1, 31, 32, 33, 320, 321, 641])
def test_products_at_tile_edges(gpu, nin, width, nout, layers, B):
    lay = mo.Layout(nin, width, nout, layers)
    p = lay.init(3)
    rng = np.random.default_rng(B)
    X, T = rng.normal(size=(B, nin)).astype(np.float32), rng.normal(size=(B, nout)).astype(np.float32)
    net = pv.Mlp(nin, width, nout, layers)
    net.set_params(p)
    Xm, Tm, Ym = pv.ManagedArray((B, nin)).set(X), pv.ManagedArray((B, nout)).set(T), pv.ManagedArray((B, nout))
    net.forward(Xm, Ym, B)
    loss, g = net.gradients(Xm, Tm, B)
    loss_o, g_o = mo.loss_grad(lay, p, X, T)
    assert rel(Ym.get(), mo.forward(lay, p, X)[0]) <= 1e-2
    assert abs(loss - loss_o) <= 1e-4 * loss_o
    for l in range(layers):
        w, b = slice(lay.woff[l], lay.woff[l] + lay.k[l] * lay.n[l]), slice(lay.boff[l], lay.boff[l] + lay.n[l])
        assert rel(g[w], g_o[w]) <= 1e-2 and rel(g[b], g_o[b]) <= 1e-2, l
    net.close()
