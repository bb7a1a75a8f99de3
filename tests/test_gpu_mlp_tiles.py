"""The training gradient at the edges of its 64-sample tiles: one sample, a tile less and more one,
and more tiles than blocks (a block's second tile, partly filled); and that it does not depend on
the order of execution.  Against the CPU restatement, relative to the largest entry of each parameter
block: 5e-3 as in the other gradient test, which averages over many samples; with few, a hidden
value and a pre-activation gradient that FP32 accumulation moves across a BF16 boundary change
their own products by 2^-8 each, so 1e-2."""
import numpy as np
import pytest

from forestfv_public_gb300.indicator import Indicator
from oracle import mlp
from test_gpu_mlp import BLOCKS, data, random_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 63, 64, 65, 152 * 64 + 65])
def test_gradient_at_tile_edges(B, built_lib):
    rng = np.random.default_rng(100 + B)
    ind = Indicator(seed=5)
    P = random_params(rng)
    ind.set_params(P)
    Xf, X, y, yd = data(rng, B)
    g, loss = ind.grad(X, yd)
    again, loss2 = ind.grad(X, yd)
    assert np.array_equal(g, again) and loss == loss2
    lref, gref = mlp.loss_and_grad(P.astype(np.float64), Xf, y)
    assert abs(loss - lref) <= 1e-3 * max(1.0, lref)
    tol = 1e-2 if B < 1000 else 5e-3
    for a, b in BLOCKS:
        err = np.abs(g[a:b] - gref[a:b]).max() / np.abs(gref[a:b]).max()
        assert err < tol, (a, b, err)
    ind.close()


def test_training_is_reproducible(built_lib):
    rng = np.random.default_rng(3)
    P = random_params(rng)
    _, X, _, yd = data(rng, 5000)
    runs = []
    for _ in range(2):
        ind = Indicator(seed=5)
        ind.set_params(P)
        losses = ind.train(X, yd, steps=7, batch=777, wd=1e-2, seed=9)
        runs.append((losses, ind.params()))
        more = ind.train(X, yd, steps=3, batch=64, seed=9, record_loss=False)
        assert more.shape == (3,)
        ind.close()
    assert np.array_equal(runs[0][0], runs[1][0]) and np.array_equal(runs[0][1], runs[1][1])
    assert np.isfinite(runs[0][0]).all()
