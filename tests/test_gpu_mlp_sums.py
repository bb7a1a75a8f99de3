"""How the training gradient is summed.  Its rounding points: the gradients of two batches of 16
samples (one tile of every product, nothing added up between tiles) against recorded ones of the
kernel that took one warp per 16 samples (tests/golden/indicator/gradient16.npz, recorded on a GB300
from its C entry ffv_mlp_grad), to the bit.

And the sum over many tiles: a batch of a million samples that repeats 1024 in order, against the mean
of the 64 gradients of 16 samples in FP64 (batch sizes are powers of two: the factor 1 / B is exact and
scales every rounded value alike).  FP32 additions rounded to nearest: an entry's longest path has at
most k = 4 * 108 (a block's tiles) + 38 (blocks) + 6 additions, each off by up to 2^-24 of the partial
sum, with a standard deviation of 0.58 of that; partial sums average 0.58 of the entries' total
magnitude: six standard deviations are 2 sqrt(k) 2^-24 = 44 * 2^-24 of it."""
import numpy as np
import pytest
import torch

from conftest import load_golden

from forestfv_public_gb300.indicator import Indicator
from test_gpu_mlp import BLOCKS, data, random_params

pytestmark = pytest.mark.gpu


def test_gradient_of_one_product_tile(built_lib):
    g = load_golden("indicator/gradient16")
    ind = Indicator(seed=5)
    for i, seed in enumerate(g["seeds"]):
        rng = np.random.default_rng(int(seed))
        ind.set_params(random_params(rng))
        _, X, _, y = data(rng, 16)
        grad, loss = ind.grad(X, y)
        for a, b in BLOCKS:
            assert np.array_equal(grad[a:b], g["grad"][i, a:b]), (int(seed), a)
        assert abs(loss - g["loss"][i]) <= 1e-6 * g["loss"][i]  # sixteen terms in another order
    ind.close()


def test_gradient_of_a_million_samples(built_lib):
    rng = np.random.default_rng(8)
    ind = Indicator(seed=5)
    ind.set_params(random_params(rng))
    _, X, _, y = data(rng, 1024)
    parts = np.stack([ind.grad(X[16 * i:16 * i + 16], y[16 * i:16 * i + 16])[0] for i in range(64)]).astype(np.float64)
    grad, _ = ind.grad(X.repeat(1024, 1), y.repeat(1024))
    ind.close()
    assert torch.cuda.get_device_properties(0).multi_processor_count >= 152  # 108 tiles a block
    off = np.abs(grad - parts.mean(0)) / np.abs(parts).mean(0)
    assert (off <= 44.0 * 2.0 ** -24).all(), [float(off[a:b].max() * 2.0 ** 24) for a, b in BLOCKS]
