"""Gradient sums whose largest activations and errors fall on different
samples, and of which most cancel, against FP64 sums of the same products.

The first two layers copy features (weights 0 and 1) and the last one is
zero, so h2 and dy are exact floats and W3's gradient is the sum of their
products and nothing else.  Bounds: the result's rounding to a float (2^-24)
with room for one unit, and 2^-40 of the products' magnitudes for the sum
(pairs of floats over runs of some hundred products, measured at 2^-41)."""
import numpy as np
import pytest

from oracle import mlp as omlp

pytestmark = pytest.mark.gpu


def _copying():
    d = {name: np.zeros(shape) for name, shape in omlp.SIZES}
    d["scale"][:] = 1
    for j in range(32):
        d["W1"][j % 12, j] = 1
        d["W2"][j, j] = 1
    return omlp.pack(d).astype(np.float32)


@pytest.mark.parametrize("outlier", [1.0, 3e3, 1e6, 1e12])
@pytest.mark.parametrize("n", [64, 128, 1024, 65536])
def test_sums_with_outliers(ctx, n, outlier):
    rng = np.random.default_rng(n)
    x = rng.uniform(0.5, 2, (n, 12)).astype(np.float32)
    t = rng.normal(0, 1, (n, 6)).astype(np.float32)
    # each half of a tile cancels to 2^-18 of its products but for the samples below
    for at in range(0, n, 64):
        x[at + 32:at + 64] = x[at:at + 32]
        t[at + 32:at + 64] = -t[at:at + 32] * np.float32(1 - 2.0 ** -18)
    for at in range(0, n, 64):  # outliers meet zeros
        x[at + 5] *= np.float32(outlier)
        t[at + 5] = 0
        t[at + 40] *= np.float32(outlier)
        x[at + 40] = 0
    m = np.zeros((n, 6), np.float32)
    m[:, :4] = 1  # a power of two: dy = -2 t / sum(m) is exact
    g = omlp.unpack(ctx.mlp_loss_grad(_copying(), x, t, m)[1])
    h2 = x[:, np.arange(32) % 12].astype(np.float64)
    dy = -2.0 * m * t.astype(np.float64) / (4 * n)
    want, size = h2.T @ dy, h2.T @ np.abs(dy)
    assert np.all(np.abs(g["W3"] - want) <= 2.0 ** -23 * np.abs(want) + 2.0 ** -40 * size)
    b3 = dy.sum(0)
    assert np.all(np.abs(g["b3"] - b3) <= 2.0 ** -23 * np.abs(b3) + 2.0 ** -50 * np.abs(dy).sum(0))
