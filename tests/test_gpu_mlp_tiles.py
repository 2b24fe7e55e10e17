"""The gradient kernel where its tiles change size (16 to 128 samples, the
smallest of which there are no more than SMs): both sides of each change and
of the tiles' halves, against FP64 sums of the same products.

The first two layers copy features (weights 0 and 1) and the last one is
zero, so activations and errors are exact floats and no unit lies within a
rounding of zero.  Bounds as in test_gpu_mlp_outliers: the result's rounding
to a float with room for one unit (2^-23), and 2^-40 of the products'
magnitudes for the sums; the loss adds the three roundings of a sample's
term."""
import numpy as np
import pytest

from oracle import mlp as omlp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("more", [-1, 0, 1, 9])
@pytest.mark.parametrize("span", [1, 2, 16, 32, 64, 128, 256])
def test_sums_at_tile_sizes(ctx, span, more):
    n = span * ctx.device_info()["sm_count"] + more if span > 2 else 8 * span + more
    rng = np.random.default_rng(n)
    d = {name: np.zeros(shape) for name, shape in omlp.SIZES}
    d["scale"][:] = 1
    for j in range(32):
        d["W1"][j % 12, j] = d["W2"][j, j] = 1
    x = (rng.integers(1, 1 << 20, (n, 12)) * 2.0 ** -20).astype(np.float32)
    t = (rng.integers(-1 << 20, 1 << 20, (n, 6)) * 2.0 ** -20).astype(np.float32)
    m = np.zeros((n, 6), np.float32)
    m[:, :4] = (rng.random((n, 4)) < 0.6) * np.float32(2)
    m[0, 0] = 0
    m[0, 0] = 2.0 ** np.ceil(np.log2(m.sum() + 1)) - m.sum()  # a power of two in all
    loss, got = ctx.mlp_loss_grad(omlp.pack(d).astype(np.float32), x, t, m)
    g = omlp.unpack(got)
    h2 = x[:, np.arange(32) % 12].astype(np.float64)
    dy = -2.0 * m.astype(np.float64) * t / m.sum(dtype=np.float64)
    want, size = h2.T @ dy, h2.T @ np.abs(dy)
    assert np.all(np.abs(g["W3"] - want) <= 2.0 ** -23 * np.abs(want) + 2.0 ** -40 * size)
    assert np.all(np.abs(g["b3"] - dy.sum(0)) <= 2.0 ** -23 * np.abs(dy.sum(0)) + 2.0 ** -50 * np.abs(dy).sum(0))
    for name in ("W1", "b1", "W2", "b2"):  # no error passes the zero layer
        assert np.all(g[name] == 0)
    want_loss = float((m.astype(np.float64) * t * t).sum() / m.sum(dtype=np.float64))
    assert abs(loss - want_loss) <= 3 * 2.0 ** -24 * want_loss
    again = ctx.mlp_loss_grad(omlp.pack(d).astype(np.float32), x, t, m)
    assert again[0] == loss and np.array_equal(again[1], got)
