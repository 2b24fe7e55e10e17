"""Loss and gradient sums beyond the floats' range, and infinite samples: what
the FP64 sums of the samples' floats give.

The rows' values are exact powers or whole multiples here, so the oracle's
FP64 sums differ from the kernel's by the floats' rounding (1.2e-5 as in
test_gpu_mlp_grad) and what exceeds FLT_MAX is an infinity of the sum's sign.
"""
import numpy as np
import pytest

from oracle import mlp as omlp

pytestmark = pytest.mark.gpu
BIG = float(np.finfo(np.float32).max)


def _network(last_layer):
    p = omlp.init(3, shift=np.zeros(12), scale=np.ones(12))
    d = omlp.unpack(p)
    if not last_layer:
        d["W3"] = d["W3"] * 0
    return omlp.pack(d).astype(np.float32)


def _samples(n):
    rng = np.random.default_rng(n)
    return (rng.normal(0, 1, (n, 12)).astype(np.float32), rng.normal(0, 1, (n, 6)).astype(np.float32),
            np.ones((n, 6), np.float32))


@pytest.mark.parametrize("at", [0, 63, 64, 127, 128, 299])
def test_infinite_loss_of_one_sample(ctx, at):
    x, t, m = _samples(300)
    t[at, 2] = 1e25  # e^2 exceeds FLT_MAX, 2 e does not
    p = _network(True)
    loss, g = ctx.mlp_loss_grad(p, x, t, m)
    assert loss == np.inf
    _, want = omlp.loss_grad(p, x, t, m)
    for name, part in omlp.unpack(want).items():
        assert np.linalg.norm(omlp.unpack(g)[name] - part) <= 1.2e-5 * np.linalg.norm(part), name


def test_infinite_error_of_one_sample(ctx):
    x, t, m = _samples(200)
    m[:] = 0
    m[70, 0], t[70, 0] = 1, -3e38  # 2 e exceeds FLT_MAX
    p = _network(True)
    loss, g = ctx.mlp_loss_grad(p, x, t, m)
    g = omlp.unpack(g)
    assert loss == np.inf
    assert g["b3"][0] == np.inf and np.all(g["b3"][1:] == 0)
    q = omlp.unpack(p)
    h2 = np.maximum(np.maximum(x[70] @ q["W1"], 0) @ q["W2"], 0)
    assert 0 < (h2 > 0).sum() < 32
    assert np.all(g["W3"][h2 > 0, 0] == np.inf) and np.all(np.isnan(g["W3"][h2 == 0, 0]))
    assert np.all(g["W3"][:, 1:] == 0)


@pytest.mark.parametrize("n", [1, 64, 100, 128, 1000])
def test_gradient_beyond_the_float_range(ctx, n):
    """Products of 1e20 and 1e19: every sum keeps its sign and is infinite
    or, where the samples of other tiles cancel them, finite."""
    p = _network(False)
    x, _, m = _samples(n)
    x *= np.float32(1e22)
    t = np.full((n, 6), -1e19 * n, np.float32)
    t[:, 1::2] *= -1
    _, want = omlp.loss_grad(p, x, t, m)
    want = omlp.unpack(want)["W3"]
    g = omlp.unpack(ctx.mlp_loss_grad(p, x, t, m)[1])["W3"]
    over = np.abs(want) > 1.001 * BIG
    assert over.sum() > 60
    assert np.array_equal(g[over], np.sign(want[over]) * np.inf)
    # a second half of the samples, in other tiles, with the opposite errors
    pad = -n % 128
    z = lambda a: np.concatenate([a, np.zeros((pad, a.shape[1]), np.float32)])
    g = ctx.mlp_loss_grad(p, np.concatenate([z(x), x]), np.concatenate([z(t), -t]), np.concatenate([z(m), m]))[1]
    g = omlp.unpack(g)["W3"]
    assert np.all(np.isfinite(g))
    assert np.all(np.abs(g) <= 2.0 ** -50 * n * 1e23 * 1e20)
