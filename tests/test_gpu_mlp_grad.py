"""The gradient kernel at its tile edges against the FP64 oracle.

Tiles are 128 samples in two halves of 64, over at most two CTAs per SM; the
sums run on a fixed grid unless the products are too large for it, then in
FP64.  The bound is on the per-sample float arithmetic: three layers of at
most 32 fused steps each way, under 200 roundings of 2^-24 = 1.2e-5, and
features of size `scale` leave that relative error as it is.
"""
import numpy as np
import pytest

from oracle import mlp as omlp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 65, 127, 128, 129, 40000])
@pytest.mark.parametrize("scale", [1.0, 1e-12, 1e17], ids=["unit", "tiny", "fp64"])
def test_gradient_at_tile_edges(ctx, n, scale):
    rng = np.random.default_rng(n)
    p = omlp.init(3, shift=np.zeros(12), scale=np.ones(12))
    x = (rng.normal(0, 1.5, (n, 12)) * scale).astype(np.float32)
    t = (rng.normal(0, 1, (n, 6)) * scale).astype(np.float32)
    m = (rng.random((n, 6)) < 0.6).astype(np.float32)
    m[0, 0] = 1.0
    loss, g = ctx.mlp_loss_grad(p, x, t, m)
    want_loss, want = omlp.loss_grad(p, x, t, m)
    assert abs(loss - want_loss) <= 1.2e-5 * want_loss
    assert np.all(g[:24] == 0)
    for name, part in omlp.unpack(want).items():
        got = omlp.unpack(g)[name]
        assert np.linalg.norm(got - part) <= 1.2e-5 * np.linalg.norm(part), name
