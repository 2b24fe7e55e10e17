"""BC where a level pulls: unvisited hubs of one, two and many 128-arc chunks
(claimed by whichever chunk finds a parent), more groups than eight per warp,
and hubs on both sides of the peak level, against FP64 Brandes."""
import numpy as np
import pytest

import oracle
from gpu_discovery_barrier_gb300 import gdb, graphgen as gg

pytestmark = pytest.mark.gpu


def _layers(seed):
    """A source, a dense middle layer holding most arcs, then hubs of 100 to
    2,000 neighbours in it and tails behind them."""
    rng = np.random.default_rng(seed)
    mid = 3000
    pairs = [(0, 1 + i) for i in range(mid)]
    pairs += list(map(tuple, 1 + rng.integers(0, mid, (60000, 2))))
    v = 1 + mid
    for d in (100, 127, 128, 129, 130, 255, 256, 257, 700, 2000):
        hub = v
        pairs += [(hub, 1 + int(m)) for m in rng.choice(mid, d, replace=False)]
        pairs += [(hub, hub + 1), (hub + 1, hub + 2)]
        v += 3
    return gg.from_edges(v, pairs)


@pytest.mark.parametrize("shape", [{}, {"max_ctas": 2}, {"max_ctas": 1, "block_size": 64}],
                         ids=["all", "two", "small"])
@pytest.mark.parametrize("name", ["layers", "rmat"])
def test_bc_pull_matches_brandes(name, shape):
    g = _layers(1) if name == "layers" else gg.rmat(20000, 24, seed=9)
    for srcs in ([0], [0, g.V - 1, g.V // 2, 1, 0]):
        want = oracle.bc_f64(g, np.array(srcs, np.uint32))
        with gdb.Ctx(**shape) as c:
            got = c.bc(c.graph(g.row_ptr, g.col), srcs)
        # the stated accuracy of the scores, 1e-4 relative
        scale = np.maximum(np.abs(want), 1e-6 * max(1.0, float(np.abs(want).max())))
        assert np.all(np.abs(got - want) <= 1e-4 * scale + 1e-6)
