"""BC where a pulled hub's path count does not fit FP32 sums of its 128-arc
chunks: one parent of 2^31 paths, first in the hub's list, and 200,000 of one
path, each chunk of which is half a unit of that count.  The hub's and its
parents' scores take four float roundings of the exact values (2.4e-7), within
1e-6 here; the paths that FP32 sums lose would be 9e-5 of them.  And the same
with a parent whose count overflows, against the float32 oracle."""
import functools

import numpy as np
import pytest

import oracle
from gpu_discovery_barrier_gb300 import gdb, graphgen as gg

pytestmark = pytest.mark.gpu


@functools.lru_cache(maxsize=None)
def _graph(stages, parents):
    """Source 0; a chain to a vertex with `parents` children; beside it
    diamonds whose last vertex has 2^stages paths, on the children's level;
    the hub behind them all, and a tail.  Returns graph, that vertex, hub."""
    depth = 2 * stages
    pairs = [(i, i + 1) for i in range(depth - 1)]  # levels 0 .. depth - 1
    v, last = depth, 0
    for _ in range(stages):
        pairs += [(last, v), (last, v + 1), (v, v + 2), (v + 1, v + 2)]
        last, v = v + 2, v + 3
    hub = v + parents
    pairs += [(depth - 1, v + i) for i in range(parents)] + [(v + i, hub) for i in range(parents)]
    pairs += [(last, hub), (hub, hub + 1)]
    return gg.from_edges(hub + 2, pairs), last, hub


@pytest.mark.parametrize("shape", [{}, {"max_ctas": 2}, {"max_ctas": 1, "block_size": 64}],
                         ids=["all", "two", "small"])
def test_hub_count_beyond_float_sums(shape):
    g, last, hub = _graph(31, 200000)
    with gdb.Ctx(**shape) as c:
        G = c.graph(g.row_ptr, g.col)
        for srcs in ([0], [0, 0]):  # a second source finds the sums empty again
            want = oracle.bc_f64(g, np.array(srcs, np.uint32))
            got = c.bc(G, srcs)
            at = np.r_[last, hub - 200000:hub + 1]
            assert np.all(np.abs(got[at] - want[at]) <= 1e-6 * want[at])


@pytest.mark.parametrize("kind", [gdb.BARRIER_XF, gdb.BARRIER_RELAUNCH], ids=["xf", "relaunch"])
def test_hub_count_overflow(kind):
    g, last, hub = _graph(130, 2000)
    want = oracle.bc_f32(g, g, [0])
    with gdb.Ctx(barrier=kind) as c:
        got = c.bc(c.graph(g.row_ptr, g.col), [0])
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    assert np.allclose(got[ok], want[ok], rtol=1e-4, atol=1e-6)
