"""MST, MIS and BC over heavy-chunk tables around the sizes where a warp's batch
of entries changes: one per warp, a few, just under and from 16 per warp (then
32), and tables that end inside a batch."""
import functools

import numpy as np
import pytest

import oracle
from gpu_discovery_barrier_gb300 import gdb, graphgen as gg

pytestmark = pytest.mark.gpu


@functools.lru_cache(maxsize=None)
def _graph(chunks):
    """Hubs of 129 to 520 arcs holding `chunks` 128-arc chunks between them,
    over a shared set of leaves, the hubs in a ring."""
    pairs, left, hub = [], chunks, 0
    degrees = []
    while left > 0:
        k = min(left, 2 + hub % 4)
        if left - k == 1:
            k += 1  # a heavy vertex has two chunks at least
        degrees.append(128 * (k - 1) + 1 + hub % 100)
        left -= k
        hub += 1
    n = len(degrees)
    for h, d in enumerate(degrees):
        # the ring's two arcs (one in a ring of two) are among the hub's d
        ring = 0 if n == 1 else 1 if n == 2 else 2
        if n > 1:
            pairs.append((h, (h + 1) % n))
        pairs += [(h, n + (7 * h + i) % 700) for i in range(d - ring)]
    g = gg.from_edges(n + 700, pairs)
    assert ((g.degrees()[:n] + 127) // 128).sum() == chunks and g.degrees()[n:].max() <= 128
    w = gg.unique_weights(g, seed=3)
    prio = gg.priorities(g.V, seed=4)
    return g, w, prio, oracle.mst(g.with_weights(w)), oracle.mis(g, prio)[0]


# 2 and 16 warps
@pytest.mark.parametrize("shape", [{"max_ctas": 1, "block_size": 64}, {"max_ctas": 1}, {}],
                         ids=["two warps", "one cta", "all"])
@pytest.mark.parametrize("chunks", [2, 3, 4, 15, 16, 17, 31, 32, 33, 63, 64, 65, 97, 255, 256, 257])
def test_chunk_tables(chunks, shape):
    g, w, prio, mst, mis = _graph(chunks)
    with gdb.Ctx(**shape) as c:
        G = c.graph(g.row_ptr, g.col, w)
        m = c.mst(G, with_arcs=True)
        assert (m["weight64"], m["edges"], m["components"]) == (mst["weight64"], mst["edges"], mst["components"])
        assert oracle.mst_edge_set(g, m["arc_in_mst"]) == oracle.mst_edge_set(g, mst["arc_in_mst"])
        assert np.array_equal(c.mis(G, prio), mis)
        for src in (0, g.V - 1):
            want = oracle.bc_f64(g, np.array([src], np.uint32))
            got = c.bc(G, [src])
            scale = np.maximum(np.abs(want), 1e-6 * max(1.0, float(np.abs(want).max())))
            assert np.all(np.abs(got - want) <= 1e-4 * scale + 1e-6)
