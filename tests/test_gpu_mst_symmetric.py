"""MST of graphs declared symmetric, whose last round is counted and not run,
under tied weights and arcs that are never chosen (1e9 and above): the forest
has the oracle's weight and size, and the same rounds, weight and edges as the
same graph undeclared."""
import numpy as np
import pytest

import oracle
from gpu_discovery_barrier_gb300 import gdb, graphgen as gg

pytestmark = pytest.mark.gpu

GRAPHS = {"grid": gg.grid(40, 33), "rmat": gg.rmat(5000, 8, seed=4), "path": gg.grid(1, 500),
          "star": gg.from_edges(700, [(0, i) for i in range(1, 700)]),
          "pieces": gg.from_edges(300, [(3 * i, 3 * i + 1) for i in range(100)]
                                  + [(3 * i + 1, 3 * i + 2) for i in range(0, 100, 2)])}


def _weights(g, kind):
    """One weight per undirected edge."""
    u = np.repeat(np.arange(g.V, dtype=np.uint64), g.degrees())
    v = g.col.astype(np.uint64)
    mix = np.minimum(u, v) * np.uint64(2654435761) + np.maximum(u, v) * np.uint64(40503)
    mix ^= mix >> np.uint64(13)
    w = {"equal": np.full(g.E, 7), "two": 1 + mix % 2, "eight": 1 + mix % 8,
         "never": np.full(g.E, gdb.LONESTAR_INF), "some never": np.where(mix % 3 == 0, 1 << 31, 1 + mix % 5),
         "most never": np.where(mix % 10 > 0, gdb.LONESTAR_INF, 999_999_999)}[kind]
    return w.astype(np.uint32)


@pytest.mark.parametrize("kind", ["equal", "two", "eight", "never", "some never", "most never"])
@pytest.mark.parametrize("name", list(GRAPHS))
def test_symmetric_mst(ctx, name, kind):
    g = GRAPHS[name]
    w = _weights(g, kind)
    want = oracle.mst(g.with_weights(w))
    got = []
    for symmetric in (False, True):
        m = ctx.mst(ctx.graph(g.row_ptr, g.col, w, symmetric=symmetric), with_arcs=True)
        assert (m["weight64"], m["edges"], m["components"]) == (want["weight64"], want["edges"], want["components"])
        assert m["arc_in_mst"].sum() == m["edges"]
        got.append((m["rounds"], m["arc_in_mst"].tolist()))
    assert got[0] == got[1]
