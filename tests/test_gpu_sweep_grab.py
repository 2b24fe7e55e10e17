"""Jacobi SSSP and MST on graphs either side of the line where sweeps hand out
one grab per warp (at most 6 arcs per vertex, no heavy vertex) instead of four:
grids whose 32-vertex groups are fewer, as many and several times the warps of
a small launch."""
import numpy as np
import pytest

import oracle
from gpu_discovery_barrier_gb300 import gdb, graphgen as gg

pytestmark = pytest.mark.gpu


def _with(g, extra):
    u = np.repeat(np.arange(g.V), g.degrees())
    return gg.from_edges(g.V, [(int(a), int(b)) for a, b in zip(u, g.col) if a < b] + extra(g))


KINDS = {"thin": lambda g: [], "hub": lambda g: [(0, i) for i in range(1, min(g.V, 200))],
         "seven": lambda g: [(i, (i * 7 + k) % g.V) for i in range(g.V) for k in (3, 11)]}


@pytest.mark.parametrize("shape", [{"max_ctas": 1, "block_size": 64}, {"max_ctas": 3}, {}], ids=["two", "48", "all"])
@pytest.mark.parametrize("rows", [5, 16, 33, 64, 200])
@pytest.mark.parametrize("kind", list(KINDS))
def test_sweeps(kind, rows, shape):
    g = _with(gg.grid(rows, 31), KINDS[kind])
    assert (g.E <= 6 * g.V) == (kind != "seven") or rows == 5
    w = gg.unique_weights(g, seed=rows)
    gw = g.with_weights(w)
    want = oracle.mst(gw)
    with gdb.Ctx(**shape) as c:
        G = c.graph(g.row_ptr, g.col, w, symmetric=True)
        assert np.array_equal(c.sssp_jacobi(G, 0), oracle.sssp_jacobi(gw, 0, literal=True))
        m = c.mst(G, with_arcs=True)
        assert (m["weight64"], m["edges"], m["components"]) == (want["weight64"], want["edges"], want["components"])
        assert oracle.mst_edge_set(g, m["arc_in_mst"]) == oracle.mst_edge_set(g, want["arc_in_mst"])
