"""MST where a round's work changes hands: graphs of 31 to 129 vertices and of
several grabs of four 32-vertex groups, chunk tables of 31 to 33 and of more
entries, and graphs declared symmetric, whose last round is not run: the same
forest and round count either way, on connected graphs and on many components."""
import numpy as np
import pytest

import oracle
from gpu_discovery_barrier_gb300 import gdb, graphgen as gg

pytestmark = pytest.mark.gpu


def _hubs(n, degree):
    """n hubs of `degree` leaves (ceil(degree / 128) chunks each) in a ring."""
    pairs = [(h, (h + 1) % n) for h in range(n)] if n > 1 else []
    for h in range(n):
        pairs += [(h, n + h * degree + i) for i in range(degree)]
    return gg.from_edges(n + n * degree, pairs)


def _pieces(n):
    """n separate pieces: paths of 2 to 40 vertices, and isolated vertices."""
    pairs, v = [], 0
    for i in range(n):
        k = 2 + i % 39
        pairs += [(v + j, v + j + 1) for j in range(k - 1)]
        v += k + i % 3
    return gg.from_edges(v, pairs)


GRAPHS = {f"grid{n}": gg.grid(1, n) for n in (31, 32, 33, 127, 128, 129)}
GRAPHS |= {"rmat5000": gg.rmat(5000, 8, seed=2), "rmat70001": gg.rmat(70001, 6, seed=3),
           "hubs31": _hubs(31, 126), "hubs33": _hubs(33, 127), "hubs20x300": _hubs(20, 300),
           "pieces": _pieces(500), "none": gg.from_edges(50, [])}


@pytest.mark.parametrize("name", list(GRAPHS))
def test_mst_rounds(ctx, name):
    g = GRAPHS[name]
    w = gg.unique_weights(g, seed=5)
    want = oracle.mst(g.with_weights(w))
    got = []
    for symmetric in (False, True):
        m = ctx.mst(ctx.graph(g.row_ptr, g.col, w, symmetric=symmetric), with_arcs=True)
        assert (m["weight64"], m["edges"], m["components"]) == \
            (want["weight64"], want["edges"], want["components"])
        assert oracle.mst_edge_set(g, m["arc_in_mst"]) == oracle.mst_edge_set(g, want["arc_in_mst"])
        got.append((m["rounds"], m["arc_in_mst"].tolist()))
    assert got[0] == got[1]
