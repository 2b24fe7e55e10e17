"""Jacobi SSSP's moved-vertex bits at the edges of their 32-vertex words, on
directed graphs with vertices of one and of several 128-arc chunks, against
the oracle's literal form."""
import numpy as np
import pytest

import oracle
from gpu_discovery_barrier_gb300 import gdb, graphgen as gg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [1, 2, 31, 32, 33, 64, 1000, 1025])
@pytest.mark.parametrize("hubs", [0, 2], ids=["light", "heavy"])
def test_jacobi_directed(V, hubs):
    rng = np.random.default_rng(V)
    pairs = list(map(tuple, rng.integers(0, V, (3 * V, 2))))
    for h in range(min(hubs, V)):  # in-arcs of the hubs, and arcs out of them
        pairs += [(h, int(u)) for u in rng.integers(0, V, 700)]
        pairs += [(int(u), h) for u in rng.integers(0, V, 40)]
    w = rng.integers(1, 1000, len(pairs))
    g = gg.from_edges(V, pairs, weights=w, symmetric=False)
    with gdb.Ctx() as c:
        G = c.graph(g.row_ptr, g.col, g.w)
        for src in {0, V // 2, V - 1}:
            assert np.array_equal(c.sssp_jacobi(G, src), oracle.sssp_jacobi(g, src, literal=True)), src
