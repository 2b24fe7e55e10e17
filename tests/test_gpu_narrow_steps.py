"""`supersteps` of an SSSP whose supersteps are narrow ones: on a path every
hop relaxes one vertex, so the count is the path's vertices whatever the CTAs
did on their own (a narrow superstep makes up to 128 hops)."""
import numpy as np
import pytest

from gpu_discovery_barrier_gb300 import gdb, graphgen as gg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [{}, {"max_ctas": 1}], ids=["all", "one"])
@pytest.mark.parametrize("n", [2, 3, 100, 127, 128, 129, 130, 257, 1000])
def test_path_supersteps(n, shape):
    g = gg.from_edges(n, [(i, i + 1) for i in range(n - 1)], np.ones(n - 1, np.uint32))
    with gdb.Ctx(**shape) as c:
        G = c.graph(g.row_ptr, g.col, g.w)
        assert np.array_equal(c.sssp(G, 0), np.arange(n))
        assert c.last_stats()["supersteps"] == n
        # one bucket per 50 vertices: the hops of every bucket's superstep
        c.set_options(sssp_delta=50, sssp_split=-1)
        assert np.array_equal(c.sssp(G, 0), np.arange(n))
        st = c.last_stats()
        assert st["phases"] >= (n - 1) // 50
        assert n <= st["supersteps"] <= n + st["phases"]
