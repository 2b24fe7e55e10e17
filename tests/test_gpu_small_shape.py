"""A traversal alone on the GPU takes one CTA per SM up to eight arcs per
thread of that shape; both sides of the line give the same distances, and a
shape the caller sets stays."""
import numpy as np
import pytest

import oracle
from gpu_discovery_barrier_gb300 import gdb, graphgen as gg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extra", [0, 2])
def test_small_graph_shape(extra):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    pairs = (sms * 512 * 8 + extra) // 2  # arcs: two per pair
    n = int(np.sqrt(2 * pairs)) + 2
    u, v = np.triu_indices(n, 1)
    w = np.random.default_rng(3).integers(1, 1000, pairs)
    g = gg.from_edges(n, list(zip(u[:pairs].tolist(), v[:pairs].tolist())), w)
    assert g.E == 2 * pairs
    want_b, want_s = oracle.bfs(g, 0), oracle.sssp_worklist(g, 0)
    with gdb.Ctx() as c:
        G = c.graph(g.row_ptr, g.col, g.w)
        for run, want in ((c.bfs, want_b), (c.sssp, want_s)):
            assert np.array_equal(run(G, 0), want)
            small = c.last_stats()["launched"] <= sms
            assert small == (extra == 0)
        c.set_options(max_ctas=7)
        assert np.array_equal(c.bfs(G, 0), want_b)
        assert c.last_stats()["launched"] == 7
