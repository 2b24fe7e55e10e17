"""The kernels of sparse graphs (at most 8 arcs per vertex on average) on both
sides of 2^21 vertices: those with hubs take three CTAs per SM above the line,
those without keep the narrow tail's two; levels against the oracle."""
import numpy as np
import pytest

import oracle
from gpu_discovery_barrier_gb300 import gdb, graphgen as gg

pytestmark = pytest.mark.gpu


def _random(V, ef):
    rng = np.random.default_rng(V)
    u, v = rng.integers(0, V, (2, ef * V))
    key = np.unique(np.concatenate([u * V + v, v * V + u]))
    key = key[key // V != key % V]
    row = np.zeros(V + 1, np.int64)
    np.cumsum(np.bincount(key // V, minlength=V), out=row[1:])
    return gg.CSR(row.astype(np.uint32), (key % V).astype(np.uint32), None, "random")


@pytest.mark.parametrize("schedule", [gdb.SCHED_PLAIN, gdb.SCHED_ADAPTIVE])
@pytest.mark.parametrize("kind,V,per_sm", [("rmat", (1 << 21) + 1, 3), ("rmat", 1 << 21, 2), ("random", (1 << 21) + 1, 2)])
def test_sparse_graph_kernels(kind, V, per_sm, schedule):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    g = gg.rmat(V, 3, seed=2) if kind == "rmat" else _random(V, 2)
    assert 0 < g.E <= 8 * g.V and (g.degrees().max() > 128) == (kind == "rmat")
    src = int(np.argmax(g.degrees()))
    want = oracle.bfs(g, src)
    with gdb.Ctx(schedule=schedule) as c:
        G = c.graph(g.row_ptr, g.col)
        assert np.array_equal(c.bfs(G, src), want)
        assert c.last_stats()["launched"] == per_sm * sms
        for shape in ({"max_ctas": 1}, {"max_ctas": 7}):
            c.set_options(**shape)
            assert np.array_equal(c.bfs(G, src), want), shape
