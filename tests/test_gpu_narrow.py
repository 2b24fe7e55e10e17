"""Narrow supersteps (CTAs relaxing small frontiers on their own) against the
oracle, where they hand work over: long chains (more hops than one superstep
makes), reaching more arcs than the slots hold, vertices of 127 to 129 arcs
(slots, then heavy chunks), hubs inside the tail, one CTA, many sources and
arcs that are never taken."""
import functools

import numpy as np
import pytest

import oracle
from gpu_discovery_barrier_gb300 import gdb, graphgen as gg, selector

pytestmark = pytest.mark.gpu


def _pairs(name):
    if name == "path":  # 128 hops a superstep, 64 levels a bucket
        return 1000, [(i, i + 1) for i in range(999)]
    if name == "comb":  # chain of vertices with 125 / 126 / 127 leaves
        n, e = 60, []
        v = n
        for i in range(n):
            if i + 1 < n:
                e.append((i, i + 1))
            for _ in range(125 + i % 3):
                e.append((i, v))
                v += 1
        return v, e
    if name == "hub":  # two long chains through a hub of 3,000 leaves
        e = [(i, i + 1) for i in range(200)] + [(200, 201 + i) for i in range(3000)]
        e += [(3200, 3201)] + [(i, i + 1) for i in range(3201, 3400)]
        return 3401, e
    if name == "bush":  # a chain into a random graph of 30 arcs per vertex
        rng = np.random.default_rng(5)
        e = [(i, i + 1) for i in range(100)]
        e += [(100 + int(a), 100 + int(b)) for a, b in rng.integers(0, 4000, (60000, 2))]
        return 4100, e
    raise KeyError(name)


@functools.lru_cache(maxsize=None)
def _graph(name):
    if name.startswith("grid"):
        r, c = map(int, name[4:].split("x"))
        g = gg.grid(r, c)
    else:
        g = gg.from_edges(*_pairs(name))
    w = gg.uniform_weights(g, 1, 1000, seed=7)
    if name == "grid61x67":  # arcs that are never taken, both ways
        u = np.repeat(np.arange(g.V), g.degrees())
        w = np.where((u * 7919 + g.col * 7919) % 5 == 0, np.uint32(gdb.LONESTAR_INF), w).astype(np.uint32)
    g = g.with_weights(w)
    return g, oracle.bfs(g, 0), oracle.sssp_worklist(g, 0)


NAMES = ["path", "comb", "hub", "bush", "grid61x67", "grid1x3000", "grid300x300"]


@pytest.mark.parametrize("shape", [{}, {"max_ctas": 1}, {"max_ctas": 5, "block_size": 64}],
                         ids=["all", "one", "small"])
@pytest.mark.parametrize("schedule", [gdb.SCHED_PLAIN, gdb.SCHED_ADAPTIVE, gdb.SCHED_LEARNED])
@pytest.mark.parametrize("name", NAMES)
def test_narrow_supersteps_match_oracle(name, schedule, shape):
    g, levels, dist = _graph(name)
    with gdb.Ctx(**shape) as c:
        c.selector_set(selector.load())
        c.set_options(schedule=schedule)
        G = c.graph(g.row_ptr, g.col, g.w)
        assert np.array_equal(c.bfs(G, 0), levels)
        assert c.last_stats()["supersteps"] == levels[levels < gdb.LONESTAR_INF].max() + 1
        assert np.array_equal(c.sssp(G, 0), dist)
        for delta in (1, 300, 100000):
            c.set_options(sssp_delta=delta, sssp_split=-1)
            assert np.array_equal(c.sssp(G, 0), dist), delta


@pytest.mark.parametrize("name", ["grid300x300", "hub"])
def test_narrow_many_sources(name):
    g, _, _ = _graph(name)
    srcs = np.array([0, g.V - 1, g.V // 2, 0], np.uint32)
    want_b = np.min([oracle.bfs(g, int(s)) for s in srcs], axis=0)
    want_s = np.min([oracle.sssp_worklist(g, int(s)) for s in srcs], axis=0)
    with gdb.Ctx(schedule=gdb.SCHED_ADAPTIVE, sssp_split=-1) as c:
        G = c.graph(g.row_ptr, g.col, g.w)
        assert np.array_equal(c.bfs_multi(G, srcs), want_b)
        assert np.array_equal(c.sssp_multi(G, srcs), want_s)
