"""BFS whose frontier is small for long, then wide: the narrow tail hands the
traversal back to its levels (with their direction choice), takes it up again
on the next thin stretch and may end in either.  Levels and their number
against the oracle; and the direction-optimising schedules inspect far fewer
arcs behind a chain than there are, as they do without the chain."""
import functools

import numpy as np
import pytest

import oracle
from gpu_discovery_barrier_gb300 import gdb, graphgen as gg, selector

pytestmark = pytest.mark.gpu


def _csr(V, pairs):
    u, v = pairs[:, 0], pairs[:, 1]
    key = np.unique(np.concatenate([u * V + v, v * V + u]))
    key = key[key // V != key % V]
    row = np.zeros(V + 1, np.int64)
    np.cumsum(np.bincount(key // V, minlength=V), out=row[1:])
    return gg.CSR(row.astype(np.uint32), (key % V).astype(np.uint32), None, "pairs")


def _chain(a, n, at):
    """n new vertices from id `at` on, hanging off vertex a."""
    c = np.arange(at, at + n)
    return np.stack([np.concatenate([[a], c[:-1]]), c], 1)


def _block(name, at):
    rng = np.random.default_rng(at)
    if name == "rmat":
        g = gg.rmat(1 << 16, 16, seed=3)
        u = np.repeat(np.arange(g.V), g.degrees())
        return g.V, np.stack([u, g.col], 1).astype(np.int64) + at
    if name == "regular":  # eight arcs per vertex: wide after six levels
        V = 60000
        p = [rng.permutation(V) for _ in range(4)]
        return V, np.concatenate([np.stack([q, np.roll(q, 1)], 1) for q in p]) + at
    if name == "star":  # one hub of many chunks
        V = 40000
        return V, np.stack([np.zeros(V - 1, np.int64), np.arange(1, V)], 1) + at
    if name == "cube":
        n = 40
        i = np.arange(n ** 3).reshape(n, n, n)
        return n ** 3, np.concatenate([np.stack([i[:-1].ravel(), i[1:].ravel()], 1),
                                       np.stack([i[:, :-1].ravel(), i[:, 1:].ravel()], 1),
                                       np.stack([i[:, :, :-1].ravel(), i[:, :, 1:].ravel()], 1)]) + at
    raise KeyError(name)


@functools.lru_cache(maxsize=None)
def _graph(blocks, link):
    """The blocks in a row, chains of `link` vertices before, between and
    behind them; the source is the first chain's end."""
    at, pairs, last = link + 1, [_chain(0, link, 1)], link
    for b in blocks.split("+"):
        V, e = _block(b, at)
        pairs += [e, np.array([[last, at]]), _chain(at + V // 2, link, at + V)]
        at += V + link
        last = at - 1
    g = _csr(at, np.concatenate(pairs))
    return g, oracle.bfs(g, 0)


CASES = [("rmat", 5), ("rmat", 20), ("rmat", 200), ("regular", 3), ("regular", 70), ("star", 12), ("cube", 30),
         ("rmat+regular", 40), ("star+star+star", 20), ("regular+cube+rmat+star", 70)]


@pytest.mark.parametrize("shape", [{}, {"max_ctas": 1}, {"max_ctas": 5, "block_size": 64}],
                         ids=["all", "one", "small"])
@pytest.mark.parametrize("schedule", [gdb.SCHED_PLAIN, gdb.SCHED_ADAPTIVE, gdb.SCHED_LEARNED])
@pytest.mark.parametrize("blocks,link", CASES)
def test_levels(blocks, link, schedule, shape):
    g, want = _graph(blocks, link)
    with gdb.Ctx(**shape) as c:
        c.selector_set(selector.load())
        c.set_options(schedule=schedule)
        G = c.graph(g.row_ptr, g.col)
        for _ in range(2):
            assert np.array_equal(c.bfs(G, 0), want)
            assert c.last_stats()["supersteps"] == want[want < gdb.LONESTAR_INF].max() + 1
        got = c.bfs_multi(G, np.array([0, 3, g.V - 1], np.uint32))
        assert np.array_equal(got, np.min([oracle.bfs(g, s) for s in (0, 3, g.V - 1)], axis=0))


@pytest.mark.parametrize("schedule", [gdb.SCHED_ADAPTIVE, gdb.SCHED_LEARNED])
@pytest.mark.parametrize("link", [12, 20, 200])
def test_directions_are_chosen_behind_a_chain(link, schedule):
    g, want = _graph("rmat", link)
    with gdb.Ctx() as c:
        c.selector_set(selector.load())
        c.set_options(schedule=schedule)
        G = c.graph(g.row_ptr, g.col)
        assert np.array_equal(c.bfs(G, 0), want)
        behind = c.last_stats()["edges_processed"]
        c.bfs(G, link + 1)
        assert behind <= c.last_stats()["edges_processed"] + g.E // 20
        assert behind < g.E // 2
