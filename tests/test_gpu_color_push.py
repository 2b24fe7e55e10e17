"""Colouring where one batch of count-downs completes many vertices at once:
every reservation holds light entries and chunks of several lanes and steps.

A root of the highest priority joins `n` middle vertices, so its entry (or
its chunks) makes all of them ready in one round; middle vertex i has
(1, 127, 128, 129, 257, 640)[i % 6] leaves, all of lower priority and each also
joined to a common sink, so that they wait for it."""
import numpy as np
import pytest

import oracle
from gpu_discovery_barrier_gb300 import gdb, graphgen as gg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [gdb.BARRIER_XF, gdb.BARRIER_RELAUNCH], ids=["xf", "relaunch"])
@pytest.mark.parametrize("n", [1, 6, 32, 33, 128, 129, 300])
def test_color_many_ready_at_once(n, kind):
    leaves = [(1, 127, 128, 129, 257, 640)[i % 6] for i in range(n)]
    V = 2 + n + sum(leaves)
    pairs, v = [], 2 + n
    for i, k in enumerate(leaves):
        pairs.append((0, 2 + i))
        pairs += [(2 + i, v + j) for j in range(k)] + [(1, v + j) for j in range(k)]
        v += k
    prio = np.empty(V, np.float32)
    prio[0], prio[1] = V, 1
    prio[2:2 + n] = V - 1 - np.arange(n)
    prio[2 + n:] = 2 + np.random.default_rng(n).permutation(V - 2 - n)
    g = gg.from_edges(V, pairs)
    with gdb.Ctx(barrier=kind) as c:
        got = c.color(c.graph(g.row_ptr, g.col), prio)
    want, _ = oracle.color(g, prio)
    assert want.min() == 1
    assert np.array_equal(got, want)
