"""MIS where a vertex's search for a smaller neighbour changes hands: lists of
7 to 9 arcs (the lane's probes), 127 to 129 (the warp's, then one chunk and a
remainder) and several chunks, the smaller neighbour first, last or absent."""
import numpy as np
import pytest

import oracle
from gpu_discovery_barrier_gb300 import gdb, graphgen as gg

pytestmark = pytest.mark.gpu

DEGREES = [1, 4, 7, 8, 9, 31, 32, 40, 127, 128, 129, 136, 256, 257, 700]


def _stars():
    """One star per degree, its leaves joined in a ring to the next star's."""
    pairs, centre, v = [], [], 0
    for d in DEGREES:
        c = v
        centre.append(c)
        pairs += [(c, c + 1 + i) for i in range(d)]
        v += d + 1
        if c:
            pairs.append((c - 1, c + d))
    return gg.from_edges(v, pairs), centre


@pytest.mark.parametrize("case", ["centres lowest", "centres highest", "last leaf lowest", "first leaf lowest",
                                  "random", "some never win"])
def test_mis_probe_edges(case):
    g, centre = _stars()
    prio = gg.priorities(g.V, seed=3)
    lo, hi = -np.arange(1, len(centre) + 1, dtype=np.float32), g.V + np.arange(len(centre), dtype=np.float32)
    if case == "centres lowest":
        prio[centre] = lo
    elif case == "centres highest":
        prio[centre] = hi
    elif case == "last leaf lowest":
        prio[centre] = 0.5
        prio += 1.0
        prio[[c + d for c, d in zip(centre, DEGREES)]] = lo
    elif case == "first leaf lowest":
        prio[centre] = 0.5
        prio += 1.0
        prio[[c + 1 for c in centre]] = lo
    elif case == "some never win":  # decided by neighbours, never chosen themselves
        prio[[c + 1 for c in centre]] = np.nan
        prio[[c + d for c, d in zip(centre, DEGREES) if d > 4]] = 1e9
        prio[centre] = lo
    if case == "some never win":
        # the reference's result: the set of the graph without those leaves
        never = ~(prio < 99999999.0)
        want, _ = oracle.mis(g, np.where(never, np.float32(9e7) + np.arange(g.V, dtype=np.float32) * 8, prio))
        assert not np.any(want[never])
    else:
        want, _ = oracle.mis(g, prio)
    for shape in ({}, {"max_ctas": 1}, {"block_size": 64}):
        with gdb.Ctx(**shape) as c:
            assert np.array_equal(c.mis(c.graph(g.row_ptr, g.col), prio), want), shape
