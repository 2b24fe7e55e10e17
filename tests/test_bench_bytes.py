"""bench.py's byte counts of a launch."""
import types

import bench


def test_mis_bytes_follow_the_arcs_inspected():
    g = types.SimpleNamespace(V=1000, E=32000)
    # column and key per inspected arc, priority, key and result per vertex
    assert bench.alg_bytes("mis", g, [], 3, 5000) == 8 * 5000 + 12 * 1000
    assert bench.alg_bytes("mis", g, [], 9, 5000) == bench.alg_bytes("mis", g, [], 3, 5000)
