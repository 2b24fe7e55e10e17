"""Graph creation: the CSR check over 16-byte column groups that start and end
anywhere, and the heavy table over tiles of 1,024 vertices."""
import numpy as np
import pytest

from gpu_discovery_barrier_gb300 import gdb

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _device_graph(ctx, row, col, shift):
    """A graph over device arrays whose columns start `shift` words past a
    16-byte boundary; also the tensors, which it borrows."""
    r = torch.from_numpy(row.astype(np.int32)).cuda()
    buf = torch.zeros(col.size + 8, dtype=torch.int32, device="cuda")
    buf[shift:shift + col.size] = torch.from_numpy(col.astype(np.int32)).cuda()
    torch.cuda.synchronize()
    return gdb.Graph(ctx, (r.data_ptr(), r.numel()), (buf.data_ptr() + 4 * shift, col.size), device=True), (r, buf)


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
@pytest.mark.parametrize("E", [1, 2, 3, 4, 5, 7, 8, 9, 40, 4099])
def test_one_bad_column_is_found(ctx, E, shift):
    V = 50
    row = np.concatenate([np.arange(V) * E // V, [E]])
    good = np.arange(E) % V
    g, keep = _device_graph(ctx, row, good, shift)
    g.close()
    for at in {0, E // 2, E - 1}:
        bad = good.copy()
        bad[at] = V
        with pytest.raises(gdb.GdbError, match="names a vertex"):
            _device_graph(ctx, row, bad, shift)


def test_bad_rows_are_found(ctx):
    col = np.zeros(3000, np.int64)
    row = np.minimum(np.arange(3001), 3000)
    for at in (1, 1023, 1024, 2999):
        bad = row.copy()
        bad[at] = bad[at + 1] + 1 if at + 1 < 3000 else 3001
        with pytest.raises(gdb.GdbError, match="decreases"):
            _device_graph(ctx, bad, col, 0)
    for at, match in ((0, "row_ptr"), (3000, "row_ptr")):
        bad = row.copy()
        bad[at] += 1
        with pytest.raises(gdb.GdbError, match=match):
            _device_graph(ctx, bad, col, 0)


@pytest.mark.parametrize("V", [1, 31, 32, 1023, 1024, 1025, 5000])
def test_heavy_table_counts(ctx, V):
    rng = np.random.default_rng(V)
    deg = rng.choice([0, 3, 128, 129, 256, 257, 1000], V)
    deg[-1] = 700
    row = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint32)
    col = rng.integers(0, V, int(row[-1])).astype(np.uint32)
    G = ctx.graph(row, col)
    assert G.info()["heavy"] == int((deg > 128).sum())
    # every arc of every chunk is walked: reach from the last vertex
    d = ctx.bfs(G, V - 1)
    out = np.unique(col[row[V - 1]:row[V]])
    assert np.all(d[out[out != V - 1]] == 1)
