"""Performance cases: the calls that programs make on this framework.

Each kind below is one call pattern through `gpu_discovery_barrier_gb300.gdb`,
over the range of graphs it is used on.  `listed` holds the named cases,
`draw` gives further ones of the same ranges.  Graphs are seeded and built on
the GPU with plain torch operations: R-MAT graphs with the repository's
parameters (0.57, 0.19, 0.19, 0.05), symmetrised, duplicates and self-loops
removed, and 4-neighbour grids; both with one weight per undirected edge.

kind      what a pass is
query     BFS, then worklist SSSP, from one source of a small resident graph,
          results in host arrays (`ctx.bfs`, `ctx.sssp`, default options)
grid      BFS and SSSP from the corner of a grid, learned schedule, results on
          the device: thousands of tiny supersteps
bfs       independent BFS from several sources, learned schedule
sssp      independent SSSP from several sources, learned schedule
jacobi    Pannotia's Jacobi SSSP, pulled over the whole graph per iteration
mis       maximal independent set from a permutation of priorities
color     greedy colouring from a permutation of priorities
bc        betweenness centrality summed over several sources
mst       a graph taken over from device arrays, its minimum spanning forest
          with the arc marks, and the graph released again: a forest is
          asked for once per graph
batch     one replay of a captured batch: BFS and SSSP from one source of each
          of many uneven graphs, results in host arrays
serve     a burst of requests (BFS, SSSP, single-source BC) on a server with
          resident graphs, until the last result is in its host array
train     training epochs of the schedule selector's network on trace rows,
          then the trained network's costs of every row (for its regret)
"""
from __future__ import annotations

import math

import numpy as np
import torch

from gpu_discovery_barrier_gb300 import gdb, selector
from gpu_discovery_barrier_gb300.graphgen import CSR

DEV = "cuda"


def listed():
    return [
        # the smallest call a host program makes: launch and read-back latency
        {"name": "query_rmat1000", "kind": "query", "graph": "rmat", "V": 1000, "ef": 8},
        # the barrier-bound configuration: 8,190 levels from the corner
        {"name": "grid4096", "kind": "grid", "rows": 4096, "cols": 4096},
        # the R-MAT scale 22 suite, app by app, 16 sources where it has sources
        {"name": "bfs16_rmat22", "kind": "bfs", "V": 1 << 22, "ef": 16, "nsrc": 16},
        {"name": "sssp16_rmat22", "kind": "sssp", "V": 1 << 22, "ef": 16, "nsrc": 16},
        {"name": "bc16_rmat22", "kind": "bc", "V": 1 << 22, "ef": 16, "nsrc": 16},
        {"name": "mis_rmat22", "kind": "mis", "V": 1 << 22, "ef": 16},
        {"name": "color_rmat22", "kind": "color", "V": 1 << 22, "ef": 16},
        {"name": "mst_rmat22", "kind": "mst", "V": 1 << 22, "ef": 16},
        # an ordinary, odd-sized graph for the Pannotia SSSP
        {"name": "jacobi_rmat1000003", "kind": "jacobi", "V": 1000003, "ef": 16},
        # many small uneven graphs at once: the batched and the serving form
        {"name": "batch64", "kind": "batch", "members": 64, "vmax": 100000},
        {"name": "serve64", "kind": "serve", "members": 24, "requests": 64, "slots": 64, "vmax": 100000},
        # the selector's training set has 135,000 rows
        {"name": "train135k", "kind": "train", "rows": 135000, "epochs": 25},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "grid", "bfs", "sssp", "bc", "mis", "color", "mst", "jacobi", "batch",
                       "serve", "train"])
    c = {"kind": kind}
    if kind == "query":
        c.update(graph=rng.choice(["rmat", "grid"]), V=_log(rng, 1000, 100000))
        if c["graph"] == "rmat":
            c["ef"] = rng.randint(8, 32)
        else:
            c["aspect"] = round(math.exp(rng.uniform(0, math.log(64))), 3)
    elif kind == "grid":
        c.update(rows=_log(rng, 64, 4096), cols=_log(rng, 64, 4096))
    elif kind in ("bfs", "sssp", "bc"):
        c.update(V=_log(rng, 4096, 1 << 22), ef=rng.randint(8, 16), nsrc=rng.randint(1, 16))
    elif kind in ("mis", "color", "mst"):
        c.update(V=_log(rng, 4096, 1 << 22), ef=rng.randint(8, 16))
    elif kind == "jacobi":
        c.update(V=_log(rng, 4096, 1 << 21), ef=rng.randint(8, 16))
    elif kind == "batch":
        c.update(members=rng.randint(8, 64), vmax=_log(rng, 10000, 100000))
    elif kind == "serve":
        c.update(members=rng.randint(8, 24), requests=rng.randint(16, 64), slots=rng.choice([8, 16, 32, 64]),
                 vmax=_log(rng, 10000, 100000))
    else:
        c.update(rows=_log(rng, 1000, 135000), epochs=rng.randint(5, 25))
    return c


# ------------------------------------------------------------------ graphs
def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) & 0x7FFFFFFFFFFFFFFF)


def _symmetric(V, u, v, w):
    """CSR (int32 tensors) of the undirected edges u - v of weight w."""
    key, order = torch.sort(torch.cat([u * V + v, v * V + u]))
    wt = torch.cat([w, w])[order].to(torch.int32)
    del order
    src = key // V
    col = (key - src * V).to(torch.int32)
    row = torch.zeros(V + 1, dtype=torch.int64, device=DEV)
    row[1:] = torch.cumsum(torch.bincount(src, minlength=V), 0)
    return row.to(torch.int32), col, wt


def _weights(m, weights, gen):
    """m edge weights: uniform in [1, weights], or a permutation of 1..m (0)."""
    if weights == 0:
        return torch.randperm(m, generator=gen, device=DEV) + 1
    return torch.randint(1, weights + 1, (m,), generator=gen, device=DEV)


def _rmat(V, ef, weights, gen):
    n = int(V * ef)
    u = torch.zeros(n, dtype=torch.int64, device=DEV)
    v = torch.zeros(n, dtype=torch.int64, device=DEV)
    for _ in range(max(1, (V - 1).bit_length())):
        r = torch.rand(n, generator=gen, device=DEV)
        u.mul_(2).add_(r >= 0.76)
        v.mul_(2).add_(((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    keep = (u < V) & (v < V) & (u != v)
    u, v = u[keep], v[keep]
    key = torch.unique(torch.minimum(u, v) * V + torch.maximum(u, v))
    u = key // V
    return _symmetric(V, u, key - u * V, _weights(key.numel(), weights, gen))


def _grid(rows, cols, weights, gen):
    i = torch.arange(rows * cols, dtype=torch.int64, device=DEV).view(rows, cols)
    u = torch.cat([i[:, :-1].reshape(-1), i[:-1].reshape(-1)])
    v = torch.cat([i[:, 1:].reshape(-1), i[1:].reshape(-1)])
    return _symmetric(rows * cols, u, v, _weights(u.numel(), weights, gen))


def _sources(row, count, gen):
    """`count` vertices that have arcs."""
    some = torch.nonzero(row[1:] > row[:-1]).view(-1)
    return some[torch.randint(some.numel(), (count,), generator=gen, device=DEV)].to(torch.int32)


def _grid_shape(V, aspect):
    rows = max(1, int(round(math.sqrt(V / aspect))))
    return rows, max(2, int(round(V / rows)))


def _members(case, gen):
    """The uneven graphs of a batch or a server, as host CSRs: vertex counts
    log-uniform in [1000, vmax], R-MAT (edge factor 8 to 32) and grids (aspect
    ratio log-uniform in [1, 64]) in turn.  The sizes are the same for every
    seed, so that passes on other inputs do the same amount of work."""
    sizes = np.random.default_rng(case["members"] * 1000003 + case["vmax"])
    out = []
    for i in range(case["members"]):
        V = int(round(math.exp(sizes.uniform(math.log(1000), math.log(case["vmax"])))))
        ef, aspect = int(sizes.integers(8, 33)), math.exp(sizes.uniform(0, math.log(64)))
        if i % 2 == 0:
            row, col, w = _rmat(V, ef, 255, gen)
        else:
            row, col, w = _grid(*_grid_shape(V, aspect), 1000, gen)
        src = int(_sources(row, 1, gen)[0])
        host = [t.cpu().numpy().view(np.uint32) for t in (row, col, w)]
        out.append(CSR(*host, name="rmat" if i % 2 == 0 else "grid", meta={"source": src}))
    return out


def _context(learned):
    ctx = gdb.Ctx()
    if learned:
        ctx.selector_set(selector.load())
        ctx.set_options(schedule=gdb.SCHED_LEARNED)
    return ctx


def _resident(ctx, row, col, w):
    """A graph over device arrays, declared symmetric (they all are here)."""
    wp = None if w is None else (w.data_ptr(), w.numel())
    return gdb.Graph(ctx, (row.data_ptr(), row.numel()), (col.data_ptr(), col.numel()), wp, device=True,
                     symmetric=True)


# ----------------------------------------------------------------- prepare
def _inputs(case, seed):
    """Everything that is drawn from the seed."""
    gen = _generator(seed)
    kind = case["kind"]
    if kind == "query":
        if case["graph"] == "rmat":
            row, col, w = _rmat(case["V"], case["ef"], 255, gen)
        else:
            row, col, w = _grid(*_grid_shape(case["V"], case["aspect"]), 1000, gen)
        return {"row": row, "col": col, "w": w, "src": int(_sources(row, 1, gen)[0])}
    if kind == "grid":
        row, col, w = _grid(case["rows"], case["cols"], 1000, gen)
        return {"row": row, "col": col, "w": w}
    if kind in ("bfs", "sssp", "bc"):
        row, col, w = _rmat(case["V"], case["ef"], 255, gen)
        return {"row": row, "col": col, "w": w, "src": _sources(row, case["nsrc"], gen)}
    if kind in ("mis", "color"):
        row, col, _ = _rmat(case["V"], case["ef"], 255, gen)
        return {"row": row, "col": col, "prio": torch.randperm(case["V"], generator=gen, device=DEV).float()}
    if kind == "jacobi":
        row, col, w = _rmat(case["V"], case["ef"], 255, gen)
        return {"row": row, "col": col, "w": w, "src": int(_sources(row, 1, gen)[0])}
    if kind == "mst":
        row, col, w = _rmat(case["V"], case["ef"], 0, gen)
        return {"row": row, "col": col, "w": w}
    if kind in ("batch", "serve"):
        d = {"graphs": _members(case, gen)}
        if kind == "serve":
            rng = np.random.default_rng(seed)
            d["requests"] = []
            for k in range(case["requests"]):
                i = k % case["members"]
                g = d["graphs"][i]
                # no BC on the grids: float32 path counts overflow there
                app = (gdb.APP_BFS, gdb.APP_SSSP, gdb.APP_BC)[(k // 2) % (3 if g.name == "rmat" else 2)]
                some = np.flatnonzero(np.diff(g.row_ptr.astype(np.int64)))
                d["requests"].append((i, app, int(some[rng.integers(some.size)])))
        return d
    # train: rows as the traces give them (log-scaled sizes, fractions and
    # flags), two of the six targets known per row, one row in eight with the
    # other four
    rng = np.random.default_rng(seed)
    n = case["rows"]
    x = rng.uniform(0, 1, (n, gdb.MLP_FEATURES)).astype(np.float32)
    x[:, :5] *= np.float32(24)
    x[:, 9] = x[:, 9] > 0.5
    t = (x[:, :1] * 0.3 + x[:, 1:2] * 0.2 + rng.normal(0, 1, (n, gdb.MLP_OUTPUTS))).astype(np.float32)
    m = np.zeros((n, gdb.MLP_OUTPUTS), np.float32)
    run = rng.uniform(0, 1, n) < 0.125
    m[~run, :2] = 1
    m[run, 2:] = 1
    p = selector.init_params(1, x.mean(0), 1.0 / np.maximum(x.std(0), 1e-3))
    return {"p": p, "x": x, "t": t, "m": m}


def prepare(case, seed):
    kind = case["kind"]
    d = _inputs(case, seed)
    ctx = _context(kind in ("grid", "bfs", "sssp", "batch", "serve"))
    s = {"kind": kind, "case": case, "ctx": ctx, **d}
    if kind == "query":
        host = [d[k].cpu().numpy().view(np.uint32) for k in ("row", "col", "w")]
        s["g"] = ctx.graph(*host, symmetric=True)
        del s["row"], s["col"], s["w"]
    elif kind == "batch":
        # the launch shape the tuner settles on for such batches
        ctx.set_options(max_ctas=ctx.device_info()["sm_count"], sssp_split=-1)
        g = ctx.graph_batch(d["graphs"])
        src = np.array([g.vertex_offset[i] + m.meta["source"] for i, m in enumerate(d["graphs"])], np.uint32)
        s["batch"] = ctx.batch(g, src)
        del s["graphs"]
    elif kind == "serve":
        gs = [ctx.graph(m.row_ptr, m.col, m.w, symmetric=True) for m in d["graphs"]]
        s["server"] = ctx.server(slots=case["slots"], pool_bytes=1 << 30)
        s["ids"] = [s["server"].add_graph(g) for g in gs]
        del s["graphs"]
    elif kind != "train":
        if kind != "mst":
            s["g"] = _resident(ctx, d["row"], d["col"], d.get("w"))
        V = d["row"].numel() - 1
        shape = (case["nsrc"], V) if kind in ("bfs", "sssp") else (V,)
        s["out"] = torch.empty(shape, dtype=torch.float32 if kind == "bc" else torch.int32, device=DEV)
        if kind == "grid":
            s["out2"] = torch.empty_like(s["out"])
        if kind == "mst":
            s["out"] = torch.empty(6, dtype=torch.int32, device=DEV)  # gdb_mst_result
            # one mark per arc, with room for the generator's duplicates
            s["flags"] = torch.zeros(2 * case["ef"] * V, dtype=torch.uint8, device=DEV)
    torch.cuda.synchronize()
    return s


# --------------------------------------------------------------------- run
def run(s):
    ctx, kind = s["ctx"], s["kind"]
    if kind == "query":
        return [ctx.bfs(s["g"], s["src"]), ctx.sssp(s["g"], s["src"])]
    if kind == "grid":
        ctx.bfs_device(s["g"], 0, s["out"].data_ptr())
        ctx.sssp_device(s["g"], 0, s["out2"].data_ptr())
        return [s["out"], s["out2"]]
    if kind == "bfs":
        ctx.bfs_sources_device(s["g"], s["src"].data_ptr(), s["src"].numel(), s["out"].data_ptr())
    elif kind == "sssp":
        ctx.sssp_sources_device(s["g"], s["src"].data_ptr(), s["src"].numel(), s["out"].data_ptr())
    elif kind == "bc":
        ctx.bc_device(s["g"], s["src"].data_ptr(), s["src"].numel(), s["out"].data_ptr())
    elif kind == "mis":
        ctx.mis_device(s["g"], s["prio"].data_ptr(), s["out"].data_ptr())
    elif kind == "color":
        ctx.color_device(s["g"], s["prio"].data_ptr(), s["out"].data_ptr())
    elif kind == "jacobi":
        ctx.sssp_jacobi_device(s["g"], s["src"], s["out"].data_ptr())
    elif kind == "mst":
        g = _resident(ctx, s["row"], s["col"], s["w"])
        ctx.mst_device(g, s["out"].data_ptr(), s["flags"].data_ptr())
        g.close()
        return [s["out"], s["flags"]]
    elif kind == "batch":
        s["batch"].run()
        return s["batch"].results()
    elif kind == "serve":
        got = [s["server"].submit(s["ids"][i], app, src)[1] for i, app, src in s["requests"]]
        s["server"].drain()
        for info in s["server"].poll(len(got)):
            if info["status"] != 0:
                raise RuntimeError("request failed: %r" % info["status"])
        return got
    else:
        p, loss = ctx.mlp_train(s["p"], s["x"], s["t"], s["m"], s["case"]["epochs"], 3e-3, 1e-4)
        return [p, loss, ctx.mlp_forward(p, s["x"])]
    return s["out"]


# -------------------------------------------------------------------- work
def _arcs(V, ef):
    """Arcs of an R-MAT graph: 2 ef V less the duplicates (about 5 %)."""
    return 1.9 * ef * V


def work(case):
    """Bytes: every input read once, every output written once (4-byte words).
    The network's arithmetic counts three products per weight and row."""
    kind = case["kind"]
    if kind == "train":
        n, params = case["rows"], 12 * 32 + 32 * 32 + 32 * 6
        return {"bytes": 4.0 * n * (12 + 6 + 6) * case["epochs"], "flops": 6.0 * n * params * case["epochs"]}
    if kind in ("batch", "serve"):
        sizes = np.random.default_rng(case["members"] * 1000003 + case["vmax"])
        words = []
        for i in range(case["members"]):
            V = int(round(math.exp(sizes.uniform(math.log(1000), math.log(case["vmax"])))))
            ef = int(sizes.integers(8, 33))
            sizes.uniform(0, math.log(64))
            E = _arcs(V, ef) if i % 2 == 0 else 4.0 * V
            words.append((2 * V + E, 2 * V + 2 * E))  # an unweighted and a weighted traversal
        if kind == "batch":
            return {"bytes": 4.0 * sum(a + b for a, b in words), "flops": 0}
        return {"bytes": 4.0 * sum(words[k % case["members"]][(k // 2) % 2] for k in range(case["requests"])),
                "flops": 0}
    if kind == "grid":
        V = case["rows"] * case["cols"]
        E = 4.0 * V
    elif kind == "query" and case["graph"] == "grid":
        V, E = case["V"], 4.0 * case["V"]
    else:
        V, E = case["V"], _arcs(case["V"], case["ef"])
    words = {"query": 2 * V + 2 * E + V, "grid": 2 * V + 2 * E + V, "bfs": V + E + V * case.get("nsrc", 1),
             "sssp": V + 2 * E + V * case.get("nsrc", 1), "bc": 2 * V + E, "mis": 3 * V + E,
             "color": 3 * V + E, "jacobi": 2 * V + 2 * E, "mst": V + 2 * E + E / 4}
    return {"bytes": 4.0 * words[kind], "flops": 0}


# ------------------------------------------------------------------- exact
def _bc_exact(row, col, sources):
    """Brandes' betweenness summed over the sources, float64, level by level."""
    V = row.numel() - 1
    deg = (row[1:] - row[:-1]).long()
    src = torch.repeat_interleave(torch.arange(V, device=DEV), deg)
    dst = col.long()
    bc = torch.zeros(V, dtype=torch.float64, device=DEV)
    for s in sources:
        level = torch.full((V,), -1, dtype=torch.int32, device=DEV)
        paths = torch.zeros(V, dtype=torch.float64, device=DEV)
        level[s], paths[s] = 0, 1.0
        steps = []
        while True:
            at = torch.nonzero(level[src] == len(steps)).view(-1)
            u, v = src[at], dst[at]
            level[v[level[v] < 0]] = len(steps) + 1
            down = level[v] == len(steps) + 1
            u, v = u[down], v[down]
            if not u.numel():
                break
            paths.index_add_(0, v, paths[u])
            steps.append((u, v))
        dep = torch.zeros(V, dtype=torch.float64, device=DEV)
        for u, v in reversed(steps):
            dep.index_add_(0, u, paths[u] / paths[v] * (1.0 + dep[v]))
        dep[s] = 0.0
        bc += dep
    return bc


def _train_exact(d, epochs, lr=3e-3, wd=1e-4):
    """The masked squared loss's full-batch Adam in float64."""
    F, H, O = gdb.MLP_FEATURES, 32, gdb.MLP_OUTPUTS
    p, x, t, m = (torch.from_numpy(np.asarray(d[k], np.float64)).to(DEV) for k in ("p", "x", "t", "m"))
    parts, at = [], 2 * F
    for shape in ((F, H), (H,), (H, H), (H,), (H, O), (O,)):
        n = int(np.prod(shape))
        parts.append(p[at:at + n].view(shape).clone())
        at += n
    xn = (x - p[:F]) * p[F:2 * F]
    m1 = [torch.zeros_like(a) for a in parts]
    m2 = [torch.zeros_like(a) for a in parts]
    loss = 0.0
    for k in range(1, epochs + 1):
        w1, b1, w2, b2, w3, b3 = parts
        h1 = torch.relu(xn @ w1 + b1)
        h2 = torch.relu(h1 @ w2 + b2)
        e = h2 @ w3 + b3 - t
        loss = float((m * e * e).sum() / m.sum())
        dy = 2.0 * m * e / m.sum()
        d2 = (dy @ w3.T) * (h2 > 0)
        d1 = (d2 @ w2.T) * (h1 > 0)
        grads = [xn.T @ d1, d1.sum(0), h1.T @ d2, d2.sum(0), h2.T @ dy, dy.sum(0)]
        rate = lr * math.sqrt(1 - 0.999 ** k) / (1 - 0.9 ** k)
        for i, g in enumerate(grads):
            g = g + wd * parts[i] if i % 2 == 0 else g
            m1[i] = 0.9 * m1[i] + 0.1 * g
            m2[i] = 0.999 * m2[i] + 0.001 * g * g
            parts[i] = parts[i] - rate * m1[i] / (m2[i].sqrt() + 1e-8)
    w1, b1, w2, b2, w3, b3 = parts
    y = torch.relu(torch.relu(xn @ w1 + b1) @ w2 + b2) @ w3 + b3
    return [torch.cat([p[:2 * F]] + [a.reshape(-1) for a in parts]), loss, y]


def exact(case, seed):
    """Outputs in 64 bits, for those that are not whole numbers (levels,
    distances, sets, colours and forests are: they have to be equal)."""
    kind = case["kind"]
    if kind == "train":
        return _train_exact(_inputs(case, seed), case["epochs"])
    if kind == "bc":
        d = _inputs(case, seed)
        return _bc_exact(d["row"], d["col"], d["src"].tolist())
    if kind == "serve":
        d = _inputs(case, seed)
        out = []
        for i, app, src in d["requests"]:
            g = d["graphs"][i]
            row, col = (torch.from_numpy(a.view(np.int32)).to(DEV) for a in (g.row_ptr, g.col))
            out.append(_bc_exact(row, col, [src]) if app == gdb.APP_BC else None)
        return out
    return None
