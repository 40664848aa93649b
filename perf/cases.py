"""Performance cases of olive_b200: the calls a program makes through the Python API.

A case names one entry point ("op"), one graph and the call's options.  The
graphs are those the package is used on: scale-free RMAT graphs (a, b, c, d =
0.57, 0.19, 0.19, 0.05, ids permuted, no self-loops or duplicates), four-
neighbour grids (long diameter, as road networks), uniform random digraphs
("er"), and block-diagonal batches of uniform random digraphs.  They are made
with torch on the GPU from the seed alone; traversal sources, seeds, weights
and gradients are drawn from the same generator.

    listed()             the fixed cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  graph handle, inputs and output buffers on the GPU
    run(state)           one call (forward + backward for the training step)
    work(case)           bytes and operations of one pass
    exact(case, seed)    the floating-point results in 64 bits
"""
import math

import numpy as np
import torch

import olive_b200 as ob

DEV = "cuda"
ALPHA = 0.85


def listed():
    return [
        # the smallest traversal: 128 x 128 grid, a few hundred levels of a few
        # hundred vertices each, so launches and latency are what counts
        dict(name="bfs-grid-128x128", op="bfs", graph="grid", rows=128, cols=128),
        # an ordinary traversal of a uniform digraph with an odd vertex count
        dict(name="bfs-er-1000003", op="bfs", graph="er", V=1000003, deg=8),
        # the largest BFS: scale-free, from the highest out-degree vertex
        dict(name="bfs-rmat24", op="bfs", graph="rmat", V=1 << 24, ef=16),
        # road-like shortest paths: long diameter, odd sides
        dict(name="sssp-grid-301x517", op="sssp", graph="grid", rows=301, cols=517, wmax=255),
        # the largest SSSP: weights U[1,255], from the highest out-degree vertex
        dict(name="sssp-rmat24", op="sssp", graph="rmat", V=1 << 24, ef=16, wmax=255),
        # a program that is handed a host graph, solves once and reads the
        # distances back: upload, reverse graph, first solve, result
        dict(name="oneshot-sssp-rmat20", op="oneshot", graph="rmat", V=1 << 20, ef=16, wmax=255),
        # 64 breadth-first searches advanced together
        dict(name="msbfs64-rmat22", op="msbfs", graph="rmat", V=1 << 22, ef=16, n=64),
        # a small PageRank with the reference's leaking dangling mass and its
        # iteration limit: 50 short passes
        dict(name="pagerank-er-20011", op="pagerank", graph="er", V=20011, deg=9, max_it=50,
             tol=0.0, dangling="leak"),
        # PageRank at the benchmark size, to an L1 change of 1e-7
        dict(name="pagerank-rmat22", op="pagerank", graph="rmat", V=1 << 22, ef=16, max_it=50,
             tol=1e-7, dangling="uniform"),
        # 32 personalised PageRank vectors on a scale-free graph
        dict(name="ppr32-rmat21", op="ppr", graph="rmat", V=1 << 21, ef=16, K=32, max_it=20,
             tol=0.0),
        # training step of weighted PageRank: forward with new weights, then
        # the adjoint with the gradients of weights and personalisation
        dict(name="wpr-step-rmat20", op="wpr", graph="rmat", V=1 << 20, ef=16, max_it=100,
             tol=0.0),
        # many small graphs in one call: BFS and 32 PPR vectors of each
        dict(name="batch-96xer", op="batch", graph="batch", count=96, vmin=1024, vmax=65536,
             deg=8, K=32, max_it=20, tol=0.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, vmax):
    """A scale-free or uniform graph of up to vmax vertices, odd sizes included."""
    if rng.random() < 0.65:
        V = _log(rng, 1000, vmax)
        if rng.random() < 0.4:   # a power of two, as generated
            V = 1 << min(max(10, round(math.log2(V))), int(math.log2(vmax)))
        return dict(graph="rmat", V=V, ef=rng.choice([8, 16, 16, 16, 24]) if V < vmax // 2 else 16)
    return dict(graph="er", V=_log(rng, 1000, vmax // 4), deg=rng.randint(4, 16))


def draw(rng):
    op = rng.choice(["bfs", "bfs", "sssp", "sssp", "oneshot", "msbfs", "pagerank", "ppr", "wpr",
                     "batch"])
    if op in ("bfs", "sssp"):
        if rng.random() < 0.35:
            c = dict(graph="grid", rows=_log(rng, 16, 700), cols=_log(rng, 16, 700))
        else:
            c = _draw_graph(rng, 1 << 24)
        c["op"] = op
        if op == "sssp":
            c["wmax"] = rng.choice([1, 15, 255, 255, 255, 1000])
        return c
    if op == "oneshot":
        return dict(_draw_graph(rng, 1 << 20), op=op, wmax=rng.choice([15, 255]))
    if op == "msbfs":
        return dict(_draw_graph(rng, 1 << 22), op=op, n=rng.choice([2, 7, 32, 33, 64, 64]))
    if op == "pagerank":
        tol = rng.choice([0.0, 1e-7])
        return dict(_draw_graph(rng, 1 << 22), op=op, max_it=50 if tol else rng.choice([10, 20, 50]),
                    tol=tol, dangling=rng.choice(["uniform", "leak"]))
    if op == "ppr":
        return dict(_draw_graph(rng, 1 << 21), op=op, K=rng.choice([1, 5, 16, 32, 32]),
                    max_it=rng.choice([10, 20]), tol=0.0)
    if op == "wpr":
        return dict(_draw_graph(rng, 1 << 20), op=op, max_it=rng.choice([30, 50, 100]), tol=0.0)
    vmax = rng.choice([2000, 9001, 65536])
    return dict(op=op, graph="batch", count=rng.randint(8, 96), vmin=max(300, vmax // 64),
                vmax=vmax, deg=rng.choice([6, 8, 10]), K=rng.choice([8, 32, 32]), max_it=20,
                tol=0.0)


# ------------------------------------------------------------------ graphs --
def _csr(key, V):
    """CSR (int32 rowptr, col) of the sorted distinct src * V + dst keys."""
    key = torch.sort(key).values
    keep = torch.ones_like(key, dtype=torch.bool)
    keep[1:] = key[1:] != key[:-1]
    key = key[keep]
    del keep
    src = torch.div(key, V, rounding_mode="floor")
    col = (key - src * V).to(torch.int32)
    rowptr = torch.searchsorted(src, torch.arange(V + 1, device=DEV)).to(torch.int32)
    return rowptr, col


def _rmat(V, ef, gen):
    scale = max(1, (V - 1).bit_length())
    M = ef << scale
    src = torch.zeros(M, dtype=torch.int32, device=DEV)
    dst = torch.zeros(M, dtype=torch.int32, device=DEV)
    for b in range(scale):
        r = torch.rand(M, generator=gen, device=DEV)
        src |= (r >= 0.76).to(torch.int32) << b
        dst |= (((r >= 0.57) & (r < 0.76)) | (r >= 0.95)).to(torch.int32) << b
        del r
    perm = torch.randperm(1 << scale, generator=gen, device=DEV)
    src, dst = perm[src.long()], perm[dst.long()]
    if V < 1 << scale:   # a ragged size: the edges among the first V ids
        ok = (src < V) & (dst < V)
        src, dst = src[ok], dst[ok]
    key = src * V + dst
    key = key[src != dst]
    del src, dst
    return _csr(key, V)


def _er(V, deg, gen):
    src = torch.randint(V, (V * deg,), generator=gen, device=DEV)
    dst = torch.randint(V, (V * deg,), generator=gen, device=DEV)
    return _csr((src * V + dst)[src != dst], V)


def _grid(rows, cols):
    V = rows * cols
    v = torch.arange(V, device=DEV)
    r, c = torch.div(v, cols, rounding_mode="floor"), v % cols
    pairs = [(v[ok] * V + v[ok] + step) for ok, step in
             ((c > 0, -1), (c < cols - 1, 1), (r > 0, -cols), (r < rows - 1, cols))]
    return _csr(torch.cat(pairs), V)


def _batch(case, gen):
    """Block-diagonal uniform digraphs: CSR and instance offsets.  The sizes
    belong to the case, the edges to the seed."""
    size = torch.Generator().manual_seed(case["count"] * 65537 + case["vmax"])
    n = torch.randint(case["vmin"], case["vmax"] + 1, (case["count"],), generator=size).to(DEV)
    off = torch.cat([torch.zeros(1, dtype=n.dtype, device=DEV), n.cumsum(0)])
    V = int(off[-1])
    inst = torch.repeat_interleave(torch.arange(case["count"], device=DEV), n * case["deg"])
    src = torch.repeat_interleave(torch.arange(V, device=DEV), case["deg"])
    dst = off[inst] + (torch.rand(len(src), generator=gen, device=DEV, dtype=torch.float64) *
                       n[inst]).long()
    rowptr, col = _csr((src * V + dst)[src != dst], V)
    return rowptr, col, off


def _graph(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    off = None
    if case["graph"] == "rmat":
        rowptr, col = _rmat(case["V"], case["ef"], gen)
    elif case["graph"] == "er":
        rowptr, col = _er(case["V"], case["deg"], gen)
    elif case["graph"] == "grid":
        rowptr, col = _grid(case["rows"], case["cols"])
    else:
        rowptr, col, off = _batch(case, gen)
    return gen, rowptr, col, off


def _inputs(case, seed):
    """Everything a call takes, as torch tensors on the GPU."""
    # training keeps one graph and changes its weights and gradients
    gen, rowptr, col, off = _graph(case, 1 if case["op"] == "wpr" else seed)
    if case["op"] == "wpr":
        gen.manual_seed(seed)
    V, E = len(rowptr) - 1, len(col)
    d = dict(V=V, E=E, rowptr=rowptr, col=col, off=off)
    deg = rowptr[1:] - rowptr[:-1]
    op = case["op"]
    if op in ("sssp", "oneshot"):
        d["w"] = torch.randint(1, case["wmax"] + 1, (E,), generator=gen, device=DEV,
                               dtype=torch.int32)
    if op in ("bfs", "sssp", "oneshot"):
        # scale-free: the highest out-degree vertex; else any vertex with an edge
        d["src"] = (int(deg.argmax()) if case["graph"] == "rmat" else
                    int(torch.nonzero(deg)[torch.randint(int((deg > 0).sum()), (1,), generator=gen,
                                                         device=DEV)]))
    elif op in ("msbfs", "ppr"):
        n = case["n"] if op == "msbfs" else case["K"]
        nz = torch.nonzero(deg).flatten()
        d["srcs"] = nz[torch.randint(len(nz), (n,), generator=gen, device=DEV)].to(torch.int32)
    elif op == "wpr":
        d["w"] = torch.exp(torch.randn(E, generator=gen, device=DEV))
        p = -torch.log1p(-torch.rand(V, generator=gen, device=DEV, dtype=torch.float64))
        d["p"] = (p / p.sum()).float()
        d["g"] = torch.randn(V, generator=gen, device=DEV)
    elif op == "batch":
        n = (off[1:] - off[:-1])[:, None]
        r = torch.rand(case["count"], case["K"], generator=gen, device=DEV, dtype=torch.float64)
        d["srcs"] = (r * n).long().to(torch.int32)
    return d


# ------------------------------------------------------------------- calls --
def prepare(case, seed):
    d = _inputs(case, seed)
    op, V, E = case["op"], d["V"], d["E"]
    s = dict(case)
    if op == "oneshot":   # host arrays, as a file reader leaves them
        s.update(rowptr=d["rowptr"].cpu().numpy().view(np.uint32),
                 col=d["col"].cpu().numpy().view(np.uint32),
                 w=d["w"].cpu().numpy().view(np.uint32), src=d["src"])
        return s
    torch.cuda.synchronize()
    s["g"] = ob.Graph.from_csr(d["rowptr"], d["col"], d["w"] if op == "sssp" else None)
    i32 = dict(dtype=torch.int32, device=DEV)
    f32 = dict(dtype=torch.float32, device=DEV)
    if op in ("bfs", "sssp"):
        s.update(src=d["src"], out=torch.empty(V, **i32))
    elif op == "msbfs":
        s.update(srcs=d["srcs"], out=torch.empty((case["n"], V), **i32))
    elif op == "pagerank":
        s["out"] = torch.empty(V, **f32)
    elif op == "ppr":
        s.update(srcs=d["srcs"], out=torch.empty((V, case["K"]), **f32))
    elif op == "wpr":
        s.update(w=d["w"], p=d["p"], grad=d["g"], r=torch.empty(V, **f32),
                 dw=torch.empty(E, **f32), dp=torch.empty(V, **f32))
    elif op == "batch":
        s.update(off=d["off"].cpu().numpy().astype(np.uint32), srcs=d["srcs"],
                 levels=torch.empty(V, **i32), out=torch.empty((V, case["K"]), **f32))
    torch.cuda.synchronize()   # the handle's stream reads what torch's stream made
    return s


def run(s):
    op = s["op"]
    if op == "bfs":
        return s["g"].bfs(s["src"], out=s["out"])
    if op == "sssp":
        return s["g"].sssp(s["src"], out=s["out"])
    if op == "oneshot":
        with ob.Graph.from_csr(s["rowptr"], s["col"], s["w"]) as g:
            return g.sssp(s["src"]).view(np.int32)
    if op == "msbfs":
        return s["g"].msbfs(s["srcs"], out=s["out"])
    if op == "pagerank":
        return s["g"].pagerank(ALPHA, s["max_it"], s["tol"], s["dangling"], out=s["out"])
    if op == "ppr":
        return s["g"].ppr(s["srcs"], ALPHA, s["max_it"], s["tol"], out=s["out"])
    if op == "wpr":
        s["g"].wpr_forward(s["p"], w=s["w"], alpha=ALPHA, max_it=s["max_it"], tol=s["tol"],
                           out=s["r"])
        s["g"].wpr_backward(s["grad"], max_it=s["max_it"], tol=s["tol"], dw_out=s["dw"],
                            dp_out=s["dp"])
        return s["r"], s["dw"], s["dp"]
    lv, ppr, iters = s["g"].batch(s["off"], s["srcs"], alpha=ALPHA, max_it=s["max_it"],
                                  tol=s["tol"], levels_out=s["levels"], ppr_out=s["out"])
    return lv, ppr


def work(case):
    """Bytes: each index, weight and vector once per sweep that needs it; a
    traversal reads its graph once and writes its result once.  Edge counts
    are the drawn ones (before duplicates go)."""
    op = case["op"]
    if case["graph"] == "rmat":
        V = case["V"]
        E = case["ef"] * V * (V / (1 << max(1, (V - 1).bit_length())))
    elif case["graph"] == "er":
        V, E = case["V"], case["V"] * case["deg"]
    elif case["graph"] == "grid":
        V = case["rows"] * case["cols"]
        E = 4 * V - 2 * (case["rows"] + case["cols"])
    else:
        V = case["count"] * (case["vmin"] + case["vmax"]) / 2
        E = V * case["deg"]
    if op == "bfs":
        return dict(bytes=4 * E + 8 * V, flops=E)
    if op in ("sssp", "oneshot"):
        return dict(bytes=8 * E + 8 * V, flops=E)
    if op == "msbfs":
        return dict(bytes=4 * E + 4 * V + 4 * V * case["n"], flops=E)
    if op == "pagerank":
        it = 20 if case["tol"] else case["max_it"]
        return dict(bytes=it * (4 * E + 12 * V), flops=it * 2 * E)
    if op == "ppr":
        it, K = case["max_it"], case["K"]
        return dict(bytes=it * (4 * E + 8 * V * K), flops=it * 2 * E * K)
    if op == "wpr":
        it = case["max_it"]
        return dict(bytes=2 * it * (8 * E + 12 * V) + 12 * E, flops=4 * it * E + 4 * E)
    it, K = case["max_it"], case["K"]
    return dict(bytes=4 * E + 8 * V + it * (4 * E + 8 * V * K), flops=it * 2 * E * K)


# ---------------------------------------------------------- 64-bit results --
def _rows(ptr):
    n = (ptr[1:] - ptr[:-1]).long()
    return torch.repeat_interleave(torch.arange(len(n), device=DEV), n)


def _reverse(rowptr, col):
    """(sources, destinations, position in the CSR) in destination order."""
    pos = torch.sort(col, stable=True).indices
    return _rows(rowptr)[pos], col.long()[pos], pos


def _matrix(ptr, idx, val, V):
    return torch.sparse_csr_tensor(ptr, idx, val, (V, V))


def _offsets(sorted_rows, V):
    return torch.searchsorted(sorted_rows, torch.arange(V + 1, device=DEV))


def exact(case, seed):
    op = case["op"]
    if op in ("bfs", "sssp", "oneshot", "msbfs"):
        return None   # whole numbers
    d = _inputs(case, seed)
    V, a = d["V"], ALPHA
    deg = (d["rowptr"][1:] - d["rowptr"][:-1]).double()
    src, dst, pos = _reverse(d["rowptr"], d["col"])
    cptr = _offsets(dst, V)
    if op == "wpr":
        w = d["w"].double()
        rows = _rows(d["rowptr"])
        W = torch.zeros(V, dtype=torch.float64, device=DEV).index_add_(0, rows, w)
        inv = torch.where(W > 0, 1 / W, torch.zeros_like(W))
        P = _matrix(d["rowptr"].long(), d["col"].long(), w * inv[rows], V)
        PT = _matrix(cptr, src, (w * inv[rows])[pos], V)
        p, g = d["p"].double(), d["g"].double()
        r = p.clone()
        for _ in range(case["max_it"]):
            r = (1 - a) * p + a * (PT @ r[:, None])[:, 0]
        lam = g.clone()
        for _ in range(case["max_it"]):
            lam = g + a * (P @ lam[:, None])[:, 0]
        t = (P @ lam[:, None])[:, 0]
        dw = a * (r * inv)[rows] * (lam[d["col"].long()] - t[rows])
        return r, dw, (1 - a) * lam
    dang = deg == 0
    scale = torch.where(dang, torch.zeros_like(deg), 1 / deg)
    A = _matrix(cptr, src, scale[src], V)
    if op == "pagerank":
        r = torch.full((V,), 1.0 / V, dtype=torch.float64, device=DEV)
        for _ in range(case["max_it"]):
            base = (1 - a) / V
            if case["dangling"] == "uniform":
                base = base + a * r[dang].sum() / V
            nr = base + a * (A @ r[:, None])[:, 0]
            change = float((nr - r).abs().sum())
            r = nr
            if change < case["tol"]:
                break
        return r
    K = case["K"]
    k = torch.arange(K, device=DEV)
    if op == "ppr":
        at = d["srcs"].long()
        inst, count = torch.zeros(V, dtype=torch.long, device=DEV), 1
        seeds = at[None, :]
    else:
        off = d["off"]
        count = case["count"]
        inst = torch.repeat_interleave(torch.arange(count, device=DEV), off[1:] - off[:-1])
        seeds = d["srcs"].long() + off[:-1, None]
    r = torch.zeros((V, K), dtype=torch.float64, device=DEV)
    r[seeds, k] = 1.0
    dv = torch.nonzero(dang).flatten()
    for _ in range(case["max_it"]):
        lost = torch.zeros((count, K), dtype=torch.float64, device=DEV)
        lost.index_add_(0, inst[dv], r[dv])
        r = a * (A @ r)
        r[seeds, k] += (1 - a) + a * lost
    return r if op == "ppr" else (None, r)
