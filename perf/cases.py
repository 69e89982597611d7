"""Timed workloads: what programs have the library do, over the sizes they use.

``listed()`` gives the standing cases, ``draw(rng)`` one more of the same
ranges.  ``prepare`` makes the graph and the sources on the GPU from a seed
and uploads the graph (the handle a program keeps), ``run`` is one call of a
public entry point, ``work`` the bytes and operations the call cannot do
without, ``exact`` the floating-point results in 64 bits from plain torch.
"""

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gal-dawn_gb300"))
from dawn_gb300 import abi, gen  # noqa: E402

FLT_MAX = float(np.finfo(np.float32).max)


def listed():
    return [
        # one query on a small social graph, distances back on the host: the
        # smallest call a program makes, all latency
        dict(name="bfs_one_small", call="bfs_one", graph="rmat", scale=12, ef=8, host=True),
        # one source on the benchmark's RMAT graph, distances kept on the GPU
        dict(name="bfs_one_large", call="bfs_one", graph="rmat", scale=22, ef=16, host=False),
        # one source on a street-like mesh: two thousand small levels
        dict(name="bfs_one_grid", call="bfs_one", graph="grid", rows=1000, cols=1049, host=False),
        # the CPU-sized configuration: directed random graph, 64 sources
        dict(name="mssp_er", call="mssp", graph="er", n=65536, degree=16.0, nsrc=64),
        # the headline configuration: RMAT-22, 64 sources in one batch
        dict(name="mssp_large", call="mssp", graph="rmat", scale=22, ef=16, nsrc=64),
        # a source list of 500 (the length of the reference's own list)
        dict(name="mssp_many", call="mssp", graph="rmat", scale=18, ef=16, nsrc=500),
        # closeness of a thousand vertices of the same graph
        dict(name="closeness", call="closeness", graph="rmat", scale=18, ef=16, nsrc=1000),
        # weighted distances of one source, real-valued lengths
        dict(name="sssp_one_large", call="sssp_one", graph="rmat", scale=22, ef=16, weights="f32"),
        # weighted distances of 64 sources, whole-number lengths
        dict(name="sssp_batch_large", call="sssp_batch", graph="rmat", scale=22, ef=16, weights="i32", nsrc=64),
        # a distance matrix on a mesh of points, real-valued lengths
        dict(name="sssp_batch_knn", call="sssp_batch", graph="knn", n=200003, weights="f32", nsrc=50),
        # betweenness from a sample of sources
        dict(name="betweenness", call="betweenness", graph="rmat", scale=16, ef=16, nsrc=150),
        # many uneven directed graphs in one call
        dict(name="multi_er", call="multi", graphs=300, nmin=1024, nmax=65536, dmin=4, dmax=32, smin=8, smax=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, top):
    """A graph of at most about ``top`` entries, of any of the four kinds."""
    kind = rng.choice(["rmat", "rmat", "er", "grid", "knn"])
    entries = _log_int(rng, 1 << 14, top)
    if kind == "rmat":
        ef = rng.choice([8, 12, 16])
        return dict(graph="rmat", ef=ef, scale=max(8, min(22, int(math.log2(entries / (2 * ef))))))
    if kind == "er":
        degree = round(rng.uniform(4, 32), 2)
        return dict(graph="er", n=min(1 << 20, max(300, int(entries / degree))), degree=degree)
    entries = min(entries, 1 << 22)  # meshes: thousands of levels, so smaller ones
    if kind == "grid":
        rows = max(8, int(math.sqrt(entries / 4) * rng.uniform(0.5, 1.5)))
        return dict(graph="grid", rows=rows, cols=max(8, entries // (4 * rows)))
    return dict(graph="knn", n=max(300, entries // 10))


def draw(rng):
    call = rng.choice(["bfs_one", "mssp", "mssp", "closeness", "sssp_one", "sssp_batch", "betweenness", "multi"])
    if call == "bfs_one":
        return dict(call=call, host=rng.random() < 0.4, **_draw_graph(rng, 1 << 27))
    if call == "mssp":
        g = _draw_graph(rng, 1 << 26)
        top = 500 if g["graph"] in ("rmat", "er") else 64
        if g["graph"] == "grid":
            g["rows"], g["cols"] = min(g["rows"], 700), min(g["cols"], 700)
        return dict(call=call, nsrc=max(2, min(_log_int(rng, 2, top), (1 << 28) // _vertices(g))), **g)
    if call == "closeness":
        g = _draw_graph(rng, 1 << 24)
        top = 1000 if g["graph"] in ("rmat", "er") else 64
        if g["graph"] == "grid":
            g["rows"], g["cols"] = min(g["rows"], 600), min(g["cols"], 600)
        return dict(call=call, nsrc=_log_int(rng, 2, top), **g)
    if call == "sssp_one":
        return dict(call=call, weights=rng.choice(["i32", "f32"]), **_draw_graph(rng, 1 << 27))
    if call == "sssp_batch":
        g = _draw_graph(rng, 1 << 25)
        if g["graph"] == "grid":
            g["rows"], g["cols"] = min(g["rows"], 400), min(g["cols"], 400)
        elif g["graph"] == "knn":
            g["n"] = min(g["n"], 200000)
        return dict(call=call, weights=rng.choice(["i32", "f32"]), nsrc=_log_int(rng, 2, 100 if g["graph"] == "rmat" else 50), **g)
    if call == "betweenness":
        g = _draw_graph(rng, 1 << 21)
        if g["graph"] == "grid":
            g["rows"], g["cols"] = min(g["rows"], 150), min(g["cols"], 150)
        elif g["graph"] == "knn":
            g["n"] = min(g["n"], 50000)
        return dict(call=call, nsrc=_log_int(rng, 16, 200), **g)
    nmin = _log_int(rng, 256, 8192)
    return dict(call="multi", graphs=_log_int(rng, 8, 300), nmin=nmin, nmax=_log_int(rng, 2 * nmin, 65536),
                dmin=4, dmax=rng.choice([12, 20, 32]), smin=rng.choice([1, 8, 30]), smax=rng.choice([33, 64, 100]))


# --- graphs -----------------------------------------------------------------


def _vertices(c):
    if c["graph"] == "rmat":
        return 1 << c["scale"]
    return c["rows"] * c["cols"] if c["graph"] == "grid" else c["n"]


def _entries(c):
    """CSR entries, to a few percent (repeated RMAT edges collapse)."""
    if c["graph"] == "rmat":
        return int(2 * c["ef"] * (1 << c["scale"]) * (1 - (0.8 + 0.075 * c["ef"]) * 2.0 ** (-0.25 * c["scale"])))
    if c["graph"] == "er":
        return int(c["n"] * c["degree"])
    if c["graph"] == "grid":
        return 4 * c["rows"] * c["cols"] - 2 * (c["rows"] + c["cols"])
    return int(9.2 * c["n"])


def _csr(n, u, v, symmetric):
    """Device int32 CSR of an edge list: no self loops, no repeats, sorted."""
    keep = u != v
    u, v = u[keep], v[keep]
    key = u * n + v
    if symmetric:
        key = torch.cat([key, v * n + u])
    del u, v, keep
    key = torch.unique(key)
    row = torch.div(key, n, rounding_mode="floor")
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    col = (key - row * n).to(torch.int32)
    return rp.to(torch.int32), col, row


def _rmat(c, g):
    n, e = 1 << c["scale"], c["ef"] << c["scale"]
    u = torch.zeros(e, dtype=torch.int64, device="cuda")
    v = torch.zeros_like(u)
    for _ in range(c["scale"]):
        r = torch.rand(e, device="cuda", generator=g)
        u.mul_(2).add_(r >= 0.76)
        v.mul_(2).add_(((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    perm = torch.randperm(n, device="cuda", generator=g)
    return _csr(n, perm[u], perm[v], True)


def _er(n, e, g):
    r = torch.randint(0, n * n, (e,), device="cuda", generator=g)
    return _csr(n, torch.div(r, n, rounding_mode="floor"), r % n, False)


def _graph(c, seed, g):
    """row_ptr, col and row of every entry on the GPU, and whether symmetric."""
    if c["graph"] == "rmat":
        return *_rmat(c, g), True
    if c["graph"] == "er":
        return *_er(c["n"], int(c["n"] * c["degree"]), g), False
    h = gen.grid(c["rows"], c["cols"], seed=seed) if c["graph"] == "grid" else gen.knn(c["n"], 8, seed=seed)
    rp = torch.from_numpy(h.row_ptr).cuda()
    row = torch.repeat_interleave(torch.arange(h.n, device="cuda"), (rp[1:] - rp[:-1]).long())
    return rp, torch.from_numpy(h.col).cuda(), row, True


def _edge_weights(kind, n, row, col, seed):
    """One length in [1, 64) per undirected edge, the same both ways."""
    lo, hi = torch.minimum(row, col.long()), torch.maximum(row, col.long())
    h = (lo * n + hi) * 0x9E3779B97F4A7C1 + (seed * 0x632BE59BD9B4E01) % (1 << 62)
    h = (h ^ (h >> 29)) * 0x94D049BB133111E
    bits = (h >> 20) & 0xFFFFFF
    if kind == "i32":
        return (1 + bits % 63).to(torch.int32)
    return (1 + bits.double() * (63.0 / (1 << 24))).to(torch.float32)


_STREAM = []


def _stream():
    """The stream that a program puts its traversals on."""
    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
    return _STREAM[0].cuda_stream


def _inputs(case, seed):
    """The case's CSR, weights (or None) and sources, from the seed alone."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    rng = np.random.default_rng(seed)
    rp, col, row, sym = _graph(case, seed, g)
    n = rp.numel() - 1
    w = _edge_weights(case["weights"], n, row, col, seed) if "weights" in case else None
    deg = (rp[1:] - rp[:-1]).cpu().numpy()
    some = np.flatnonzero(deg > 0).astype(np.int32)  # sources that have somewhere to go
    nsrc = case.get("nsrc", 1)
    return dict(n=n, rp=rp, col=col, sym=sym, w=w, row=row, sources=rng.choice(some, nsrc, replace=nsrc > some.size))


def _handle(n, rp, col, sym, w=None):
    torch.cuda.synchronize()
    wtype = abi.W_NONE if w is None else (abi.W_I32 if w.dtype == torch.int32 else abi.W_F32)
    return abi.Graph(raw=dict(n=n, m=col.numel(), row_ptr=rp.data_ptr(), col=col.data_ptr(),
                              val=0 if w is None else w.data_ptr(), wtype=wtype, symmetric=sym, stream=_stream(),
                              device=True))


def _prepare_multi(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    # the sizes belong to the case, the edges and the sources to the seed
    sizes, rng = np.random.default_rng(case["graphs"]), np.random.default_rng(seed)
    ns = sizes.integers(case["nmin"], case["nmax"] + 1, case["graphs"])
    es = np.round(ns * sizes.uniform(case["dmin"], case["dmax"], case["graphs"])).astype(np.int64)
    counts = sizes.integers(case["smin"], case["smax"] + 1, case["graphs"])
    off = np.concatenate([[0], np.cumsum(ns)])
    size, base = torch.from_numpy(ns).cuda(), torch.from_numpy(off[:-1]).cuda()
    part = torch.repeat_interleave(torch.arange(case["graphs"], device="cuda"), torch.from_numpy(es).cuda())
    u, v = (base[part] + (torch.rand(part.numel(), device="cuda", generator=g, dtype=torch.float64) * size[part]).long()
            for _ in range(2))
    rp, col, _ = _csr(int(off[-1]), u, v, False)
    h = _handle(int(off[-1]), rp, col, False)
    h.set_parts(off)
    sources = [rng.integers(0, int(n), int(k)).astype(np.int32) for n, k in zip(ns, counts)]
    dist = torch.empty(h.multi_out_size(sources), dtype=torch.int32, device="cuda")
    return dict(call="multi", h=h, sources=sources, dist=dist)


def prepare(case, seed):
    if case["call"] == "multi":
        return _prepare_multi(case, seed)
    x = _inputs(case, seed)
    h = _handle(x["n"], x["rp"], x["col"], x["sym"], x["w"])
    s = dict(call=case["call"], h=h, sources=x["sources"], host=case.get("host", False))
    if case["call"] in ("bfs_one", "mssp", "sssp_one", "sssp_batch") and not s["host"]:
        kind = torch.float32 if case.get("weights") == "f32" else torch.int32
        s["dist"] = torch.empty((len(x["sources"]), x["n"]), dtype=kind, device="cuda")
    return s


def run(s):
    h, call = s["h"], s["call"]
    if call in ("bfs_one", "mssp"):
        if s["host"]:
            return h.bfs(s["sources"])[0]
        h.bfs_device(s["sources"], s["dist"].data_ptr(), stats=False)
        return s["dist"]
    if call in ("sssp_one", "sssp_batch"):
        h.sssp_device(s["sources"], s["dist"].data_ptr(), stats=False)
        return s["dist"]
    if call == "closeness":
        cc, total, reached = h.closeness(s["sources"])
        return dict(cc=cc, total=total, reached=reached)
    if call == "betweenness":
        return h.betweenness(s["sources"])[0]
    h.multi_bfs_ptr(s["sources"], s["dist"].data_ptr(), device=True, stats=False)
    return s["dist"]


def work(case):
    """CSR and sources read once, results written once; one addition and one
    comparison per (entry, source) where values are summed or minimised."""
    if case["call"] == "multi":
        n = case["graphs"] * (case["nmin"] + case["nmax"]) // 2
        rows = (case["smin"] + case["smax"]) // 2
        return dict(bytes=4 * n + 4 * n * (case["dmin"] + case["dmax"]) // 2 + 4 * n * rows, flops=0)
    n, m, nsrc = _vertices(case), _entries(case), case.get("nsrc", 1)
    out = {"closeness": 24 * nsrc, "betweenness": 8 * n}.get(case["call"], 4 * n * nsrc)
    weighted = "weights" in case
    return dict(bytes=4 * (n + 1) + 4 * m * (2 if weighted else 1) + 4 * nsrc + out,
                flops=2 * m * nsrc if weighted or case["call"] == "betweenness" else 0)


# --- results in 64 bits -------------------------------------------------------


def _levels(adj, n, sources):
    """Hop distances (n x sources, -1 unreached); adj holds v's in-edges in row v."""
    k = len(sources)
    lev = torch.full((n, k), -1, dtype=torch.int32, device="cuda")
    lev[torch.from_numpy(sources).long().cuda(), torch.arange(k, device="cuda")] = 0
    d = 0
    while True:
        new = (adj @ (lev == d).double() > 0) & (lev < 0)
        if not bool(new.any()):
            return lev, d
        d += 1
        lev[new] = d


def _adjacency(x, transposed):
    n, m = x["n"], x["col"].numel()
    one = torch.ones(m, dtype=torch.float64, device="cuda")
    if not transposed or x["sym"]:
        return torch.sparse_csr_tensor(x["rp"].long(), x["col"].long(), one, size=(n, n))
    order = torch.argsort(x["col"].long() * n + x["row"])
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(torch.bincount(x["col"], minlength=n), 0)
    return torch.sparse_csr_tensor(rp, x["row"][order], one, size=(n, n))


def _exact_closeness(x):
    n, tin = x["n"], _adjacency(x, True)
    total, reached = [], []
    for i in range(0, len(x["sources"]), 64):
        lev = _levels(tin, n, x["sources"][i:i + 64])[0]
        total.append(lev.clamp(min=0).long().sum(0))
        reached.append((lev > 0).long().sum(0))
    total, reached = torch.cat(total).double(), torch.cat(reached)
    cc = torch.where(total > 0, (n - 1) / total, torch.zeros_like(total))
    return dict(cc=cc.cpu().numpy(), total=total.cpu().numpy(), reached=reached.cpu().numpy())


def _exact_betweenness(x):
    n, tin, tout = x["n"], _adjacency(x, True), _adjacency(x, False)
    bc = torch.zeros(n, dtype=torch.float64, device="cuda")
    for i in range(0, len(x["sources"]), 64):
        lev, deepest = _levels(tin, n, x["sources"][i:i + 64])
        delta = torch.zeros(lev.shape, dtype=torch.float64, device="cuda")
        for d in range(deepest - 1, 0, -1):
            amount = tin @ (lev == d).double()
            term = torch.where(lev == d + 1, 1.0 / amount.clamp(min=1.0) + delta, 0.0)
            at = lev == d
            delta[at] = (tout @ term)[at]
        bc += torch.where(lev > 0, delta, 0.0).sum(1)
    return bc.cpu().numpy()


def _exact_distances(x):
    """Bellman-Ford from all sources together.  The graph and its lengths are
    the same both ways (or turned round first), so row v holds v's in-edges."""
    n, k = x["n"], len(x["sources"])
    rp, tail, w = x["rp"].long(), x["col"].long(), x["w"].double()
    if not x["sym"]:
        order = torch.argsort(tail * n + x["row"])
        rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        rp[1:] = torch.cumsum(torch.bincount(tail, minlength=n), 0)
        tail, w = x["row"][order], w[order]
    d = torch.full((n, k), math.inf, dtype=torch.float64, device="cuda")
    at = torch.from_numpy(x["sources"]).long().cuda(), torch.arange(k, device="cuda")
    d[at] = 0.0
    step = 0
    while True:
        new = torch.segment_reduce(d[tail] + w[:, None], "min", offsets=rp, axis=0, initial=math.inf, unsafe=True)
        new = torch.minimum(new, d)
        step += 1
        if step % 8 == 0 and bool((new == d).all()):
            break
        d = new
    return torch.where(torch.isinf(d), FLT_MAX, d).t().contiguous()


def exact(case, seed):
    if case["call"] == "closeness":
        return _exact_closeness(_inputs(case, seed))
    if case["call"] == "betweenness":
        return _exact_betweenness(_inputs(case, seed))
    if case.get("weights") == "f32":
        return _exact_distances(_inputs(case, seed))
    return None  # whole numbers
