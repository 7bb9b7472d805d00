"""Performance cases: the calls a user of the library makes, over the sizes it is used at.

A case names an algorithm (``task``), a seeded synthetic graph (``family``,
``scale``, ``ef`` edges drawn per vertex, ``order`` of the vertex ids, ``trim``:
an odd share of the vertices kept, few of them without edges) and a
partitioning (``parts`` blocks of equal vertex count, or ``parts`` random parts
that are not id ranges).  The graphs are built here
with torch from the seed alone and handed to the library as host CSR arrays,
as a program with its own data does; the handles are built once in
``prepare()`` and kept, except by the ``upload`` task, whose pass is the whole
call from host arrays to the result.

Large results go to page-locked arrays the caller keeps (``out=``); small
graphs (below 2^18 vertices) use the methods' default, a new array a call.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import partitionandconquer_b200 as pc

DAMPING, PR_ITERS, CDLP_ITERS, WMAX = 0.85, 20, 10, 255


def _case(name, task, scale, ef=16, family="rmat", order="degree", trim=False, parts=1, blocks=True, option=""):
    return {"name": name, "task": task, "family": family, "scale": scale, "ef": ef, "order": order,
            "trim": trim, "parts": parts, "blocks": blocks, "option": option}


def listed():
    return [
        # the smallest call: counting a 1 K-vertex graph that is resident, as interactive analytics do
        _case("tc_rmat10", "tc", 10, parts=4),
        # the headline workload: triangle counting on RMAT-24 in 1024 partitions
        _case("tc_rmat24", "tc", 24, parts=1024),
        # the whole call of a drop-in caller: host CSR to result, with validation and the partition view
        _case("upload_rmat20", "upload", 20, trim=True, parts=64),
        # clustering coefficients and all-edge similarity of an ordinary social-network-sized graph
        _case("lcc_rmat20", "lcc", 20, trim=True, parts=64),
        _case("jaccard_rmat20", "jaccard", 20, parts=64),
        # the frontier algorithms at the size the benchmark suite runs them at (RMAT-22, 256 partitions)
        _case("bfs_rmat22", "bfs", 22, parts=256),
        _case("sssp_rmat22", "sssp", 22, parts=256),
        _case("pagerank_rmat22", "pagerank", 22, parts=256),
        _case("kcore_rmat22", "kcore", 22, parts=256),
        # a small graph with seed-hashed priorities: the launches and rounds count
        _case("mis_rmat16", "mis", 16, parts=64, option="hashed"),
        # label propagation on a ragged graph whose partitions are not id ranges
        _case("cdlp_rmat20", "cdlp", 20, ef=13, trim=True, parts=37, blocks=False),
        # many small graphs in one call: counts, coefficients and levels of each
        _case("batch_96", "batch", 12, parts=96),
    ]


def draw(rng):
    task = rng.choice(["tc", "upload", "lcc", "jaccard", "bfs", "sssp", "pagerank", "kcore", "mis", "cdlp", "batch"])
    top = {"tc": 22, "upload": 20, "lcc": 20, "jaccard": 20, "batch": 12}.get(task, 22)
    scale = rng.randint(10, top)
    if task == "batch":
        c = _case("", task, scale, ef=rng.randint(6, 20), parts=int(round(math.exp(rng.uniform(math.log(5), math.log(96))))))
    else:
        blocks = rng.random() < 0.75
        c = _case("", task, scale, ef=rng.randint(5, 17), family="er" if rng.random() < 0.25 else "rmat",
                  trim=task != "jaccard" and rng.random() < 0.5,
                  parts=int(round(math.exp(rng.uniform(0, math.log(512 if blocks else 64))))), blocks=blocks)
        if task in ("bfs", "sssp", "pagerank", "kcore", "mis", "cdlp") and rng.random() < 0.3:
            c["order"] = "raw"  # ids as they came: hubs anywhere
        if task == "pagerank":
            c["option"] = rng.choice(["fp32", "fp64"])
        elif task == "mis":
            c["option"] = rng.choice(["hashed", "ids"])
        elif task == "sssp":
            c["option"] = rng.choice(["auto", "bellman_ford"])
    del c["name"]
    return c


# ---- graphs ----------------------------------------------------------------------

def _draw_edges(family, scale, ne, gen):
    """ne endpoint pairs (int64) of the family's distribution."""
    if family == "er":
        return tuple(torch.randint(1 << scale, (ne,), generator=gen, device="cuda") for _ in range(2))
    us, vs = [], []
    for lo in range(0, ne, 1 << 26):  # RMAT(0.57, 0.19, 0.19, 0.05), one quadrant a level
        k = min(1 << 26, ne - lo)
        u = torch.zeros(k, dtype=torch.int64, device="cuda")
        v = torch.zeros(k, dtype=torch.int64, device="cuda")
        for _ in range(scale):
            r = torch.rand(k, generator=gen, device="cuda")
            low = r >= 0.76
            u = u * 2 + low
            v = v * 2 + (((r >= 0.57) & ~low) | (r >= 0.95))
        us.append(u)
        vs.append(v)
    return torch.cat(us), torch.cat(vs)


def _symmetric(u, v, n, order, vertices, edges, gen):
    """(offsets int64[vertices+1], ids int32[m]) on the GPU: both directions,
    sorted, no loops, no repeats; `edges` (if not 0) random ones of them."""
    keep = u != v
    u, v = u[keep], v[keep]
    key = torch.unique(torch.minimum(u, v) * n + torch.maximum(u, v))
    if edges:
        key = key[torch.randperm(key.numel(), generator=gen, device="cuda")[:edges]]
    u, v = key // n, key % n
    del key
    deg = torch.bincount(u, minlength=n) + torch.bincount(v, minlength=n)
    if order == "degree":
        old = torch.sort(deg, descending=True, stable=True).indices
    else:
        old = torch.arange(n, device="cuda")
    new = torch.empty(n, dtype=torch.int64, device="cuda")
    new[old] = torch.arange(n, device="cuda")
    u, v = new[u], new[v]
    if vertices < n:
        keep = torch.maximum(u, v) < vertices
        u, v, n = u[keep], v[keep], vertices
    key = torch.sort(torch.cat((u * n + v, v * n + u))).values
    del u, v
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rows = key // n
    off[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    return off, (key - rows * n).to(torch.int32)


def _graph(c, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed * 7919 + c["scale"])
    n = 1 << c["scale"]
    drawn = n * c["ef"]
    vertices = (n * 9 // 16) | 1 if c["trim"] else n
    # one value per entry comes back: a fixed number of them, below what is left of the draws without repeats
    edges = int(drawn * min(0.9, 0.6 + 0.03 * (c["scale"] - 10))) if c["task"] == "jaccard" else 0
    return _symmetric(*_draw_edges(c["family"], c["scale"], drawn, gen), n, c["order"], vertices, edges, gen)


def _arena(c, seed):
    """`parts` graphs of scales up to the case's in one block-diagonal CSR, with each graph's first vertex."""
    rng = np.random.default_rng(c["parts"])
    offs, adjs, voff = [torch.zeros(1, dtype=torch.int64, device="cuda")], [], [0]
    base = 0
    for k in range(c["parts"]):
        one = dict(c, scale=int(rng.integers(max(6, c["scale"] - 4), c["scale"] + 1)), ef=int(rng.integers(8, 2 * c["ef"] + 1)))
        off, adj = _graph(one, seed * 1009 + k)
        offs.append(off[1:] + base)
        adjs.append(adj + voff[-1])
        base += adj.numel()
        voff.append(voff[-1] + off.numel() - 1)
    return torch.cat(offs), torch.cat(adjs), np.asarray(voff, np.uint64)


def _weights(off, adj):
    """Weights 1..WMAX, the same for both directions of an edge."""
    u = _rows(off)
    v = adj.long()
    h = torch.minimum(u, v) * 0x9E3779B1 + torch.maximum(u, v) * 0x85EBCA77
    return (((h >> 7) ^ (h >> 19)) % WMAX + 1).abs().clamp(1, WMAX).to(torch.int32)


def _rows(off):
    return torch.repeat_interleave(torch.arange(off.numel() - 1, device="cuda"), off[1:] - off[:-1])


def _host(t, pinned=False):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t) if pinned else t.cpu()
    a = h.numpy()
    return a.view(np.uint64) if a.dtype == np.int64 else a


def _partition(c, n, seed):
    if c["parts"] <= 1:
        return None
    if c["blocks"]:
        return pc.equal_vertex_partition(n, c["parts"])
    return np.random.default_rng(seed + 17).integers(0, c["parts"], n, dtype=np.int32)


# ---- what is measured ------------------------------------------------------------

RESULT = {"lcc": ("n", torch.float64), "jaccard": ("m", torch.float32), "bfs": ("n", torch.int32),
          "sssp": ("n", torch.int32), "pagerank": ("n", torch.float32), "kcore": ("n", torch.int32),
          "mis": ("n", torch.int32), "cdlp": ("n", torch.int32)}


def prepare(case, seed):
    c, task = case, case["task"]
    if task == "batch":
        off, adj, voff = _arena(c, seed)
        return {"case": c, "batch": pc.Batch(_host(off), _host(adj), voff)}
    off, adj = _graph(c, seed)
    n, m = off.numel() - 1, adj.numel()
    w = _weights(off, adj) if task == "sssp" else None
    source = int(adj[(seed * 104729 + 13) % m]) if m else 0
    pinned = task == "upload"
    vl, el, w = _host(off, pinned), _host(adj, pinned), None if w is None else _host(w)
    del off, adj
    torch.cuda.empty_cache()
    st = {"case": c, "seed": seed, "source": source, "v2p": _partition(c, n, seed), "out": None}
    if task == "upload":
        st["arrays"] = (vl, el)
        return st
    st["g"] = pc.Graph(vlist=vl, elist=el, weights=w)
    st["pg"] = pc.Partitioned_Graph(st["g"], st["v2p"])
    if task in RESULT and n >= 1 << 18:
        size, dtype = RESULT[task]
        if task == "pagerank" and c["option"] == "fp64":
            dtype = torch.float64
        st["out"] = torch.empty(n if size == "n" else m, dtype=dtype, pin_memory=True).numpy()
    if task == "cdlp":
        st["labels"] = np.arange(n, dtype=np.int32)
    return st


def run(state):
    c, task = state["case"], state["case"]["task"]
    if task == "batch":
        r = state["batch"].run()
        return {"tc": r["tc"], "lcc": r["lcc"], "bfs": r["bfs"]}
    if task == "upload":
        g = pc.Graph(vlist=state["arrays"][0], elist=state["arrays"][1])
        pg = pc.Partitioned_Graph(g, state["v2p"])
        count = pg.solve_triangle_counting_merge()
        pg.close()
        g.close()
        return count
    pg, out = state["pg"], state["out"]
    if task == "tc":
        return pg.solve_triangle_counting_merge()
    if task == "lcc":
        return pg.solve_lcc_merge(out=out)
    if task == "jaccard":
        return pg.jaccard_edges(out=out)
    if task == "bfs":
        return pg.solve_bfs(state["source"], out=out)
    if task == "sssp":
        method = pc.SSSP_BELLMAN_FORD if c["option"] == "bellman_ford" else pc.SSSP_AUTO
        return pg.solve_sssp(state["source"], out=out, method=method)
    if task == "pagerank":
        return pg.page_rank(DAMPING, PR_ITERS, fp64=c["option"] == "fp64", out=out)
    if task == "kcore":
        return pg.solve_kcore(out=out)
    if task == "mis":
        return pg.solve_mis(seed=state["seed"] if c["option"] == "hashed" else None, out=out)
    return pg.solve_cdlp(state["labels"], CDLP_ITERS, out=out)


def work(case):
    """The CSR (and weights) read once and the result written once; 2 flops an edge and iteration."""
    c, task = case, case["task"]
    n = 1 << c["scale"]
    m = 2 * c["ef"] * n
    if task == "batch":
        n, m = n * c["parts"] * 0.39, 1.4 * m * c["parts"] * 0.39
        return {"bytes": 8 * n + 4 * m + 8 * c["parts"] + 12 * n, "flops": 0}
    out = {"tc": 8, "upload": 8, "lcc": 8 * n, "jaccard": 4 * m, "cdlp": 8 * n}.get(task, 4 * n)
    if c["option"] == "fp64":
        out = 8 * n
    iters = {"pagerank": PR_ITERS, "cdlp": CDLP_ITERS}.get(task, 0)
    return {"bytes": 8 * n + 4 * m + (4 * m if task == "sssp" else 0) + out, "flops": 2 * m * iters}


# ---- values in 64 bits -----------------------------------------------------------

def _edge_triangles(off, adj):
    """Common neighbours of the ends of every CSR entry (int64), by listing the paths c > b > a of sorted rows."""
    n, m = off.numel() - 1, adj.numel()
    row, col = _rows(off), adj.long()
    down = torch.nonzero(col < row).flatten()  # the entries (c, b), b < c
    key = row * n + col  # ascending
    dkey = key[down]
    first = off[row[down]]
    rank = down - first  # b's place in row c: the ids below it come first
    ends = torch.cumsum(rank, 0)
    hits = torch.zeros(m, dtype=torch.int64, device="cuda")
    lo, total = 0, int(ends[-1]) if ends.numel() else 0
    while lo < down.numel():
        done = int(ends[lo - 1]) if lo else 0
        hi = max(lo + 1, int(torch.searchsorted(ends, torch.tensor(done + (1 << 26), device="cuda"), right=True)))
        r = rank[lo:hi]
        pair = torch.repeat_interleave(torch.arange(lo, hi, device="cuda"), r)
        at = torch.arange(pair.numel(), device="cuda") - (torch.cumsum(r, 0) - r)[pair - lo] + first[pair]
        want = col[down[pair]] * n + col[at]  # the entry (b, a)
        pos = torch.searchsorted(dkey, want).clamp_(max=dkey.numel() - 1)
        ok = dkey[pos] == want
        for e in (down[pair[ok]], at[ok], down[pos[ok]]):
            hits += torch.bincount(e, minlength=m)
        lo = hi
    twin = torch.searchsorted(key, torch.maximum(row, col) * n + torch.minimum(row, col))
    return hits[twin], row, col


def exact(case, seed):
    c, task = case, case["task"]
    if task == "batch":
        off, adj, _ = _arena(c, seed)
    elif task in ("lcc", "jaccard", "pagerank"):
        off, adj = _graph(c, seed)
    else:
        return None  # whole numbers
    n = off.numel() - 1
    deg = (off[1:] - off[:-1]).double()
    if task == "pagerank":
        base = (1.0 - DAMPING) / n
        A = torch.sparse_csr_tensor(off, adj.long(), torch.ones(adj.numel(), dtype=torch.float64, device="cuda"), (n, n))
        x = deg / DAMPING / n
        for _ in range(PR_ITERS):
            x = base + A @ torch.where(deg > 0, x * DAMPING / deg.clamp(min=1), torch.zeros_like(x))
        return x
    hits, row, col = _edge_triangles(off, adj)
    if task == "jaccard":
        common = hits.double()
        return common / (deg[row] + deg[col] - common)
    lcc = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, row, hits.double())
    lcc = torch.where(deg > 0, lcc / (deg * (deg - 1)), torch.zeros_like(lcc))
    return {"tc": None, "lcc": lcc, "bfs": None} if task == "batch" else lcc
