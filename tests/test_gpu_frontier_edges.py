"""The frontier kernels at the sizes where their splits of work change: rows
around the bounds of a light row, a chunk and a warp's buffer, stars, long
paths, empty rows, dense cores, graphs of one and two vertices; ids in any
order.  Every result is a whole number and equals the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

INT_MAX = 2**31 - 1


def csr(n, a, b):
    a, b = np.asarray(a, np.int64), np.asarray(b, np.int64)
    a, b = a[a != b], b[a != b]
    key = np.unique(np.concatenate([a * n + b, b * n + a]))
    vl = np.zeros(n + 1, np.uint64)
    np.cumsum(np.bincount(key // n, minlength=n), out=vl[1:])
    return vl, (key % n).astype(np.int32)


def build(kind):
    rng = np.random.default_rng(7)
    if kind == "one":
        return csr(1, [], [])
    if kind == "two":
        return csr(2, [0], [1])
    if kind == "clique":
        return csr(300, *np.triu_indices(300, 1))
    if kind == "path":
        p = rng.permutation(3000)
        return csr(3000, p[:-1], p[1:])
    if kind == "rows":
        # centres whose rows end around 32, 128, 256, 512, 1024 and 4096 entries, over shared leaves, joined in a ring
        sizes = [s + d for s in (32, 128, 256, 512, 1024, 4096) for d in (-1, 0, 1)]
        n = 6000
        ids = rng.permutation(n)
        a, b = [], []
        for i, s in enumerate(sizes):
            a.append(np.full(s - 2, ids[i]))
            b.append(ids[100 + rng.choice(5000, s - 2, replace=False)])
            a.append([ids[i]])
            b.append([ids[(i + 1) % len(sizes)]])
        return csr(n, np.concatenate(a), np.concatenate(b))  # ids[5100:] are isolated
    if kind == "layers":
        # layers of growing width, each complete to the next one: frontiers from 1 to 2000 and back
        widths = [1, 3, 40, 300, 2000, 300, 40, 3, 1]
        starts = np.concatenate([[0], np.cumsum(widths)])
        a, b = [], []
        for i in range(len(widths) - 1):
            x, y = np.meshgrid(np.arange(starts[i], starts[i + 1]), np.arange(starts[i + 1], starts[i + 2]))
            keep = rng.random(x.size) < (1.0 if x.size < 20000 else 0.2)
            a.append(x.ravel()[keep])
            b.append(y.ravel()[keep])
        p = rng.permutation(starts[-1])
        return csr(int(starts[-1]), p[np.concatenate(a)], p[np.concatenate(b)])
    # a core with a tail of trees: many peeling levels
    n = 9000
    u = rng.zipf(1.3, 150000) % n
    v = rng.zipf(1.3, 150000) % n
    p = rng.permutation(n)
    return csr(n, p[u], p[v])


@pytest.mark.parametrize("kind", ["one", "two", "clique", "path", "rows", "layers", "zipf"])
def test_frontier_edges(gpu, O, kind):
    pc = gpu
    vl, el = build(kind)
    n = vl.size - 1
    rng = np.random.default_rng(3)
    lo, hi = np.repeat(np.arange(n), np.diff(vl).astype(np.int64)), el.astype(np.int64)
    w = ((np.minimum(lo, hi) * 7919 + np.maximum(lo, hi) * 104729) % 255).astype(np.int32)  # 0..254, symmetric
    g = pc.Graph(vlist=vl, elist=el, weights=w)
    views = [(pc.Partitioned_Graph(g, None), None)]
    if n > 2:
        part = rng.integers(0, 5, n).astype(np.int32)
        pg = pc.Partitioned_Graph(g, part)
        pg.reorder()
        views.append((pg, pg.vertex_map()))  # old -> new ids
    core, prio = O.kcore(vl, el)[0], pc.vertex_priority(5, n)
    for pg, o2n in views:
        api = (lambda x: x) if o2n is None else (lambda x, m=np.argsort(o2n): x[m])
        for src in sorted({0, n // 3, n - 1}):
            s = src if o2n is None else int(o2n[src])
            np.testing.assert_array_equal(pg.solve_bfs(s), api(O.bfs(vl, el, src)))
            want = api(O.sssp(vl, el, w, src))
            for method, delta in ((pc.SSSP_AUTO, 0), (pc.SSSP_BELLMAN_FORD, 0), (pc.SSSP_DELTA_STEPPING, 3),
                                  (pc.SSSP_DELTA_STEPPING, 100), (pc.SSSP_DELTA_STEPPING, INT_MAX)):
                np.testing.assert_array_equal(pg.solve_sssp(s, method=method, delta=delta), want)
        np.testing.assert_array_equal(pg.solve_kcore(), api(core))
        if o2n is None:  # priorities are the caller's ids
            np.testing.assert_array_equal(pg.solve_mis(), O.mis(vl, el))
            np.testing.assert_array_equal(pg.solve_mis(seed=5), O.mis(vl, el, priority=prio))
        pg.close()
    g.close()
