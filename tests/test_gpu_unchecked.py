"""Counts of an adjacency that was not validated and is not symmetric: a scan of an
in-neighbour's row ends with the row, also where the pivot is not in it and where
the row has no smaller ids at all.  The count is the pivot form's, the triples
a < b < c with c in N(b), a in N(c) and a in N(b); every set variant and the
per-vertex mode must give it."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def directed(n, m, seed):
    rng = np.random.default_rng(seed)
    a, b = (n * rng.random(m) ** 2.5).astype(np.int64), (n * rng.random(m) ** 2.5).astype(np.int64)
    key = np.unique((a * n + b)[a != b])
    key = key[(key // n) % 5 != 3]  # rows without entries
    vl = np.zeros(n + 1, np.uint64)
    np.cumsum(np.bincount(key // n, minlength=n), out=vl[1:])
    return vl, (key % n).astype(np.int32)


def triples(vl, el):
    n = vl.size - 1
    rows = [el[int(vl[u]):int(vl[u + 1])] for u in range(n)]
    sets = [set(r.tolist()) for r in rows]
    t = np.zeros(n, np.int64)
    for b in range(n):
        for c in rows[b][rows[b] > b].tolist():
            for a in rows[c][rows[c] < b].tolist():
                if a in sets[b]:
                    t[a] += 1
                    t[b] += 1
                    t[c] += 1
    return t


@pytest.mark.parametrize("n,m", [(50, 900), (3000, 40000), (70001, 60000)])
def test_counts_of_a_directed_csr(gpu, n, m):
    pc = gpu
    vl, el = directed(n, m, n)
    t = triples(vl, el)
    assert t.sum() > 0
    deg = np.diff(vl).astype(np.float64)
    with np.errstate(divide="ignore", invalid="ignore"):
        lcc = np.where(deg < 1, 0.0, 2.0 * t / (deg * (deg - 1)))
    g = pc.Graph(vlist=vl, elist=el, validate=False)
    saved = pc.selector.get_heuristic()
    try:
        pg = pc.Partitioned_Graph(g, None)
        for name, v in pc.VARIANTS.items():
            if name != "matrix":
                assert pg.triangle_count(variant=v) == t.sum() // 3, name
        for p in ([0.0, 0.0, 0.0, np.inf], [0.0, np.inf, 0.0, np.inf], [0.0, np.inf, np.inf, np.inf],
                  [np.inf, np.inf, np.inf, np.inf]):
            pc.selector.set_heuristic(p)
            np.testing.assert_array_equal(pg.solve_lcc_merge(), lcc)
            assert np.asarray(pg.jaccard_edges()).size == el.size
        pg.close()
    finally:
        pc.selector.set_heuristic(saved)
        g.close()
