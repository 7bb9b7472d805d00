"""The bitmap kernels' scans at the sizes where they can go wrong: rows that
end at, before and after the bounds of a 16-byte vector, of a group's step and
of the hash's 256 keys, with pivots and prefix ids on both sides of every set's
bounds.  Counts, LCC and all-edge Jaccard against the oracle; the results are
whole numbers and single IEEE divisions of them, so they are equal."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 3, 4, 5, 7, 8, 9, 31, 32, 33, 127, 128, 129, 255, 256, 257, 258, 300]


def edge_graph(n, seed):
    """A dense random core of 400 ids spread over [0, n) around the sets'
    bounds, and for every length d two vertices adjacent to d core ids."""
    rng = np.random.default_rng(seed)
    marks = [x + o for x in (1 << 13, 1 << 15, 1 << 16) for o in (-2, -1, 0, 1, 2) if x + o < n - 50]
    core = np.unique(np.concatenate([np.arange(60), marks, rng.integers(0, n - 60, 400)]).astype(np.int64))
    u, v = np.triu_indices(core.size, 1)
    keep = rng.random(u.size) < 0.4
    src, dst = [core[u[keep]]], [core[v[keep]]]
    for i, d in enumerate(LENGTHS):
        for top, pick in ((n - 1 - i, core[:d]), (n - 1 - len(LENGTHS) - i, rng.permutation(core)[:d])):
            src.append(np.full(pick.size, top))
            dst.append(pick)
    a, b = np.concatenate(src), np.concatenate(dst)
    a, b = a[a != b], b[a != b]
    key = np.unique(np.concatenate([a * n + b, b * n + a]))
    vl = np.zeros(n + 1, np.uint64)
    np.cumsum(np.bincount(key // n, minlength=n), out=vl[1:])
    return vl, (key % n).astype(np.int32)


@pytest.mark.parametrize("n", [3000, 20011, 40001, 70001])
def test_scan_edges(gpu, O, n):
    pc = gpu
    vl, el = edge_graph(n, n)
    t, lcc, jac = O.tc_merge(vl, el), O.lcc(vl, el), O.jaccard_edges(vl, el)
    g = pc.Graph(vlist=vl, elist=el)
    saved = pc.selector.get_heuristic()
    try:
        for v2p in (None, pc.equal_vertex_partition(n, 7), (np.arange(n) % 5).astype(np.int32)):
            pg = pc.Partitioned_Graph(g, v2p)
            for name, v in pc.VARIANTS.items():
                if name != "matrix":
                    assert pg.triangle_count(variant=v) == t, name
            # every bitmap group size, then the hash variant everywhere it can run
            for p in ([0.0, 0.0, 0.0, np.inf], [0.0, np.inf, 0.0, np.inf], [0.0, np.inf, np.inf, np.inf],
                      [np.inf, np.inf, np.inf, np.inf]):
                pc.selector.set_heuristic(p)
                assert pg.triangle_count() == t, p
                np.testing.assert_array_equal(pg.solve_lcc_merge(), lcc)
                np.testing.assert_array_equal(pg.jaccard_edges(), jac)
            pg.close()
    finally:
        pc.selector.set_heuristic(saved)
        g.close()
