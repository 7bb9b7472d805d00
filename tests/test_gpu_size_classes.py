"""Graphs on both sides of the sizes where the pull sweeps' row classes and the
persistent kernels' grids change (2^22, 2^24 and 2^26 entries), against the oracle.

The tolerances of PageRank over k iterations: fp64 sums of up to 2^18 terms in any
order are within 2^18 2^-53 = 3e-11 of each other and errors shrink by the damping
from one iteration to the next, so 1e-9; fp32 vectors add 2^-24 an iteration, at
most 2^-24 / (1 - 0.85) + 2^-24 = 4.6e-7 in all, so 1e-6."""
from __future__ import annotations

import json

import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu

BOUNDS = (64, 128, 512, 1024, 2048)  # every bound of a row class


def check_pull(pc, O, pg, vl, el, iters=4):
    n = vl.size - 1
    want = O.pagerank_f64(vl, el, 0.85, iters)
    np.testing.assert_allclose(pg.page_rank(0.85, iters, fp64=True), want, rtol=1e-9, atol=0)
    np.testing.assert_allclose(pg.page_rank(0.85, iters), want, rtol=1e-6, atol=0)
    labels = np.random.default_rng(2).permutation(n).astype(np.int32)
    np.testing.assert_array_equal(pg.solve_cdlp(labels, 3), O.cdlp(vl, el, labels, 3))


@pytest.mark.parametrize("entries", [1 << 20, 5 << 20, 17 << 20, 68 << 20])
def test_rows_around_the_class_bounds(gpu, O, entries):
    """Random rows of about 40 entries, and rows of d - 1, d and d + 1 entries for every bound d."""
    pc = gpu
    rng = np.random.default_rng(entries)
    n = entries // 40 | 1
    special = [d + o for d in BOUNDS for o in (-1, 0, 1)]
    ids = rng.permutation(n)
    centres, leaves, rest = ids[:len(special)], ids[len(special):len(special) + 3000], ids[len(special) + 3000:]
    a = [np.full(s, c) for s, c in zip(special, centres)]
    b = [rng.choice(leaves, s, replace=False) for s in special]
    k = entries // 2
    a.append(rest[rng.integers(0, rest.size, k)])
    b.append(rest[rng.integers(0, rest.size, k)])
    g = pc.Graph.from_edges(np.concatenate(a), np.concatenate(b), n, relabel=False)
    vl, el = g.get_csr_vlist(), g.get_csr_elist()
    deg = np.diff(vl.astype(np.int64))
    assert deg[centres].tolist() == special
    assert 0.9 * entries < el.size < 1.02 * entries + 20000
    pg = pc.Partitioned_Graph(g, None)
    check_pull(pc, O, pg, vl, el)
    pg.close()
    g.close()


@pytest.mark.parametrize("relabel", [True, False])
def test_all_frontier_algorithms_past_2_24_entries(gpu, O, relabel):
    pc = gpu
    vl, el, _ = pc.HostCSR.rmat(20, 16, 7, relabel=relabel).arrays()
    n = 1_000_003  # not a power of two, the last vertices cut off
    row = np.repeat(np.arange(vl.size - 1, dtype=np.int32), np.diff(vl.astype(np.int64)))
    keep = (row < n) & (el < n)
    row, el = row[keep], el[keep]
    vl = np.zeros(n + 1, np.uint64)
    np.cumsum(np.bincount(row, minlength=n), out=vl[1:])
    assert el.size > 1 << 24
    lo, hi = np.minimum(row, el).astype(np.int64), np.maximum(row, el).astype(np.int64)
    w = ((lo * 7919 + hi * 104729) % 255).astype(np.int32)
    g = pc.Graph(vlist=vl, elist=el, weights=w)
    pg = pc.Partitioned_Graph(g, pc.equal_vertex_partition(n, 64))
    check_pull(pc, O, pg, vl, el)
    hub = int(np.argmax(np.diff(vl.astype(np.int64))))
    for src in (hub, n - 1):
        np.testing.assert_array_equal(pg.solve_bfs(src), O.bfs(vl, el, src))
    want = O.sssp(vl, el, w, hub)
    for method, delta in ((pc.SSSP_AUTO, 0), (pc.SSSP_BELLMAN_FORD, 0), (pc.SSSP_DELTA_STEPPING, 40)):
        np.testing.assert_array_equal(pg.solve_sssp(hub, method=method, delta=delta), want)
    np.testing.assert_array_equal(pg.solve_kcore(), O.kcore(vl, el)[0])
    np.testing.assert_array_equal(pg.solve_mis(), O.mis(vl, el))
    np.testing.assert_array_equal(pg.solve_mis(seed=9), O.mis(vl, el, priority=pc.vertex_priority(9, n)))
    pg.close()
    g.close()


def test_rmat22_pull(gpu, O):
    """Past 2^26 entries, degree-ordered: hub rows of 10^5 entries."""
    pc = gpu
    g = pc.Graph.rmat_device(22, 16, 1)
    vl, el = g.get_csr_vlist(), g.get_csr_elist()
    assert el.size > 1 << 26
    pg = pc.Partitioned_Graph(g, pc.equal_vertex_partition(vl.size - 1, 256))
    check_pull(pc, O, pg, vl, el)
    pg.close()
    g.close()


def test_per_edge_counts_with_binned_items(gpu, O):
    """All-edge Jaccard where the items are in the order of their in-neighbours' rows
    (rows beyond L2): rows of all lengths against the oracle, and the counts behind
    all values add up to six times the triangles."""
    pc = gpu
    g = pc.Graph.rmat_device(22, 16, 1)
    vl, el = g.get_csr_vlist(), g.get_csr_elist()
    n = vl.size - 1
    pg = pc.Partitioned_Graph(g, pc.equal_vertex_partition(n, 61))
    jac = np.asarray(pg.jaccard_edges())
    off = vl.astype(np.int64)
    rows = np.unique(np.geomspace(1, n - 1, 400).astype(np.int64))
    rows = rows[np.diff(off)[rows] <= 4096]  # a longer row takes the oracle minutes
    want = O.jaccard_rows(vl, el, rows)
    got = np.concatenate([jac[off[u]:off[u + 1]] for u in rows])
    np.testing.assert_array_equal(got, want)
    pinned = json.loads((GOLDEN / "pinned_counts.json").read_text())["rmat22_ef16_s1"]["T"]
    assert O.jaccard_audit(vl, el, jac) == (6 * pinned, 0, 0)
    pg.close()
    g.close()
