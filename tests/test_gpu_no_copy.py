"""Triangle counts, LCC and all-edge Jaccard on the CSR itself, the path of views whose
oriented copy has no room (declined here by pc_selftest_limits): row starts and
ends at every place of a 16-byte vector, every set shape and variant, the matrix
form and its tails, partitions that are not id ranges, and rows of a directed
graph.  Against the oracle; whole numbers and single IEEE divisions, so equal."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_scan_edges import edge_graph
from test_gpu_unchecked import directed, triples

pytestmark = pytest.mark.gpu

PLANS = ([0.0, 0.0, 0.0, np.inf], [0.0, np.inf, 0.0, np.inf], [0.0, np.inf, np.inf, np.inf],
         [np.inf, np.inf, np.inf, np.inf], [0.0, 0.0, 0.0, 0.0])  # the last: matrix wherever it can run


@pytest.fixture
def plans(gpu):
    gpu.selftest_limits(oriented_copy=0)
    saved = gpu.selector.get_heuristic()
    yield PLANS
    gpu.selector.set_heuristic(saved)
    gpu.selftest_limits()


def check(pc, plans, vl, el, t, lcc, jac, v2ps):
    g = pc.Graph(vlist=vl, elist=el)
    for v2p in v2ps:
        pg = pc.Partitioned_Graph(g, v2p)
        for name, v in pc.VARIANTS.items():
            if name != "matrix":
                got, st = pg.triangle_count(variant=v, stats=True)
                assert got == t, name
                assert st.variant_hist[v] == sum(st.variant_hist)  # the variant asked for is the one that ran
        for p in plans:
            pc.selector.set_heuristic(p)
            assert pg.triangle_count() == t, p
            np.testing.assert_array_equal(pg.solve_lcc_merge(), lcc)
            np.testing.assert_array_equal(pg.jaccard_edges(), jac)
        pg.close()
    g.close()


@pytest.mark.parametrize("n", [3000, 20011, 70001])
def test_scan_edges(gpu, O, plans, n):
    vl, el = edge_graph(n, n)
    check(gpu, plans, vl, el, O.tc_merge(vl, el), O.lcc(vl, el), O.jaccard_edges(vl, el),
          (None, gpu.equal_vertex_partition(n, 7), (np.arange(n) % 5).astype(np.int32)))


@pytest.mark.parametrize("relabel", [True, False])
def test_rmat(gpu, O, plans, relabel):
    vl, el, _ = gpu.HostCSR.rmat(17, 16, 5, relabel=relabel).arrays()  # ids past 2^16: matrix tails, split sets
    check(gpu, plans, vl, el, O.tc_merge(vl, el), O.lcc(vl, el), O.jaccard_edges(vl, el), (None,))


def test_directed(gpu, plans):
    pc = gpu
    vl, el = directed(3000, 40000, 3000)
    t = triples(vl, el)
    g = pc.Graph(vlist=vl, elist=el, validate=False)
    pg = pc.Partitioned_Graph(g, None)
    for name, v in pc.VARIANTS.items():
        if name != "matrix":
            assert pg.triangle_count(variant=v) == t.sum() // 3, name
    deg = np.diff(vl).astype(np.float64)
    with np.errstate(divide="ignore", invalid="ignore"):
        lcc = np.where(deg < 1, 0.0, 2.0 * t / (deg * (deg - 1)))
    for p in plans[:4]:
        pc.selector.set_heuristic(p)
        np.testing.assert_array_equal(pg.solve_lcc_merge(), lcc)
    pg.close()
    g.close()
