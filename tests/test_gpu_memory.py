"""The oriented copy never makes a call fail for want of device memory.  Under a limit
on it, the least memory is searched with which a call succeeds on a view without the
copy.  With that limit and with every one above it, the call must succeed, and give
the same result, on a view that may build the copy and on one that holds it."""
from __future__ import annotations

import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OOM = 2
STEP = 64 * 1024

CALLS = {
    "count": lambda pg: pg.triangle_count(),
    "lcc": lambda pg: pg.solve_lcc_merge(),
    "jaccard": lambda pg: pg.jaccard_edges(),
    "bfs": lambda pg: pg.solve_bfs(0),
    "sssp": lambda pg: pg.solve_sssp(0),
    "pagerank": lambda pg: pg.page_rank(0.85, 3),
    "pagerank64": lambda pg: pg.page_rank(0.85, 3, fp64=True),
    "kcore": lambda pg: pg.solve_kcore(),
    "mis": lambda pg: pg.solve_mis(seed=3),
    "cdlp": lambda pg: pg.solve_cdlp(np.arange(1 << 17, dtype=np.int32), 3),
}


class Runner:
    def __init__(self, pc, graph, call):
        self.pc, self.g, self.call = pc, graph, call

    def run(self, limit, copy, held):
        """The result with `limit` bytes for the library, None when it runs out of memory."""
        self.pc.selftest_limits(oriented_copy=copy)
        pg = self.pc.Partitioned_Graph(self.g, None)
        try:
            if held:
                pg.triangle_count()
            self.pc.selftest_limits(memory_bytes=limit, oriented_copy=copy)
            return self.call(pg)
        except self.pc.PCError as e:
            assert e.status == OOM, str(e)
            return None
        finally:
            self.pc.selftest_limits()
            pg.close()

    def least(self, held):
        lo, hi = 0, 1 << 34  # fails with lo, works with hi
        assert self.run(hi, False, held) is not None
        while hi - lo > STEP:
            mid = (lo + hi) // 2
            if self.run(mid, False, held) is None:
                lo = mid
            else:
                hi = mid
        return hi


@pytest.mark.parametrize("name", list(CALLS))
def test_no_call_needs_the_copy(gpu, name):
    gc.collect()
    g = gpu.Graph.rmat_device(17, 16, 3, wmax=255)  # 2^17 vertices
    copy = 4 * int(g.get_csr_elist().size)  # no less than its size
    r = Runner(gpu, g, CALLS[name])
    want = r.run(1 << 34, True, False)
    for held in (False, True):
        least = r.least(held)
        for more in (0, copy // 8, copy // 4, copy // 2, copy, 2 * copy):
            got = r.run(least + more, True, held)
            assert got is not None, (held, more)
            np.testing.assert_array_equal(got, want)
    g.close()


@pytest.mark.parametrize("name", ["count", "jaccard"])
def test_rows_beyond_l2(gpu, name):
    """... where the item lists may be put in another order, which takes as much again."""
    gc.collect()
    g = gpu.Graph.rmat_device(22, 16, 1)
    r = Runner(gpu, g, CALLS[name])
    want = r.run(1 << 34, True, False)
    least = r.least(False)
    for more in range(0, 1 << 30, 1 << 26):
        got = r.run(least + more, True, False)
        assert got is not None, more
        np.testing.assert_array_equal(got, want)
    g.close()
