"""LCC where nearly every prefix id is a hit and lies past the ids with exact bits: the
hits are counted by the slot of the pivot set's hash.  Cliques smaller and larger
than the hash's 256 keys, with edges between them, ids shuffled or not, one and
many in-neighbours per item."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,count", [(3, 9000), (64, 400), (256, 60), (257, 60), (300, 50), (700, 3)])
@pytest.mark.parametrize("copy", [1, 0])
def test_cliques(gpu, O, size, count, copy):
    pc = gpu
    rng = np.random.default_rng(size)
    n = 9000 + size * count
    u, v = np.triu_indices(size, 1)
    base = 9000 + np.arange(count)[:, None] * size
    a = np.concatenate([(base + u).ravel(), rng.integers(0, n, 3 * n)])
    b = np.concatenate([(base + v).ravel(), rng.integers(0, n, 3 * n)])
    for p in (np.arange(n), rng.permutation(n)):
        x, y = p[a[a != b]], p[b[a != b]]
        key = np.unique(np.concatenate([x * n + y, y * n + x]))
        vl = np.zeros(n + 1, np.uint64)
        np.cumsum(np.bincount(key // n, minlength=n), out=vl[1:])
        el = (key % n).astype(np.int32)
        want, saved = O.lcc(vl, el), pc.selector.get_heuristic()
        g = pc.Graph(vlist=vl, elist=el)
        pc.selftest_limits(oriented_copy=copy)
        try:
            pg = pc.Partitioned_Graph(g, pc.equal_vertex_partition(n, 3))
            np.testing.assert_array_equal(pg.solve_lcc_merge(), want)
            pc.selector.set_heuristic([np.inf] * 4)  # the hash variant everywhere it can run
            np.testing.assert_array_equal(pg.solve_lcc_merge(), want)
            pg.close()
        finally:
            pc.selftest_limits()
            pc.selector.set_heuristic(saved)
        g.close()
