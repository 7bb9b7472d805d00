"""k-core cascades of one vertex a round: long chains are peeled by one CTA, which
must not keep the others waiting at the step's barrier for the whole chain.  The
limit of 250 ms is far below the chain's 200,000 rounds (0.5 s) and far above the
2^14 rounds of a step (45 ms)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shuffled", [False, True])
def test_long_path(gpu, shuffled):
    n = 400_000
    p = np.random.default_rng(1).permutation(n) if shuffled else np.arange(n)
    a, b = np.concatenate([p[:-1], p[1:]]), np.concatenate([p[1:], p[:-1]])
    order = np.lexsort((b, a))
    vl = np.zeros(n + 1, np.uint64)
    np.cumsum(np.bincount(a, minlength=n), out=vl[1:])
    g = gpu.Graph(vlist=vl, elist=b[order].astype(np.int32))
    pg = gpu.Partitioned_Graph(g, None)
    gpu.selftest_limits(barrier_ms=250)
    try:
        np.testing.assert_array_equal(pg.solve_kcore(), np.ones(n, np.int32))
    finally:
        gpu.selftest_limits()
    pg.close()
    g.close()
