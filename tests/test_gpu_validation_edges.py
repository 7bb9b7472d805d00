"""The upload's check of the adjacency at the edges of its chunks of 512 entries:
rows that start or end there, rows over many chunks, rows without entries, and
single wrong entries at the first and last places of a chunk and of its
vectors."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _star(leaves, gap):
    """Vertex 0 and its leaves, `gap` vertices without neighbours before each of them."""
    ids = 1 + gap + np.arange(leaves, dtype=np.int64) * (gap + 1)
    n = int(ids[-1]) + 1 + gap
    deg = np.zeros(n + 1, np.uint64)
    deg[1] = leaves
    deg[1 + ids] = 1
    return np.cumsum(deg, dtype=np.uint64), np.concatenate([ids, np.zeros(leaves)]).astype(np.int32), ids


def _clique(k):
    el = np.tile(np.arange(k, dtype=np.int32), (k, 1))
    return np.arange(0, k * (k - 1) + 1, k - 1, dtype=np.uint64), el[~np.eye(k, dtype=bool)]


@pytest.mark.parametrize("leaves", [1, 255, 256, 257, 512, 1500, 3_000_000])
@pytest.mark.parametrize("gap", [0, 3])
def test_star(gpu, leaves, gap):
    vl, el, ids = _star(leaves, gap)

    def status(p, v):
        bad = el.copy()
        bad[p] = v
        with pytest.raises(gpu.PCError) as e:
            gpu.Graph(vlist=vl, elist=bad)._device()
        assert e.value.status == 1
        return str(e.value)

    assert gpu.Graph(vlist=vl, elist=el).solve_triangle_counting_merge() == 0
    m = 2 * leaves
    places = [p for p in (0, 1, 127, 128, 511, 512, 1023, 1024, leaves - 1, leaves, m - 1) if p < m]
    for p in places if leaves < 10_000 else (511, 512, m - 1):
        assert "outside" in status(p, -1)
        assert "outside" in status(p, vl.size - 1)
        assert "self-loop" in status(p, 0 if p < leaves else ids[p - leaves])
        if 0 < p < leaves:
            assert "ascending" in status(p, el[p - 1])
        if p >= leaves and leaves > 1:  # a leaf that names another one
            assert "symmetric" in status(p, ids[p - leaves - 1])


@pytest.mark.parametrize("k", [2, 5, 129, 513, 600])
def test_clique(gpu, k):
    vl, el = _clique(k)
    assert gpu.Graph(vlist=vl, elist=el).solve_triangle_counting_merge() == k * (k - 1) * (k - 2) // 6
    for p in {q for q in (1, 127, 128, 511, 512, 1024, el.size - 1) if 0 < q < el.size and q not in vl}:
        bad = el.copy()
        bad[p - 1], bad[p] = el[p], el[p - 1]
        with pytest.raises(gpu.PCError) as e:
            gpu.Graph(vlist=vl, elist=bad)._device()
        assert "ascending" in str(e.value)
