"""Triangles of a graph whose rows L2 does not hold, where the bitmap items are
taken in the order of their in-neighbours' rows: the per-vertex counts must add
up to three times the pinned count (2 t(u) = lcc(u) d(u) (d(u) - 1), a whole
number that fp64 holds), with one and with many partitions."""
from __future__ import annotations

import json

import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("parts", [1, 61])
def test_per_vertex_counts_add_up(gpu, parts):
    rec = json.loads((GOLDEN / "pinned_counts.json").read_text())["rmat22_ef16_s1"]
    g = gpu.Graph.rmat_device(*rec["args"])
    deg = np.diff(g.get_csr_vlist().astype(np.int64)).astype(np.float64)
    pg = gpu.Partitioned_Graph(g, gpu.equal_vertex_partition(rec["n"], parts))
    assert pg.triangle_count() == rec["T"]
    lcc = np.asarray(pg.solve_lcc_merge())
    twice = np.where(deg > 1, np.nan_to_num(lcc) * deg * (deg - 1), 0.0)
    assert int(np.rint(twice / 2).astype(np.int64).sum()) == 3 * rec["T"]
    pg.close()
    g.close()
