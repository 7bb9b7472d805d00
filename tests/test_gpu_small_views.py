"""Many small graphs with views in use at once: a view's arena follows its graph's size."""
from __future__ import annotations

import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = """
import os, sys
sys.path[:0] = [{root!r}, {root!r} + "/tests"]
import numpy as np
import partitionandconquer_b200 as pc
from conftest import csr_from_edges
os.environ["PC_MEMORY_LIMIT_MB"] = "64"
vl, el = csr_from_edges(6, [(0, 1), (1, 2), (2, 0), (3, 4)])
keep = []
for _ in range(300):
    g = pc.Graph(vlist=vl, elist=el)
    pg = pc.Partitioned_Graph(g, None)
    assert pg.triangle_count() == 1
    assert pg.solve_bfs(0).tolist()[:3] == [-1, 1, 1]
    assert pg.solve_kcore().tolist() == [2, 2, 2, 1, 1, 0]
    keep.append((g, pg))
"""


def test_three_hundred_views_in_64_mb(gpu):
    """In a process of its own, where the library holds nothing else (4 MB a view: 1.2 GB)."""
    r = subprocess.run([sys.executable, "-c", CHILD.format(root=str(ROOT))], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
