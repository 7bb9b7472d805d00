"""A batch without room for the oriented copy scans the CSR, with the same results, and
so needs no more device memory than its CSR, 4 bytes per entry and 28 per vertex."""
from __future__ import annotations

import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT
from test_gpu_batch_shapes import graphs

pytestmark = pytest.mark.gpu


def arena(gs):
    voff = np.concatenate([[0], np.cumsum([vl.size - 1 for vl, _ in gs])]).astype(np.uint64)
    vls, els, m = [np.zeros(1, np.uint64)], [], 0
    for (vl, el), v0 in zip(gs, voff):
        vls.append(vl[1:] + np.uint64(m))
        els.append(el + np.int32(v0))
        m += el.size
    return np.concatenate(vls), np.concatenate(els), voff


@pytest.mark.parametrize("order", [0, 1])
def test_batch_on_the_csr(gpu, O, order):
    gs = graphs(order)
    gpu.selftest_limits(oriented_copy=0)
    try:
        b = gpu.Batch(*arena(gs))
    finally:
        gpu.selftest_limits()
    want = {"tc": np.array([O.tc_merge(*g) for g in gs], np.uint64), "lcc": np.concatenate([O.lcc(*g) for g in gs]),
            "bfs": np.concatenate([O.bfs(*g, 0) for g in gs])}
    for tasks in (1, 2, 3, 4, 5, 6, 7):
        r = b.run(tasks)
        for bit, key in ((1, "tc"), (2, "lcc"), (4, "bfs")):
            if tasks & bit:
                np.testing.assert_array_equal(r[key], want[key], err_msg=f"{key} of tasks {tasks}")
    b.close()


CHILD = """
import os, sys
sys.path[:0] = [{root!r}, {root!r} + "/tests"]
import numpy as np
import partitionandconquer_b200 as pc
from oracle import oracle as O
from test_gpu_batch_memory import arena
if {kind!r} == "paths":  # every inner vertex is a pivot with in-neighbours
    n = 5000
    a = np.arange(n, dtype=np.int32)
    el = np.stack([a - 1, a + 1], 1).ravel()[1:-1]
    vl = np.minimum(np.maximum(2 * np.arange(n + 1) - 1, 0), 2 * n - 2).astype(np.uint64)
    gs = [(vl, el)] * 40
else:
    gs = [pc.HostCSR.rmat(s, 8, s).arrays()[:2] for s in (8, 10, 12, 14)]
vl, el, voff = arena(gs)
N, M, G = vl.size - 1, el.size, voff.size - 1
need = 8 * (N + 1) + 4 * (M + 64) + 8 * (G + 1) + 4 * M + 28 * N + 16 * G + 64
os.environ["PC_MEMORY_LIMIT_MB"] = repr(need / 2**20)
r = pc.Batch(vl, el, voff).run(7)
np.testing.assert_array_equal(r["tc"], np.array([O.tc_merge(*g) for g in gs], np.uint64))
np.testing.assert_array_equal(r["lcc"], np.concatenate([O.lcc(*g) for g in gs]))
np.testing.assert_array_equal(r["bfs"], np.concatenate([O.bfs(*g, 0) for g in gs]))
"""


@pytest.mark.parametrize("kind", ["paths", "rmat"])
def test_memory_of_a_batch(gpu, kind):
    """In a process of its own, where the library holds nothing else."""
    r = subprocess.run([sys.executable, "-c", CHILD.format(root=str(ROOT), kind=kind)], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr
