"""Batches whose graphs differ in everything the kernel sizes by: graphs with
and without edges, of one vertex, past the ids with exact bits and with more
high ids in a pivot's set than its hash holds; every subset of the tasks.
Against the oracle, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def csr(n, a, b):
    a, b = a[a != b], b[a != b]
    key = np.unique(np.concatenate([a * n + b, b * n + a]))
    vl = np.zeros(n + 1, np.uint64)
    np.cumsum(np.bincount(key // n, minlength=n), out=vl[1:])
    return vl, (key % n).astype(np.int32)


def graphs(order):
    rng = np.random.default_rng(11)
    none = np.zeros(0, np.int64)
    out = [csr(1, none, none), csr(700, none, none), csr(2, np.array([0]), np.array([1]))]
    # hubs at the first ids, a path behind them (many BFS levels)
    out.append(csr(5000, np.concatenate([rng.zipf(1.5, 60000) % 5000, np.arange(4000, 4999)]),
                   np.concatenate([rng.integers(0, 4000, 60000), np.arange(4001, 5000)])))
    # a dense core of 700 ids past 2^13, a star over all of them
    core = rng.choice(np.arange(9000, 20000), 700, replace=False)
    u, v = np.triu_indices(700, 1)
    k = rng.random(u.size) < 0.6
    out.append(csr(20001, np.concatenate([core[u[k]], np.zeros(20000, np.int64)]),
                   np.concatenate([core[v[k]], np.arange(1, 20001)])))
    out.append(csr(300, *np.triu_indices(300, 1)))
    return out if order else out[::-1]


@pytest.mark.parametrize("order", [0, 1])
def test_batch_shapes(gpu, O, order):
    pc = gpu
    gs = graphs(order)
    voff = np.concatenate([[0], np.cumsum([vl.size - 1 for vl, _ in gs])]).astype(np.uint64)
    vls, els, m = [np.zeros(1, np.uint64)], [], 0
    for (vl, el), v0 in zip(gs, voff):
        vls.append(vl[1:] + np.uint64(m))
        els.append(el + np.int32(v0))
        m += el.size
    b = pc.Batch(np.concatenate(vls), np.concatenate(els), voff)
    want = {"tc": np.array([O.tc_merge(*g) for g in gs], np.uint64), "lcc": np.concatenate([O.lcc(*g) for g in gs]),
            "bfs": np.concatenate([O.bfs(*g, 0) for g in gs])}
    b.set_schedule(512 if order else 256, 2, order)
    for tasks in (1, 2, 3, 4, 5, 6, 7, 7):
        r = b.run(tasks)
        for bit, key in ((1, "tc"), (2, "lcc"), (4, "bfs")):
            if tasks & bit:
                np.testing.assert_array_equal(r[key], want[key], err_msg=f"{key} of tasks {tasks}")
            else:
                assert r[key] is None
        assert r["items"] == len(gs) * bin(tasks).count("1")
    b.close()
