"""The default configuration of batched BFS on both sides of the edge counts at
which it changes: directed graphs (2^20), symmetric ones with and without
bottom-up levels; depths of every source against single-source queries, checks
against the depths."""
import numpy as np
import pytest

import onegraph_gb300 as og

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,E,direct", [
    (40_001, (1 << 20) - 1, False), (40_001, 1 << 20, False), (300_007, 1 << 20, True), (1000, (1 << 20) + 5, False),
])
def test_directed(V, E, direct):
    rng = np.random.default_rng(E)
    src = np.sort((rng.random(E) ** 2 * V).astype(np.int64))
    off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=V))]).astype(np.uint64)
    check(og.Graph.from_arrays(off, rng.integers(0, V, E).astype(np.uint32)), direct, og.BFS_AUTO, rng)


@pytest.mark.parametrize("direction", [og.BFS_AUTO, og.BFS_TOP_DOWN])
def test_symmetric(direction):
    check(og.Graph.rmat(17, 12, on_gpu=True), True, direction, np.random.default_rng(7))


def check(g, direct, direction, rng):
    kw = {}
    if direct:
        p = g.plan(budget=1 << 40, flags=og.CFG_DIRECT | og.CFG_BATCH)
        kw = dict(budget=p["vertex_bytes"] + p["fixed_bytes"] + g.E * p["edge_bits"] // 16, advisek=0.7, direct=True)
    e = og.Engine(g, batch=True, **kw)
    e.set_param(og.PARAM_BFS_DIRECTION, direction)
    for n in (1, 5, 64):
        srcs = rng.integers(0, g.V, n).astype(np.uint32)
        depths, checks = e.bfs_batch(srcs)
        for i, s in enumerate(srcs):
            np.testing.assert_array_equal(depths[i], e.bfs(int(s)))
            reached = depths[i][depths[i] <= g.V]
            assert checks[i].tolist() == [reached.size, int(reached.astype(np.int64).sum())]
        _, again = e.bfs_batch(srcs, out=False)
        np.testing.assert_array_equal(again, checks)
    e.close()
