"""Device-driven rounds (one cooperative kernel per query, one CTA for small BFS
frontiers) where they hand over or fill up: frontiers of exactly the small
limits (4096 vertices, 16384 edges) and one more, hubs, long paths, layers that
grow past the limits and shrink again, isolated sources, vertex counts around
bitmap words and scan groups; results against the oracle and, for BFS, the
counters of the host-driven loop."""
import numpy as np
import pytest

import onegraph_gb300 as og
import oracle

from test_gpu_engine import budget_for

pytestmark = pytest.mark.gpu


def layered(widths, seed=0, extra=0):
    """Layer i + 1's vertices each have one neighbour in layer i (round robin),
    plus `extra` random edges between consecutive layers; symmetric."""
    rng = np.random.default_rng(seed)
    start = np.concatenate([[0], np.cumsum(widths)])
    us, vs = [], []
    for i in range(len(widths) - 1):
        a, b = start[i] + np.arange(widths[i]), start[i + 1] + np.arange(widths[i + 1])
        us.append(a[np.arange(b.size) % a.size])
        vs.append(b)
        if extra:
            us.append(rng.choice(a, extra))
            vs.append(rng.choice(b, extra))
    return csr(np.concatenate(us), np.concatenate(vs), int(start[-1]))


def csr(u, v, V):
    u, v = np.concatenate([u, v]), np.concatenate([v, u])
    key = np.unique(u.astype(np.int64) * V + v)
    off = np.concatenate([[0], np.cumsum(np.bincount(key // V, minlength=V))]).astype(np.uint64)
    return off, (key % V).astype(np.uint32)


GRAPHS = {
    "one": lambda: (np.zeros(2, np.uint64), np.zeros(0, np.uint32)),
    "pair": lambda: csr(np.array([0]), np.array([32]), 33),
    "path": lambda: layered([1] * 6001),
    "star4096": lambda: layered([1, 4096, 1]),
    "star4097": lambda: layered([1, 4097, 1]),
    "star_hub": lambda: layered([1, 20000]),
    "edges16384": lambda: layered([1, 64, 64 * 255]),   # 64 x 255 + 64 edges in the second level
    "edges_over": lambda: layered([1, 64, 64 * 257]),
    "grow_shrink": lambda: layered([1, 10, 300, 5000, 9000, 5000, 300] + [40] * 30 + [6000] * 6 + [7] * 20, 1, 2000),
}


@pytest.mark.parametrize("name", list(GRAPHS))
@pytest.mark.parametrize("mode", ["resident", "direct"])
def test_bfs_rounds(name, mode):
    off, col = GRAPHS[name]()
    V = off.size - 1
    g = og.Graph.from_arrays(off, col)
    if mode == "direct" and g.E < 8:
        pytest.skip("nothing to split")
    g.set_symmetric(True)
    kw = {} if mode == "resident" else dict(budget=budget_for(g, max(g.E // 3, 2048), og.CFG_DIRECT), advisek=0.5,
                                           direct=True)
    e = og.Engine(g, **kw)
    for direction in (og.BFS_TOP_DOWN, og.BFS_AUTO):
        e.set_param(og.PARAM_BFS_DIRECTION, direction)
        for s in sorted({0, V // 2, V - 1}):
            e.set_param(og.PARAM_LEVEL_LOOP, og.LOOP_AUTO)
            d = e.bfs(s)
            dev = dict(e.stats)
            np.testing.assert_array_equal(oracle.normalise_bfs(d, V), oracle.bfs(off, col, s)[0])
            np.testing.assert_array_equal(e.fetch(og.ALGO_BFS), d)
            e.set_param(og.PARAM_LEVEL_LOOP, og.LOOP_HOST)
            np.testing.assert_array_equal(e.bfs(s), d)
            for k in ("iterations", "frontier_sum", "edges_static", "edges_dynamic"):
                assert dev[k] == e.stats[k], (direction, s, k, dev[k], e.stats[k])
    e.close()


@pytest.mark.parametrize("name", list(GRAPHS))
@pytest.mark.parametrize("delta", [0, 1, 7, 4000000000])
def test_sssp_and_cc_rounds(name, delta):
    off, col = GRAPHS[name]()
    V = off.size - 1
    rng = np.random.default_rng(V)
    w = rng.integers(1, 65, col.size).astype(np.uint32)
    pairs = np.stack([col, w], 1)
    g = og.Graph.from_arrays(off, pairs, kind=og.WEIGHTED)
    modes = [{}]
    if g.E >= 8:
        modes.append(dict(budget=budget_for(g, max(g.E // 3, 2048), og.CFG_DIRECT), advisek=0.5, direct=True))
    for kw in modes:
        e = og.Engine(g, **kw)
        e.set_param(og.PARAM_SSSP_DELTA, delta)
        e.set_param(og.PARAM_CC_METHOD, og.CC_LABEL_PROPAGATION)
        for s in sorted({0, V - 1}):
            np.testing.assert_array_equal(e.sssp(s), oracle.sssp_dijkstra(off, pairs, s))
        if delta == 0:
            np.testing.assert_array_equal(e.cc(), oracle.cc(off, col)[0])
        e.close()
