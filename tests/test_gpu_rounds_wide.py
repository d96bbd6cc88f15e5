"""Device-driven rounds on graphs of 2^28 vertices and more, whose list
reservations give fewer bits to edges: a path, a star and a few random edges
among many isolated vertices, against the same small graph."""
import numpy as np
import pytest

import onegraph_gb300 as og
import oracle

from test_gpu_rounds import layered

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [(1 << 28) - 1, 1 << 28, (1 << 28) + 33])
def test_wide_graph(V):
    """The small graph's vertices are spread over the wide one's ids in order."""
    soff, scol = layered([1] * 20 + [5000, 3, 40_000, 1], 2, 500)
    n = soff.size - 1
    ids = np.linspace(0, V - 1, n).astype(np.int64)
    deg = np.zeros(V + 1, np.uint64)
    deg[ids + 1] = np.diff(soff)
    off = np.cumsum(deg, dtype=np.uint64)
    col = ids[scol].astype(np.uint32)
    w = np.random.default_rng(1).integers(1, 65, col.size).astype(np.uint32)
    g = og.Graph.from_arrays(off, np.stack([col, w], 1), kind=og.WEIGHTED)
    g.set_symmetric(True)
    e = og.Engine(g, budget=64 << 30, advisek=1.0)
    for direction in (og.BFS_TOP_DOWN, og.BFS_AUTO):
        e.set_param(og.PARAM_BFS_DIRECTION, direction)
        d = e.bfs(int(ids[0]))
        assert e.stats["launches"] < e.stats["iterations"]  # device-driven, not a launch or more a round
        assert (d == V + 1).sum() == V - n
        np.testing.assert_array_equal(oracle.normalise_bfs(np.where(d[ids] == V + 1, n + 1, d[ids]).astype(np.uint32), n),
                                      oracle.bfs(soff, scol, 0)[0])
    for delta in (0, 8):
        e.set_param(og.PARAM_SSSP_DELTA, delta)
        d = e.sssp(int(ids[0]))
        assert e.stats["launches"] < e.stats["iterations"]
        assert (d == 0xFFFFFFFF).sum() == V - n
        np.testing.assert_array_equal(d[ids], oracle.sssp_dijkstra(soff, np.stack([scol, w], 1), 0))
    e.close()
