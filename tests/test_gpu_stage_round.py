"""Staged rounds (one launch over a ring of tile slots): rings of two slots up
to the most in use, lists of fewer tiles than the ring and of many rings,
partial last tiles, every record type.  Outputs equal those of direct mode
over the same split; PageRank sums every tile the same way in both modes."""
import numpy as np
import pytest

import onegraph_gb300 as og

from test_gpu_engine import budget_for

pytestmark = pytest.mark.gpu


def arrays(V, E, seed):
    rng = np.random.default_rng(seed)
    src = np.sort(rng.integers(0, V, E))
    src[: E // 9] = src[0]  # one vertex over many tiles
    src.sort()
    off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=V))]).astype(np.uint64)
    return off, rng.integers(0, V, E).astype(np.uint32), rng


def pair(g, slots, **kw):
    """Staged and direct engines without a static region; the staged one has room for `slots` staged tiles."""
    flags = og.CFG_NO_STATIC | (og.CFG_PR if kw.get("pagerank") else 0)
    p = g.plan(budget=1 << 40, flags=flags)
    room = slots * 2048 * p["stage_edge_bytes"]
    staged = og.Engine(g, budget=p["vertex_bytes"] + p["fixed_bytes"] + room + 4096, no_static=True, **kw)
    direct = og.Engine(g, budget=1 << 30, no_static=True, direct=True, **kw)
    tiles = (g.E + 2047) // 2048
    assert staged.plan["chunk_edges"] == 2048 * min(slots // 2, tiles), staged.plan
    return staged, direct


@pytest.mark.parametrize("V,E,slots", [
    (1000, 2047, 2),            # one tile
    (3000, 100001, 2),          # two slots: gather and relax alternate
    (3000, 100001, 6),
    (50000, 4096 * 40, 8),      # full last tile
    (50000, 1000003, 126),
    (20000, 9000001, 3000),     # more staging than the ring uses; second buffer partly used
    (20000, 9000001, 8800),     # ring within the first buffer
])
def test_staged_equals_direct(V, E, slots):
    off, col, rng = arrays(V, E, V + slots)
    src = int(np.argmax(np.diff(off.astype(np.int64))))
    g = og.Graph.from_arrays(off, col)
    a, b = pair(g, slots)
    np.testing.assert_array_equal(a.bfs(src), b.bfs(src))
    assert a.stats["edges_dynamic"] == b.stats["edges_dynamic"] and a.stats["edges_static"] == 0
    np.testing.assert_array_equal(a.cc(), b.cc())
    a.close(), b.close(), g.close()
    for wmax in (200, 60000, 1 << 20):
        w = rng.integers(1, wmax + 1, E).astype(np.uint32)
        w[0] = wmax
        g = og.Graph.from_arrays(off, np.stack([col, w], 1), kind=og.WEIGHTED)
        a, b = pair(g, slots)
        np.testing.assert_array_equal(a.sssp(src), b.sssp(src))
        a.close(), b.close(), g.close()
    g = og.Graph.from_arrays(off, col, np.maximum(np.bincount(col, minlength=V), 1).astype(np.uint32), kind=og.PR)
    a, b = pair(g, slots)
    np.testing.assert_array_equal(a.pr(max_rounds=5), b.pr(max_rounds=5))
    np.testing.assert_array_equal(a.pr_l1(0.85, 0.0, 3), b.pr_l1(0.85, 0.0, 3))
    a.close(), b.close(), g.close()
