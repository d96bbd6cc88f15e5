"""Rounds whose two regions are compacted in one launch: a split inside a bitmap
word, on a word boundary, one empty region, an empty frontier.  The host loop
and multi-source SSSP read their counts from it; results equal those of a
fully resident engine."""
import numpy as np
import pytest

import onegraph_gb300 as og

from test_gpu_engine import budget_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,split", [(1000, 0), (1000, 500), (1000, 512), (1000, 1000), (40000, 8191), (40000, 32768)])
def test_split_places(V, split):
    """The vertices below `split` fit the static region, the next one does not."""
    rng = np.random.default_rng(V + split)
    deg = rng.integers(1, 6, V)
    if 0 < split < V:
        deg[split] = 200000
    off = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint64)
    E = int(off[-1])
    col = rng.integers(0, V, E).astype(np.uint32)
    w = rng.integers(1, 65, E).astype(np.uint32)
    w[0] = 64
    g = og.Graph.from_arrays(off, np.stack([col, w], 1), kind=og.WEIGHTED)
    ref = og.Engine(g, budget=1 << 28, advisek=1.0, sssp_batch=4)
    kw = dict(budget=1 << 28, advisek=1.0)
    if split == 0:
        kw = dict(budget=1 << 28, no_static=True, direct=True)
    elif split < V:
        kw = dict(budget=budget_for(g, int(off[split]) + 16, og.CFG_DIRECT | og.CFG_SSSP_BATCH(4)), advisek=1.0,
                  direct=True)
    e = og.Engine(g, sssp_batch=4, **kw)
    assert e.plan["static_vertices"] == split
    srcs = [0, V - 1, V // 2, min(split, V - 1)]
    want = [ref.sssp(s) for s in srcs]
    got, _ = e.sssp_batch(srcs)
    for i in range(4):
        np.testing.assert_array_equal(got[i], want[i])
    e.set_param(og.PARAM_LEVEL_LOOP, og.LOOP_HOST)
    for s, x in zip(srcs, want):
        np.testing.assert_array_equal(e.sssp(s), x)
        np.testing.assert_array_equal(e.bfs(s), ref.bfs(s))
    e.close(), ref.close(), g.close()
