"""Delta PageRank over partial lists in direct mode, whose records are read over
the host link in position order and handed to their owners: tiles of one
vertex, of one-edge vertices, partial last tiles, records of 12 to 49 bits.
The staged engine gathers the same columns first and adds them in the same
order, so ranks agree bit for bit."""
import numpy as np
import pytest

import onegraph_gb300 as og

from test_gpu_stage_round import pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,hub,wmax", [(2049, 2048, 0), (5000, 9001, 0), (4097, 0, 64), (70_001, 30_000, 0xFFFFFFFF),
                                        (300_007, 2047, 64)])
def test_direct_delta_equals_staged(V, hub, wmax):
    rng = np.random.default_rng(V)
    deg = np.where(rng.random(V) < 0.5, 1, rng.integers(0, 40, V))
    deg[V // 3] = hub
    off = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint64)
    col = rng.integers(0, V, int(off[-1])).astype(np.uint32)
    if wmax:
        w = rng.integers(1, wmax + 1, col.size).astype(np.uint32)
        w[0], w[-1] = 1, wmax
        g = og.Graph.from_arrays(off, np.stack([col, w], 1), kind=og.WEIGHTED)
    else:
        g = og.Graph.from_arrays(off, col, np.maximum(np.bincount(col, minlength=V), 1).astype(np.uint32), kind=og.PR)
    a, b = pair(g, 6, pagerank=bool(wmax))
    for thr, rounds in ((0.2, 2), (0.05, 4), (0.001, 0)):
        np.testing.assert_array_equal(a.pr(thr, rounds), b.pr(thr, rounds))
        assert a.stats["iterations"] == b.stats["iterations"]
        assert a.stats["frontier_sum"] == b.stats["frontier_sum"]
    assert a.stats["frontier_sum"] < V * a.stats["iterations"]  # partial lists were among them
    a.close(), b.close(), g.close()
