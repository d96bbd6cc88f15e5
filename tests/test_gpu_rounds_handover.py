"""Rounds that the device-driven kernel hands over to launches of their own (more
than 4096 tiles of 2048 edges from HBM, 32768 over the link; bottom-up levels
of graphs from 2^24 vertices), between rounds that it runs itself: results and
counters are those of the host-driven loop, the relax timer covers both kinds."""
import numpy as np
import pytest

import onegraph_gb300 as og

pytestmark = pytest.mark.gpu

COUNTERS = ("iterations", "frontier_sum", "edges_static", "edges_dynamic")


def both(e, call):
    """The call by the device-driven rounds and by the host loop: (result, stats) each."""
    res = []
    for loop in (og.LOOP_AUTO, og.LOOP_HOST):
        e.set_param(og.PARAM_LEVEL_LOOP, loop)
        r = call()
        res.append((r, dict(e.stats)))
    e.set_param(og.PARAM_LEVEL_LOOP, og.LOOP_AUTO)
    return res


def engine(g, share):
    """All edges resident (share >= 1), or `share` of them and the rest over the link."""
    p = g.plan(budget=1 << 44, flags=og.CFG_DIRECT)
    e = og.Engine(g, budget=p["vertex_bytes"] + p["fixed_bytes"] + int(max(share, 0) * g.E * p["edge_bits"] / 8) + 65536,
                  advisek=1.0, direct=True, no_static=share == 0)
    assert (e.plan["dynamic_edges"] == 0) == (share >= 1)
    return e


@pytest.mark.parametrize("scale,ef,share", [
    (19, 16, 1.1),   # 8 thousand tiles a full round: handed over from HBM
    (19, 16, 0.9),   # both regions, mostly static
    (19, 16, 0.3),   # over the link: the kernel's own rounds
    (22, 16, 0.2),   # 62 thousand tiles, link
    (22, 16, 0),     # one region
    (20, 7, 1.1),    # about the limit: some rounds above it, some below
])
def test_handed_rounds_equal_the_host_loop(scale, ef, share):
    g = og.Graph.rmat(scale, ef, seed=scale, weight_seed=5, weighted=True, on_gpu=True)
    e = engine(g, share)
    src = int(np.argmax(g.degrees()))
    quiet = int(np.flatnonzero(g.degrees() == 1)[0])
    e.set_param(og.PARAM_CC_METHOD, og.CC_LABEL_PROPAGATION)
    e.set_param(og.PARAM_BFS_DIRECTION, og.BFS_TOP_DOWN)
    for s in (src, quiet):
        (d, ds), (h, hs) = both(e, lambda: e.bfs(s))
        np.testing.assert_array_equal(d, h)
        assert [ds[k] for k in COUNTERS] == [hs[k] for k in COUNTERS]
        for delta in (0, 4, 4000000000):
            e.set_param(og.PARAM_SSSP_DELTA, delta)
            (d, ds), (h, hs) = both(e, lambda: e.sssp(s))
            np.testing.assert_array_equal(d, h)
    (d, ds), (h, hs) = both(e, lambda: e.cc())
    np.testing.assert_array_equal(d, h)
    handed = scale == 22 or share >= 0.9 and ef == 16
    assert (ds["launches"] > 1) if handed else share >= 1 or ds["launches"] == 1
    # the timer: on or off, the results are the same, and the time lies within the query's
    e.set_param(og.PARAM_RELAX_TIMER, 1)
    np.testing.assert_array_equal(e.cc(), h)
    assert 0 < e.stats["ms_relax"] <= e.stats["ms_dynamic"] * 1.001 <= e.stats["ms_total"] * 1.001
    e.set_param(og.PARAM_RELAX_TIMER, 0)
    e.cc()
    assert e.stats["ms_relax"] == 0
    e.close()


@pytest.mark.parametrize("V,share", [((1 << 24) - 1, 1.1), (1 << 24, 1.1), ((1 << 24) + 33, 0.4)])
def test_bottom_up_levels(V, share):
    """A hub with half of the vertices around it, each of which has one of the
    other half: around the vertex count from which a bottom-up level is a launch
    of its own.  An even V leaves the last vertex alone."""
    half = (V - 1) // 2
    i = np.arange(1, half + 1, dtype=np.uint32)
    col = np.concatenate([i, np.stack([np.zeros(half, np.uint32), i + np.uint32(half)], 1).ravel(), i])
    deg = np.concatenate([[half], np.full(half, 2), np.ones(half, np.int64), np.zeros(V - 1 - 2 * half, np.int64)])
    off = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint64)
    g = og.Graph.from_arrays(off, col)
    g.set_symmetric(True)
    e = engine(g, share)
    want = np.full(V, V + 1, np.uint32)
    want[0], want[1:half + 1], want[half + 1:2 * half + 1] = 1, 2, 3
    (d, ds), (h, hs) = both(e, lambda: e.bfs(0))
    np.testing.assert_array_equal(d, want)
    np.testing.assert_array_equal(h, want)
    assert [ds[k] for k in COUNTERS] == [hs[k] for k in COUNTERS]
    (d, ds), (h, hs) = both(e, lambda: e.bfs(2 * half))
    np.testing.assert_array_equal(d, h)
    assert d[2 * half] == 1 and d[half] == 2 and d[0] == 3 and d[half + 1] == 5
    assert [ds[k] for k in COUNTERS] == [hs[k] for k in COUNTERS]
    e.close()
