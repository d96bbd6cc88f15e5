"""The caller's result array: written once, with the whole result, and not at
all by a query that ends in an error."""
import threading

import numpy as np
import pytest

import onegraph_gb300 as og
import oracle

from test_gpu_engine import budget_for
from test_gpu_rounds import csr, layered

pytestmark = pytest.mark.gpu

SENTINEL = 0xA5A5A5A5


def graph(V, kind):
    """A ring with chords; V is no power of two, so a record of all ones holds
    a column that is no vertex."""
    rng = np.random.default_rng(V)
    off, col = csr(np.concatenate([np.arange(V), rng.integers(0, V, 6 * V)]),
                   np.concatenate([(np.arange(V) + 1) % V, rng.integers(0, V, 6 * V)]), V)
    if kind == og.WEIGHTED:
        return og.Graph.from_arrays(off, np.stack([col, rng.integers(1, 65, col.size).astype(np.uint32)], 1), kind=kind)
    return og.Graph.from_arrays(off, col)


@pytest.mark.parametrize("algo", ["bfs", "sssp", "cc"])
@pytest.mark.parametrize("V", [1003, 300_007])
@pytest.mark.parametrize("pinned", [False, True])
def test_error_leaves_the_array_alone(algo, V, pinned):
    """The kernels' bounds checks turn a column that is no vertex into
    OG_E_DEVICE.  The engine is created on records with such a column: some of
    the page-locked stream's words are all ones."""
    g = graph(V, og.WEIGHTED if algo == "sssp" else og.PLAIN)
    words = g.records()["words"]
    words[words.size // 2: words.size // 2 + 8] = 0xFFFFFFFF
    kw = dict(budget=budget_for(g, max(g.E // 4, 2048), og.CFG_DIRECT), advisek=0.1, direct=True)
    e = og.Engine(g, **kw)
    assert e.plan["static_edges"] < g.E // 2 - 64
    e.set_param(og.PARAM_CC_METHOD, og.CC_LABEL_PROPAGATION)
    out = og.pinned_empty(V, np.uint32) if pinned else np.empty(V, np.uint32)
    out[:] = SENTINEL
    for _ in range(2):
        with pytest.raises(og.OGError, match="out-of-range"):
            e.cc(out) if algo == "cc" else getattr(e, algo)(0, out)
        assert (out == SENTINEL).all()
    e.close()


def test_no_partial_result_between_passes():
    """A frontier that crosses the one-CTA limit (4096 vertices) ten times and
    stays small between, so that the search goes back and forth between the
    two kernels; a second thread looks at the array meanwhile."""
    widths = [1]
    for _ in range(10):
        widths += [6000, 6000] + [9] * 40
    off, col = layered(widths)
    V = off.size - 1
    g = og.Graph.from_arrays(off, col)
    g.set_symmetric(True)
    e = og.Engine(g)
    e.set_param(og.PARAM_BFS_DIRECTION, og.BFS_TOP_DOWN)
    out = og.pinned_empty(V, np.uint32)
    want = oracle.bfs(off, col, 0)[0]
    last = V - 1  # reached by the last level
    seen, stop = [], threading.Event()

    def watch():
        while not stop.is_set():
            if out[last] == V + 1:  # "unreached": a result of a search that had not ended
                seen.append(1)

    t = threading.Thread(target=watch)
    t.start()
    try:
        for _ in range(30):
            out[:] = SENTINEL
            e.bfs(0, out)
            assert out[last] == len(widths)
    finally:
        stop.set()
        t.join()
    assert not seen
    np.testing.assert_array_equal(oracle.normalise_bfs(out, V), want)
    e.close()


@pytest.mark.parametrize("V", [8, 32_767, 32_768, 32_769])
@pytest.mark.parametrize("direct", [False, True])
def test_both_ways_of_delivery(V, direct):
    """Results of up to 32768 vertices are stored by the kernel, larger ones are
    copied: page-locked, pageable, and left on the device."""
    g = graph(V, og.WEIGHTED)
    off, pairs = np.array(g.offsets), np.array(g.edges)
    col = pairs[:, 0].copy()
    kw = dict(budget=budget_for(g, max(g.E // 4, 2048), og.CFG_DIRECT), advisek=0.1, direct=True) if direct else {}
    e = og.Engine(g, **kw)
    e.set_param(og.PARAM_CC_METHOD, og.CC_LABEL_PROPAGATION)
    want = {"bfs": oracle.normalise_bfs(oracle.bfs(off, col, 1)[0], V), "sssp": oracle.sssp_dijkstra(off, pairs, 1),
            "cc": oracle.cc(off, col)[0]}
    calls = {"bfs": (lambda o: e.bfs(1, o), og.ALGO_BFS), "sssp": (lambda o: e.sssp(1, o), og.ALGO_SSSP),
             "cc": (lambda o: e.cc(o), og.ALGO_CC)}
    for name, (call, algo) in calls.items():
        for out in (np.full(V, SENTINEL, np.uint32), og.pinned_empty(V, np.uint32)):
            got = call(out)
            assert got is out
            np.testing.assert_array_equal(oracle.normalise_bfs(got, V) if name == "bfs" else got, want[name])
            np.testing.assert_array_equal(e.fetch(algo), got)
        assert call(False) is None
        got = e.fetch(algo)
        np.testing.assert_array_equal(oracle.normalise_bfs(got, V) if name == "bfs" else got, want[name])
    e.close()
