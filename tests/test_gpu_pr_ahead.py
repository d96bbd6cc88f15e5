"""PageRank iterations launched ahead of the host's check: how many, and what the
statistics say about their time."""
import numpy as np
import pytest

import onegraph_gb300 as og

from test_gpu_engine import budget_for

pytestmark = pytest.mark.gpu

PER_ITERATION = 4  # pull, fixup, update, end of the iteration


def graph(V, E, seed=0):
    rng = np.random.default_rng(seed)
    src = np.sort(rng.integers(0, V, E))
    off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=V))]).astype(np.uint64)
    col = (rng.random(E) ** 3 * V).astype(np.uint32)
    return og.Graph.from_arrays(off, col, np.maximum(np.bincount(col, minlength=V), 1).astype(np.uint32), kind=og.PR)


def test_launches_follow_the_tolerance():
    """A loose run after a tight one is not launched as far ahead as the tight
    one went: at most the first batch and the one that reaches the end."""
    g = graph(3000, 60_000)
    e = og.Engine(g)
    tight = e.pr_l1(0.85, 1e-9, 500)
    its, launches = e.stats["iterations"], e.stats["launches"]
    assert its > 40 and launches <= PER_ITERATION * (its + 4) + 8
    for damping, tol in ((0.85, 1e-1), (0.5, 1e-9), (0.85, 1e-3)):
        e.pr_l1(damping, tol, 500)
        n = e.stats["iterations"]
        assert n < its - 20, (damping, tol, n)
        assert e.stats["launches"] <= PER_ITERATION * max(n + 4, 8) + 8, (damping, tol, n, e.stats["launches"])
        again = e.stats["residual"]
        e.pr_l1(damping, tol, 500)  # the same again: known how far
        assert e.stats["iterations"] == n and e.stats["residual"] == again
        assert e.stats["launches"] <= PER_ITERATION * n + 8
    np.testing.assert_array_equal(e.pr_l1(0.85, 1e-9, 500), tight)
    e.close()


@pytest.mark.parametrize("mode", ["resident", "direct"])
@pytest.mark.parametrize("V,E", [(2000, 30_000), (200_000, 3_000_000)])
def test_pull_times_are_measured(mode, V, E):
    """The first pull of an engine finds cold caches and code; times a number of
    iterations it would exceed the query's own time."""
    g = graph(V, E, 1)
    kw = {}
    if mode == "direct":
        kw = dict(budget=budget_for(g, E // 8, og.CFG_DIRECT), advisek=0.5, direct=True)
    per = []
    for _ in range(6):
        e = og.Engine(g, **kw)
        assert (e.plan["dynamic_edges"] > 0) == (mode == "direct")
        for its in (7, 100, 1):
            e.pr_l1(0.85, 0.0, its)
            st = e.stats
            pull = st["ms_dynamic"] + st["ms_static"]
            assert st["iterations"] == its and 0 < pull <= st["ms_total"], (its, st)
            assert (st["ms_dynamic"] == 0) == (mode == "resident") and (st["ms_static"] == 0) == (mode == "direct")
            if its == 100:
                per.append((pull / its, st["ms_total"] / its))
        e.close()
    # the pulls are most of an iteration on a graph of 15 edges a vertex, and never more than it
    assert V < 100_000 or all(p > 0.3 * t for p, t in per), per
