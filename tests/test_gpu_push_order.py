"""Push PageRank where the dynamic region's atomics start as soon as they are
launched (direct mode without a static region, staged chunks of one tile, with
and without static edges): every iteration's sums are cleared before the first
contribution arrives.  A lost contribution shows as a rank below the FP64
oracle's by much more than FP32 rounding."""
import numpy as np
import pytest

import onegraph_gb300 as og
import oracle

pytestmark = pytest.mark.gpu

MODES = {
    "direct_no_static": dict(direct=True, no_static=True),
    "direct": dict(direct=True, advisek=0.5),
    "staged_no_static": dict(no_static=True),
    "staged": dict(advisek=0.02),
}


@pytest.mark.parametrize("V,E", [(4000, 60_000), (1_500_001, 3_000_000)])
@pytest.mark.parametrize("mode", list(MODES))
def test_push_sums_start_from_zero(mode, V, E):
    rng = np.random.default_rng(V)
    src = np.sort(rng.integers(0, V, E))
    off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=V))]).astype(np.uint64)
    col = rng.integers(0, V, E).astype(np.uint32)
    outdeg = np.bincount(col, minlength=V).astype(np.uint32)
    iters = 8
    want, _, _ = oracle.pr_l1(off, col, outdeg, 0.85, 0.0, iters)
    g = og.Graph.from_arrays(off, col, outdeg, kind=og.PR)
    t = g.transpose()
    kw = MODES[mode]
    flags = og.CFG_PR | (og.CFG_DIRECT if "direct" in kw else 0) | (og.CFG_NO_STATIC if "no_static" in kw else 0)
    p = t.plan(budget=1 << 40, flags=flags)
    # direct: two fifths of the records; staged: two buffers of a tile and a little
    edges = E * 2 // 5 * p["edge_bits"] // 8 if "direct" in kw else 2 * 2048 * p["stage_edge_bytes"] + 4096
    e = og.Engine(t, budget=p["vertex_bytes"] + p["fixed_bytes"] + edges, pagerank=True, **kw)
    assert e.plan["dynamic_edges"] > 0
    for _ in range(3):
        r = e.pr_l1_push(0.85, 0.0, iters)
        # FP32 sums of a vertex's contributions: each addition rounds by 2^-24 of the sum, the
        # error of an iteration is damped by 0.85 in the next ones
        deg = np.diff(off.astype(np.int64))
        bound = (deg.max() + 8) * 2.0 ** -24 / (1 - 0.85) * want.max()
        assert np.abs(r - want).max() <= bound
        assert e.stats["iterations"] == iters
    e.close()
