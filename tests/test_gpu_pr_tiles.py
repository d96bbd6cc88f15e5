"""PageRank pull where its tiles can go wrong: vertices spanning several tiles,
a vertex ending exactly at a tile's end, one-edge vertices filling a tile, the
last partial tile, record widths up to 64 bits, contiguous and partial lists
(the delta form after vertices drop out), every region layout.  One iteration
of the L1 form is compared with the same sums in FP64: an FP32 sum of d
non-negative terms in any order is within d 2^-24 of it, relatively."""
import numpy as np
import pytest

import onegraph_gb300 as og

from test_gpu_engine import configs

pytestmark = pytest.mark.gpu


def graph(degrees, V, seed, weighted=False, wmax=64):
    """In-lists of the given lengths, then one-edge vertices up to V."""
    rng = np.random.default_rng(seed)
    deg = np.ones(V, np.int64)
    deg[:len(degrees)] = degrees
    off = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint64)
    col = rng.integers(0, V, int(off[-1])).astype(np.uint32)
    if weighted:
        w = rng.integers(1, wmax + 1, col.size).astype(np.uint32)
        w[0], w[-1] = 1, wmax
        return og.Graph.from_arrays(off, np.stack([col, w], 1), kind=og.WEIGHTED), off, col, deg
    od = np.bincount(col, minlength=V).astype(np.uint32)
    return og.Graph.from_arrays(off, col, od, kind=og.PR), off, col, od


@pytest.mark.parametrize("degrees,V,weighted,wmax", [
    ([2048, 2048, 1], 5000, False, 0),        # starts and ends on tile boundaries
    ([1, 2047, 0, 9001, 3, 0, 2049], 3001, False, 0),
    ([20000], 1111, False, 0),                # one vertex over ten tiles
    ([0, 5, 70000, 4], 40001, False, 0),
    ([100] * 50, 9000, True, 64),             # column and weight bits
    ([3000, 1], 70001, True, 0xFFFFFFFF),     # 17 + 32-bit records
])
def test_pull_tiles(degrees, V, weighted, wmax):
    g, off, col, od = graph(degrees, V, V, weighted, wmax)
    deg = np.diff(off.astype(np.int64))
    inv = np.where(od > 0, 1.0 / np.maximum(od, 1), 0.0) / V
    row = np.repeat(np.arange(V), deg)
    want = 0.15 / V + 0.85 * np.bincount(row, weights=inv[col], minlength=V)
    bound = want * (deg + 16) * 2.0 ** -24  # + 16: the rounding of 1/V, 1/outdeg, the update
    for cname, kw in configs(g, og.CFG_PR if weighted else 0):
        e = og.Engine(g, pagerank=weighted, **kw)
        r = e.pr_l1(0.85, 0.0, 1)
        assert (np.abs(r.astype(np.float64) - want) <= bound).all(), cname
        np.testing.assert_array_equal(r, e.pr_l1(0.85, 0.0, 1), err_msg=cname)
        e.close()


@pytest.mark.parametrize("V,seed", [(4097, 1), (33333, 2)])
def test_delta_form_with_a_partial_list(V, seed):
    """Two rounds of the delta form, the second over a partial list (the cursor
    form).  The threshold lies in the widest gap of the first round's changes,
    so FP32 and FP64 list the same vertices; a vertex whose second change is
    within 1e-3 of it may go either way and is left out."""
    rng = np.random.default_rng(seed)
    g, off, col, od = graph(list(rng.integers(0, 60, V // 2)) + [5000], V, seed)
    deg = np.diff(off.astype(np.int64))
    row = np.repeat(np.arange(V), deg)
    inv = np.where(od > 0, 1.0 / np.maximum(od, 1), 0.0)

    def pull(rank):
        return 0.15 + 0.85 * np.bincount(row, weights=(rank * inv)[col], minlength=V)

    r1 = pull(np.ones(V))
    d = np.sort(np.abs(r1 - 1.0))
    mid = d[V // 4: 3 * V // 4]
    k = int(np.argmax(np.diff(mid)))
    thr = float(mid[k] + mid[k + 1]) / 2
    assert mid[k + 1] - mid[k] > 1e-4
    act = np.abs(r1 - 1.0) > thr
    assert 0.1 < act.mean() < 0.9
    rank = np.where(act, r1, 1.0)
    r2 = pull(rank)
    d2 = np.abs(r2 - rank)
    want = np.where(act & (d2 > thr), r2, rank)
    sure = np.abs(d2 - thr) > 1e-3
    assert sure.mean() > 0.9
    # the error of the first round's ranks reaches the second through its sums
    bound = want * (2 * deg + deg.max() + 32) * 2.0 ** -24
    for cname, kw in configs(g):
        e = og.Engine(g, **kw)
        r = e.pr(thr, 2)
        assert (np.abs(r - want) <= bound)[sure].all(), cname
        e.close()
