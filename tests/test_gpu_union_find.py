"""Sampling union-find CC: vertices with no, one and two neighbours, first
neighbours above and below their vertex, lists in any order, many components,
chains, record widths above 32 bits (single-word reads), labels bit for bit."""
import numpy as np
import pytest

import onegraph_gb300 as og
import oracle

from test_gpu_engine import configs
from test_gpu_rounds import GRAPHS, csr

pytestmark = pytest.mark.gpu


def forest(V, seed):
    """Random pairs joining about half of the vertices into small components."""
    rng = np.random.default_rng(seed)
    return csr(rng.integers(0, V, V // 3), rng.integers(0, V, V // 3), V)


CASES = dict(GRAPHS, forest=lambda: forest(50_001, 1),
             zigzag=lambda: csr(np.arange(10000) ^ 1, (np.arange(10000) * 7919 + 1) % 10000, 10000))


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("order", ["sorted", "reversed", "wide"])
def test_union_find_labels(name, order):
    off, col = CASES[name]()
    if order == "reversed":  # each list backwards
        row = np.repeat(np.arange(off.size - 1), np.diff(off.astype(np.int64)))
        col = col[np.lexsort((-col.astype(np.int64), row))]
    if order == "wide":
        w = np.full(col.size, 7, np.uint32)
        w[:1] = 0xFFFFFFFF
        g = og.Graph.from_arrays(off, np.stack([col, w], 1), kind=og.WEIGHTED)
    else:
        g = og.Graph.from_arrays(off, col)
    g.set_symmetric(True)
    want = oracle.cc(off, col)[0]
    for cname, kw in (configs(g) if g.E >= 8 else [("resident", {})]):
        e = og.Engine(g, **kw)
        e.set_param(og.PARAM_CC_METHOD, og.CC_UNION_FIND)
        np.testing.assert_array_equal(e.cc(), want, err_msg=cname)
        np.testing.assert_array_equal(e.cc(), want, err_msg=cname)
        e.close()
