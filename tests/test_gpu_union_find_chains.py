"""Union-find CC on graphs whose first neighbours form long chains: grids
numbered by rows and columns, paths in order and backwards, combs, a grid with
permuted ids; labels bit for bit against the oracle's, and sizes on both sides
of what one sweep of the compression holds in flight."""
import numpy as np
import pytest

import onegraph_gb300 as og
import oracle

from test_gpu_rounds import csr

pytestmark = pytest.mark.gpu


def grid(w, h, perm=None):
    V = w * h
    rng = np.random.default_rng(V)
    i = np.arange(V)
    right, down = i[i % w != w - 1], i[i + w < V]
    u, v = np.concatenate([right, down]), np.concatenate([right + 1, down + w])
    keep = rng.random(u.size) < 0.9
    u, v = u[keep], v[keep]
    if perm is not None:
        p = np.random.default_rng(perm).permutation(V)
        u, v = p[u], p[v]
    return csr(u, v, V)


def comb(n, teeth):
    """A spine 0..n-1 with a tooth of `teeth` vertices under every 97th."""
    spine = np.arange(n - 1)
    us, vs, at = [spine], [spine + 1], n
    for s in range(0, n, 97):
        t = np.concatenate([[s], at + np.arange(teeth)])
        us.append(t[:-1])
        vs.append(t[1:])
        at += teeth
    return csr(np.concatenate(us), np.concatenate(vs), at)


def path(n, step=1):
    i = np.arange(n) if step > 0 else np.arange(n)[::-1]
    return csr(i[:-1], i[1:], n)


CASES = {
    "rows": lambda: grid(701, 499), "columns": lambda: grid(13, 40_003), "wide": lambda: grid(350_000, 2),
    "permuted": lambda: grid(701, 499, 3), "path": lambda: path(600_003), "backwards": lambda: path(65_537, -1),
    "comb": lambda: comb(50_000, 300),
}


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("direct", [False, True])
def test_long_chains(name, direct):
    off, col = CASES[name]()
    g = og.Graph.from_arrays(off, col)
    g.set_symmetric(True)
    kw = {}
    if direct:
        p = g.plan(budget=1 << 40, flags=og.CFG_DIRECT)
        kw = dict(budget=p["vertex_bytes"] + p["fixed_bytes"] + g.E * p["edge_bits"] // 16, advisek=0.8, direct=True)
    e = og.Engine(g, **kw)
    want = np.empty(g.V, np.uint32)
    oracle.cc_uf_mt_raw(g.V, off.ctypes.data, col.ctypes.data, 1, 4, want)
    for _ in range(2):
        np.testing.assert_array_equal(e.cc(), want)
    e.close()
