"""What a user of this framework has it do, as cases that can be timed.

A case is one call (or one burst of requests) through the Python entry points
on a graph that the program has loaded and planned: the engine, the server and
the page-locked result buffers are made by prepare() and kept, the sources are
new inputs of the call.  Graphs are drawn with torch from the seed: R-MAT with
the benchmark's quadrants over any number of vertices, and road-like grids.
"""
import numpy as np
import torch

import onegraph_gb300 as og

ABC = og.RMAT_ABC  # quadrant probabilities of the benchmark graphs
TOL = 1e-6         # L1 stop of the precision PageRank (the entry point's default)
THRESHOLD = 1e-3   # per-vertex stop of the reference's PageRank
DAMPING = 0.85


def listed():
    return [
        # The smallest call: one BFS of a graph of a thousand vertices, result
        # in a new array.  Launches and waits are all there is.
        {"name": "bfs small", "op": "bfs", "graph": "rmat", "V": 1003, "ef": 16, "mode": "resident"},
        # The benchmark's resident BFS (scale 20, direction-optimizing).
        {"name": "bfs resident", "op": "bfs", "graph": "rmat", "V": 1 << 20, "ef": 16, "mode": "resident"},
        # A road-like graph: about a thousand levels with small frontiers.
        {"name": "bfs road", "op": "bfs", "graph": "grid", "V": 701 * 499, "ef": 2, "mode": "resident"},
        # An ordinary resident SSSP query of a served graph, odd size.
        {"name": "sssp resident", "op": "sssp", "graph": "rmat", "V": 300007, "ef": 16, "mode": "resident"},
        # The path the framework exists for: SSSP with most edges in host
        # memory, a quarter of them resident as in the benchmark.
        {"name": "sssp oom", "op": "sssp", "graph": "rmat", "V": 1 << 24, "ef": 16, "mode": "direct", "part": 0.25},
        # Several SSSP sources sharing one pass, as the server runs them.
        {"name": "sssp batch", "op": "sssp_batch", "graph": "rmat", "V": 1 << 20, "ef": 16, "mode": "direct",
         "part": 0.5, "n": 8},
        # 64 BFS sources in one pass over an out-of-memory graph, byte depths
        # fetched.
        {"name": "bfs batch", "op": "bfs_batch", "graph": "rmat", "V": 1 << 23, "ef": 16, "mode": "direct",
         "part": 0.4, "n": 64},
        # Components of a symmetric out-of-memory graph.
        {"name": "cc oom", "op": "cc", "graph": "rmat", "V": 1 << 23, "ef": 16, "mode": "direct", "part": 0.4},
        # Label propagation, what a graph that is not symmetric gets; odd size.
        {"name": "cc directed", "op": "cc_directed", "graph": "rmat", "V": 2000003, "ef": 12, "mode": "resident"},
        # The precision study's PageRank, run to its default tolerance, most
        # edges resident as in the benchmark.
        {"name": "pr l1", "op": "pr_l1", "graph": "rmat", "V": 1 << 23, "ef": 16, "mode": "direct", "part": 1.2},
        # The reference's PageRank in its default mode: staged chunks of the
        # edges that do not fit.
        {"name": "pr delta staged", "op": "pr", "graph": "rmat", "V": 777777, "ef": 14, "mode": "staged", "part": 0.5},
        # The served mix (60 % BFS, 30 % SSSP, 10 % PageRank) over two resident
        # graphs, every result fetched.
        {"name": "serve", "op": "serve", "graph": "rmat", "V": 1 << 19, "ef": 16, "mode": "resident", "n": 48},
    ]


# vertices each kind of call is drawn over: from a handful of launches to the
# listed largest
RANGE = {
    "bfs": (1000, 1 << 23), "sssp": (1000, 1 << 24), "sssp_batch": (4000, 1 << 20),
    "bfs_batch": (4000, 1 << 23), "cc": (1000, 1 << 23), "cc_directed": (1000, 2000003),
    "pr_l1": (4000, 1 << 23), "pr": (4000, 777777), "serve": (4000, 1 << 19),
}


def draw(rng):
    op = rng.choice(list(RANGE))
    lo, hi = RANGE[op]
    V = int(round(lo * (hi / lo) ** rng.random()))
    c = {"op": op, "graph": "rmat", "V": V, "ef": rng.randint(8, 16 if op not in ("cc_directed", "pr") else 12),
         "mode": rng.choice(["resident", "direct", "staged"])}
    if op == "bfs" and rng.random() < 0.3:
        c.update(graph="grid", V=min(V, 350000), ef=2, mode="resident")
    if op in ("bfs_batch", "sssp_batch") and c["mode"] == "staged":
        c["mode"] = "direct"
    if op == "serve":
        c["mode"] = "resident"
    if c["mode"] != "resident":
        c["part"] = round(rng.uniform(0.25, 1.2 if op == "pr_l1" else 0.8), 2)
    if op == "bfs_batch":
        c["n"] = rng.randint(1, 64)
    if op == "sssp_batch":
        c["n"] = rng.randint(2, 8)
    if op == "serve":
        c["n"] = rng.randint(8, 48)
    return c


# ------------------------------------------------------------------- graphs

def device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def rmat_tuples(V, count, gen):
    """Endpoints of R-MAT tuples over V vertices (ids permuted, the part of the
    square beyond V folded back)."""
    dev = device()
    a, b, c = ABC
    u = torch.zeros(count, dtype=torch.int64, device=dev)
    v = torch.zeros(count, dtype=torch.int64, device=dev)
    for _ in range(max(1, (V - 1).bit_length())):
        r = torch.rand(count, generator=gen, device=dev)
        u = (u << 1) | (r >= a + b)
        v = (v << 1) | (((r >= a) & (r < a + b)) | (r >= a + b + c))
    perm = torch.randperm(V, generator=gen, device=dev)
    return perm[u % V], perm[v % V]


def grid_edges(V, gen):
    """Right and down neighbours of a grid about 7:5, a tenth of them dropped."""
    dev = device()
    w = max(2, int(round((V * 7 / 5) ** 0.5)))
    i = torch.arange(V, device=dev)
    right = i[(i % w != w - 1) & (i + 1 < V)]
    down = i[i + w < V]
    u, v = torch.cat([right, down]), torch.cat([right + 1, down + w])
    keep = torch.rand(u.numel(), generator=gen, device=dev) >= 0.1
    return u[keep], v[keep]


def csr(case, seed, symmetric):
    """(offsets, columns) as int64 tensors: sorted lists, no loops, no repeats."""
    V = case["V"]
    gen = torch.Generator(device=device())
    gen.manual_seed(seed)
    if case["graph"] == "grid":
        u, v = grid_edges(V, gen)
    else:
        u, v = rmat_tuples(V, V * case["ef"], gen)
    keep = u != v
    u, v = u[keep], v[keep]
    key = torch.cat([u * V + v, v * V + u]) if symmetric else u * V + v
    key = torch.unique(key)
    off = torch.zeros(V + 1, dtype=torch.int64, device=key.device)
    off[1:] = torch.cumsum(torch.bincount(key // V, minlength=V), 0)
    return off, key % V, gen


def u32(t):
    return t.to(torch.int32).cpu().numpy().view(np.uint32)


def make_graph(case, seed, kind, symmetric=True):
    off, col, gen = csr(case, seed, symmetric)
    offsets = off.cpu().numpy().view(np.uint64)
    if kind == og.WEIGHTED:
        w = torch.randint(1, 65, (col.numel(),), generator=gen, device=col.device)
        g = og.Graph.from_arrays(offsets, u32(torch.stack([col, w], 1)), kind=kind)
    elif kind == og.PR:  # lists are in-neighbours
        outdeg = torch.bincount(col, minlength=case["V"])
        g = og.Graph.from_arrays(offsets, u32(col), u32(outdeg), kind=kind)
    else:
        g = og.Graph.from_arrays(offsets, u32(col), kind=kind)
    if symmetric:
        g.set_symmetric(True)
    deg = off[1:] - off[:-1]
    return g, torch.nonzero(deg)[:, 0].cpu().numpy()


def make_engine(case, g, **kw):
    """The engine of the case's mode: everything resident (the default budget),
    or a budget that holds the vertex state and `part` of the edges."""
    if case["mode"] == "resident":
        return og.Engine(g, **kw)
    direct = case["mode"] == "direct"
    flags = ((og.CFG_DIRECT if direct else 0) | (og.CFG_PR if kw.get("pagerank") else 0) |
             (og.CFG_BATCH if kw.get("batch") else 0) | og.CFG_SSSP_BATCH(kw.get("sssp_batch", 0)))
    p = g.plan(budget=1 << 40, flags=flags)
    share = int(case["part"] * g.E * p["edge_bits"] / 8) + 4096
    # the advised share of what the budget leaves for edges is resident, the
    # rest is staging
    return og.Engine(g, budget=p["vertex_bytes"] + p["fixed_bytes"] + share, advisek=0.8, direct=direct, **kw)


# -------------------------------------------------------------------- cases

KIND = {"bfs": og.PLAIN, "sssp": og.WEIGHTED, "sssp_batch": og.WEIGHTED, "bfs_batch": og.PLAIN, "cc": og.PLAIN,
        "cc_directed": og.PLAIN, "pr_l1": og.PR, "pr": og.PR}


class State:
    pass


def prepare(case, seed):
    s = State()
    s.case, op, V = case, case["op"], case["V"]
    rng = np.random.default_rng(seed)
    if op == "serve":
        return prepare_serve(s, case, seed, rng)
    s.g, s.live = make_graph(case, seed, KIND[op], op not in ("cc_directed", "pr_l1", "pr"))
    s.e = make_engine(case, s.g, batch=op == "bfs_batch", sssp_batch=case["n"] if op == "sssp_batch" else 0)
    s.srcs = rng.choice(s.live, case.get("n", 1), replace=s.live.size < case.get("n", 1)).astype(np.uint32)
    n = s.srcs.size
    if V < 4096:
        s.out = None  # a small result goes to a new array
    elif op == "bfs_batch":
        s.out = og.pinned_empty((n, V), np.uint8)
    elif op == "sssp_batch":
        s.out = og.pinned_empty((n, V), np.uint32)
    else:
        s.out = og.pinned_empty(V, np.float32 if op in ("pr", "pr_l1") else np.uint32)
    return s


def serve_cases(case):
    """The two served graphs: the case's own and one of a quarter of it."""
    return [dict(case, V=max(1000, case["V"] // 4)), case]


def serve_requests(case, live, rng):
    """(graph, algorithm, source) of the mix: the same kinds in every burst,
    other sources."""
    kinds = np.random.default_rng(4)
    algos = kinds.choice([og.ALGO_BFS, og.ALGO_SSSP, og.ALGO_PR], case["n"], p=[0.6, 0.3, 0.1])
    algos[:3] = [og.ALGO_PR, og.ALGO_SSSP, og.ALGO_BFS]
    graphs = kinds.choice(2, case["n"], p=[0.6, 0.4])
    return [(int(k), int(a), int(rng.choice(live[k]))) for k, a in zip(graphs, algos)]


def prepare_serve(s, case, seed, rng):
    s.srv = og.Server(workers=4)
    s.graphs, live = [], []
    for k, c in enumerate(serve_cases(case)):
        g, ids = make_graph(c, seed + k * 7919, og.WEIGHTED)
        s.srv.add_graph(g, budget=0, advisek=1.0, direct=True, pagerank=True, sssp_batch=16)
        s.graphs.append(g)
        live.append(ids)
    s.requests = serve_requests(case, live, rng)
    s.outs = [og.pinned_empty(s.graphs[k].V, np.float32 if a == og.ALGO_PR else np.uint32)
              for k, a, _ in s.requests]
    return s


def i32(a):
    """The same 32-bit words as int32 (torch indexes no uint32 arrays)."""
    return a.view(np.int32) if a.dtype == np.uint32 else a


def run(s):
    op = s.case["op"]
    if op == "bfs":
        return i32(s.e.bfs(int(s.srcs[0]), s.out))
    if op == "sssp":
        return i32(s.e.sssp(int(s.srcs[0]), s.out))
    if op in ("cc", "cc_directed"):
        return i32(s.e.cc(s.out))
    if op == "pr_l1":
        return s.e.pr_l1(damping=DAMPING, tol=TOL, out=s.out)
    if op == "pr":
        return s.e.pr(THRESHOLD, out=s.out)
    if op == "sssp_batch":
        dist, checks = s.e.sssp_batch(s.srcs, s.out)
        return [i32(dist), checks.view(np.int64)]
    if op == "bfs_batch":
        depths, clamped, checks = s.e.bfs_batch_u8(s.srcs, s.out)
        return [depths, checks.view(np.int64), int(clamped)]
    for (k, algo, src), out in zip(s.requests, s.outs):
        s.srv.submit(k, algo, source=src, iterations=5, out=out)
    left = len(s.requests)
    while left:
        left -= len(s.srv.poll())
    return [i32(o) for o in s.outs]


def work(case):
    """Every edge and offset read once, every result written once; additions
    for PageRank (per iteration, 48 to the tolerance) and one comparison per
    edge and source elsewhere."""
    op, V, n = case["op"], case["V"], case.get("n", 1)
    once = 1 if op in ("cc_directed", "pr_l1", "pr") else 2
    if op == "serve":
        total = {"bytes": 0, "flops": 0}
        for c, share in zip(serve_cases(case), (0.6, 0.4)):
            E = 2 * c["V"] * c["ef"]
            total["bytes"] += 8 * E + 8 * c["V"] + n * share * 4 * c["V"]
            total["flops"] += n * share * E
        return total
    E = V * (1.8 if case["graph"] == "grid" else case["ef"]) * once
    weighted = op in ("sssp", "sssp_batch")
    out = n * V * (1 if op == "bfs_batch" else 4)
    iters = {"pr_l1": 48, "pr": 20}.get(op, 1)
    return {"bytes": E * (8 if weighted else 4) + 8 * V + out, "flops": E * iters * n}


# ------------------------------------------------------------ 64-bit results

def pr_inputs(case, seed, symmetric):
    off, col, _ = csr(case, seed, symmetric)
    V = case["V"]
    row = torch.repeat_interleave(torch.arange(V, device=col.device), off[1:] - off[:-1])
    outdeg = (off[1:] - off[:-1]).double() if symmetric else torch.bincount(col, minlength=V).double()
    inv = torch.where(outdeg > 0, 1.0 / outdeg.clamp(min=1), torch.zeros_like(outdeg))
    return row, col, inv


def pull(rank, row, col, inv):
    return torch.zeros_like(rank).index_add_(0, row, (rank * inv)[col])


def exact_l1(case, seed, symmetric, tol, iters):
    row, col, inv = pr_inputs(case, seed, symmetric)
    V = case["V"]
    rank = torch.full((V,), 1.0 / V, dtype=torch.float64, device=col.device)
    for _ in range(iters):
        new = (1 - DAMPING) / V + DAMPING * pull(rank, row, col, inv)
        delta = float((new - rank).abs().sum())
        rank = new
        if delta < tol:
            break
    return rank.cpu().numpy()


def exact_delta(case, seed):
    row, col, inv = pr_inputs(case, seed, False)
    V = case["V"]
    rank = torch.ones(V, dtype=torch.float64, device=col.device)
    active = torch.ones(V, dtype=torch.bool, device=col.device)
    for _ in range(10000):
        new = 0.15 + 0.85 * pull(rank, row, col, inv)
        active = active & ((new - rank).abs() > THRESHOLD)
        rank = torch.where(active, new, rank)
        if not bool(active.any()):
            break
    return rank.cpu().numpy()


def exact(case, seed):
    op = case["op"]
    if op == "pr_l1":
        return exact_l1(case, seed, False, TOL, 200)
    if op == "pr":
        return exact_delta(case, seed)
    if op == "serve":
        rng = np.random.default_rng(seed)
        live, ranks = [], []
        for k, c in enumerate(serve_cases(case)):
            off, _, _ = csr(c, seed + k * 7919, True)
            live.append(torch.nonzero(off[1:] - off[:-1])[:, 0].cpu().numpy())
            ranks.append(exact_l1(c, seed + k * 7919, True, 0.0, 5))
        return [ranks[k] if a == og.ALGO_PR else None for k, a, _ in serve_requests(case, live, rng)]
    return None
