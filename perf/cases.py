"""Performance cases: the traversals that a program runs through this package.

Each case is one call (or one batch) of a public entry point on a resident
graph.  Graphs come from the package's generators (RMAT, 2D grid) or, for a
vertex count that is no power of two, from CSR arrays of a random graph that
are uploaded as a program with its own data would upload them.  Weights are
uint32 in [1, 255], as in the package's benchmark.
"""
import math
import random

import numpy as np
import torch

import grus_framework_gb300 as grus

ITERS = 20       # PageRank iterations, the benchmark's count
DAMPING = 0.85


def listed():
    return [
        # the smallest call: one BFS on a graph of a few thousand vertices,
        # where launches and level barriers are all there is
        dict(name="bfs_rmat12", op="bfs", graph="rmat", scale=12, ef=16, source="hub", host=False),
        # an ordinary BFS with the default output (a new numpy array), on an
        # uploaded graph of odd size without hubs
        dict(name="bfs_uniform_host", op="bfs", graph="uniform", n=1000003, ef=8, source="edge", host=True),
        # the headline traversal: scale-free, 16.8 M vertices, 0.5 G edges
        dict(name="bfs_rmat24", op="bfs", graph="rmat", scale=24, ef=16, source="hub", host=False),
        # the high-diameter traversal (road-like): thousands of small levels
        dict(name="bfs_grid", op="bfs", graph="grid", rows=4096, cols=4096, source="corner", host=False),
        # shortest paths on a scale-free graph
        dict(name="sssp_rmat22", op="sssp", graph="rmat", scale=22, ef=16, source="hub", host=False),
        # shortest paths on a road-like graph of odd sides
        dict(name="sssp_grid", op="sssp", graph="grid", rows=1021, cols=1531, source="corner", host=False),
        # component labels of a scale-free graph
        dict(name="cc_rmat22", op="cc", graph="rmat", scale=22, ef=16, host=False),
        # ranks of a small directed graph of odd size (the default numpy output)
        dict(name="pagerank_small", op="pagerank", graph="uniform", n=50021, ef=12, host=True),
        # ranks of a large directed scale-free graph
        dict(name="pagerank_rmat24", op="pagerank", graph="rmat", scale=24, ef=16, host=False),
        # 64 traversals of one graph at once
        dict(name="bfs64_rmat23", op="bfs_multi", graph="rmat", scale=23, ef=16, sources=64),
        # 32 shortest-path searches of one graph at once
        dict(name="sssp32_rmat20", op="sssp_multi", graph="rmat", scale=20, ef=16, sources=32),
        # a batch of mixed queries over graphs of mixed sizes
        dict(name="batch_mixed", op="batch", lo=14, hi=19, graphs=12, sssp=6, bfs=2, replay=True),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def graph(scale_hi, n_hi, side_hi, kinds=("rmat", "uniform", "grid")):
        kind = rng.choice(kinds)
        if kind == "rmat":
            return dict(graph="rmat", scale=rng.randint(10, scale_hi), ef=rng.randint(8, 24))
        if kind == "uniform":
            return dict(graph="uniform", n=log(1000, n_hi), ef=rng.randint(4, 24))
        return dict(graph="grid", rows=log(40, side_hi), cols=log(40, side_hi))

    op = rng.choice(["bfs", "bfs", "sssp", "sssp", "cc", "pagerank", "bfs_multi", "sssp_multi", "batch"])
    if op == "bfs":
        return dict(op=op, **graph(23, 3000000, 2500), source=rng.choice(["hub", "edge"]), host=rng.random() < 0.25)
    if op == "sssp":
        return dict(op=op, **graph(21, 2000000, 1000), source=rng.choice(["hub", "edge"]), host=rng.random() < 0.25)
    if op == "cc":
        # graphs with more than one component: sparse where uniform
        c = graph(22, 3000000, 0, ("rmat", "uniform"))
        return dict(c, op=op, ef=c["ef"] if c["graph"] == "rmat" else rng.randint(1, 4), host=rng.random() < 0.25)
    if op == "pagerank":
        return dict(op=op, **graph(23, 3000000, 0, ("rmat", "uniform")), host=rng.random() < 0.25)
    if op == "bfs_multi":
        return dict(op=op, **graph(22, 2000000, 0, ("rmat", "uniform")), sources=rng.randint(2, 64))
    if op == "sssp_multi":
        return dict(op=op, **graph(19, 500000, 0, ("rmat", "uniform")), sources=rng.randint(2, 32))
    lo = rng.randint(10, 15)
    return dict(op=op, lo=lo, hi=lo + rng.randint(1, 4), graphs=rng.randint(2, 10), sssp=rng.randint(1, 8),
                bfs=rng.randint(0, 4), replay=rng.random() < 0.5)


def _uniform_csr(n, degree, seed, directed):
    """Random graph without self loops or duplicates, about `degree` out-edges
    a vertex; weights (symmetric ones when undirected) by a hash of the ends."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    m = n * degree if directed else n * degree // 2
    a = torch.randint(n, (m,), generator=gen, device="cuda")
    b = torch.randint(n, (m,), generator=gen, device="cuda")
    a, b = a[a != b], b[a != b]
    if not directed:
        a, b = torch.cat((a, b)), torch.cat((b, a))
    key = torch.unique(a * n + b)
    src, dst = key // n, key % n
    offs = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    offs[1:] = torch.cumsum(torch.bincount(src, minlength=n), 0)
    w = (torch.minimum(src, dst) * 2654435761 + torch.maximum(src, dst) * 40503 + seed) // 64 % 255 + 1
    return [x.to(torch.int32).cpu().numpy().view(np.uint32) for x in (offs, dst, w)]


def _graph(case, seed, weighted=False, directed=False):
    kind = case["graph"]
    if kind == "rmat":
        return grus.Graph.rmat(case["scale"], case["ef"], seed + 1, symmetric=not directed, weighted=weighted)
    if kind == "grid":
        return grus.Graph.grid2d(case["rows"], case["cols"], seed + 1, weighted=weighted)
    offs, cols, w = _uniform_csr(case["n"], case["ef"], seed + 1, directed)
    return grus.Graph.from_csr(offs, cols, w if weighted else None, symmetric=not directed)


def _tails(g, k, seed):
    """k vertices with out-edges: the tails of random edges."""
    offs = g.copy_offsets()
    edges = np.random.RandomState(seed % (1 << 32)).randint(0, max(int(g.m), 1), k)
    return (np.searchsorted(offs, edges, side="right") - 1).astype(np.uint32)


def _source(case, g, seed):
    if case["source"] == "hub":
        return int(g.max_degree_vertex)
    if case["source"] == "corner":
        r = random.Random(seed)
        return r.randrange(min(64, case["rows"])) * case["cols"] + r.randrange(min(64, case["cols"]))
    return int(_tails(g, 1, seed)[0])


def prepare(case, seed):
    op = case["op"]
    st = dict(op=op, host=case.get("host", False))
    if op == "batch":
        rng = random.Random(seed)
        graphs = []
        for i in range(case["graphs"]):
            scale = case["lo"] + i % (case["hi"] - case["lo"] + 1)
            graphs.append(grus.Graph.rmat(scale, rng.randint(8, 32), seed * 64 + i + 1, weighted=True))
        queries = []
        for i, g in enumerate(graphs):
            srcs = _tails(g, case["sssp"] + case["bfs"], seed + i)
            queries += [(i, grus.ALGO_SSSP if j < case["sssp"] else grus.ALGO_BFS, int(s)) for j, s in enumerate(srcs)]
        for g in graphs:
            g.build_index()
        st["batch"] = grus.Batch(graphs)
        st["queries"], st["replay"] = queries, case["replay"]
        st["offsets"], total = st["batch"].layout(queries)
        st["out"] = torch.empty(total, dtype=torch.int32, device="cuda")
        return st
    directed = op == "pagerank"
    g = st["g"] = _graph(case, seed, weighted=op in ("sssp", "sssp_multi"), directed=directed)
    n = int(g.n)
    if op == "pagerank":
        g.build_csc()
    if op == "bfs":
        g.build_index()
    if op in ("bfs", "sssp"):
        st["src"] = _source(case, g, seed)
    if op in ("bfs_multi", "sssp_multi"):
        st["srcs"] = _tails(g, case["sources"], seed)
        st["out"] = torch.empty((case["sources"], n), dtype=torch.int32, device="cuda")
    elif not st["host"]:
        st["out"] = torch.empty(n, dtype=torch.float32 if op == "pagerank" else torch.int32, device="cuda")
    return st


def run(st):
    op, out = st["op"], st.get("out")
    if op == "bfs":
        r = grus.bfs(st["g"], st["src"], out=out)
    elif op == "sssp":
        r = grus.sssp(st["g"], st["src"], out=out)
    elif op == "cc":
        r = grus.cc(st["g"], out=out)
    elif op == "pagerank":
        r = grus.pagerank(st["g"], DAMPING, ITERS, out=out)
    elif op == "bfs_multi":
        r = grus.bfs_multi(st["g"], st["srcs"], out=out)
    elif op == "sssp_multi":
        r = grus.sssp_multi(st["g"], st["srcs"], out=out)
    else:
        st["batch"].run(st["queries"], out, st["offsets"], use_graph=st["replay"])
        r = out
    return r


def _size(case):
    """Vertices and stored edges; the generators' own counts up to the
    duplicates that they drop."""
    both = 1 if case["op"] == "pagerank" else 2
    if case["graph"] == "rmat":
        n = 1 << case["scale"]
        return n, both * n * case["ef"]
    if case["graph"] == "grid":
        r, c = case["rows"], case["cols"]
        return r * c, 2 * (2 * r * c - r - c)
    return case["n"], case["n"] * case["ef"]


def work(case):
    """The graph read once and the outputs written once; PageRank reads its
    edges in every iteration."""
    op = case["op"]
    if op == "batch":
        total = 0
        for i in range(case["graphs"]):
            n = 1 << (case["lo"] + i % (case["hi"] - case["lo"] + 1))
            total += 4 * n + 8 * 2 * 20 * n + 4 * n * (case["sssp"] + case["bfs"])
        return {"bytes": total, "flops": 0}
    n, m = _size(case)
    if op == "pagerank":
        return {"bytes": ITERS * (4 * m + 8 * n) + 4 * n, "flops": 2 * ITERS * m}
    per_edge = 8 if op in ("sssp", "sssp_multi") else 4
    return {"bytes": 4 * (n + 1) + per_edge * m + 4 * n * case.get("sources", 1), "flops": 0}


def exact(case, seed):
    """PageRank in 64 bits; the other outputs are whole numbers."""
    if case["op"] != "pagerank":
        return None
    offs, cols, _ = prepare(case, seed)["g"].copy_csr()
    offs = torch.from_numpy(offs.astype(np.int64)).cuda()
    cols = torch.from_numpy(cols.view(np.int32)).cuda()
    n, m = offs.numel() - 1, cols.numel()
    deg = (offs[1:] - offs[:-1]).double()
    inv = torch.where(deg > 0, 1.0 / deg.clamp(min=1.0), torch.zeros_like(deg))
    rank = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    step = 1 << 26
    for _ in range(ITERS):
        c, acc = rank * inv, torch.zeros(n, dtype=torch.float64, device="cuda")
        for e in range(0, m, step):
            hi = min(m, e + step)
            src = torch.searchsorted(offs, torch.arange(e, hi, device="cuda"), right=True) - 1
            acc.index_add_(0, cols[e:hi].long(), c[src])
        rank = (1.0 - DAMPING) / n + DAMPING * acc
    return rank.cpu().numpy() if case.get("host") else rank
