"""GPU: traversals that the one-cluster kernel runs or finishes, bit-exact
against the oracle and against the persistent kernel alone (tail_cluster=2).

The graphs sit where its lists can go wrong: sizes around the cluster's 16
home ranges, entries at and past one 64-edge piece, more near vertices than
the lists hold, more far vertices than the far lists hold, weights far above
and far below Delta, chains whose ids jump between homes at every step.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(n, pairs, weights):
    """Symmetric CSR of undirected (u, v) pairs with one weight each."""
    u, v = np.array(pairs, np.int64).reshape(-1, 2).T
    w = np.asarray(weights, np.int64)
    src, dst, wt = np.r_[u, v], np.r_[v, u], np.r_[w, w]
    order = np.lexsort((dst, src))
    offs = np.zeros(n + 1, np.uint32)
    offs[1:] = np.cumsum(np.bincount(src, minlength=n))
    return offs, dst[order].astype(np.uint32), wt[order].astype(np.uint32)


def _path(n, perm=None):
    ids = np.arange(n) if perm is None else perm
    return np.stack([ids[:-1], ids[1:]], 1)


def _cases():
    rng = np.random.default_rng(11)
    for n in (2, 15, 16, 17, 33, 1000):
        p = _path(n)
        yield f"path{n}", n, p, rng.integers(1, 256, len(p)), 0
    n = 3001
    p = _path(n, rng.permutation(n))
    yield "jumping_path", n, p, rng.integers(1, 256, len(p)), int(p[0, 0])
    yield "heavy_weights", n, p, rng.integers(1 << 16, 1 << 19, len(p)), int(p[0, 0])
    yield "unit_weights", n, p, np.ones(len(p), np.int64), int(p[1500, 0])
    for leaves in (63, 64, 65, 129, 2500):
        p = np.r_[_path(20), np.stack([np.full(leaves, 19), 20 + np.arange(leaves)], 1)]
        yield f"broom{leaves}", 20 + leaves, p, rng.integers(1, 256, len(p)), 0
    # every leaf has a second edge, so all of them are pushed: near lists of
    # 16 x 2,048 entries overflow at once
    k = 60000
    fan = np.stack([np.full(k, 199), 200 + np.arange(k)], 1)
    rim = np.stack([200 + np.arange(0, k, 2), 200 + np.arange(1, k, 2)], 1)
    p = np.r_[_path(200), fan, rim]
    yield "near_overflow", 200 + k, p, rng.integers(1, 20, len(p)), 0
    # ... and, beyond Delta, far lists of 16 x 8,192
    k = 180000
    fan = np.stack([np.full(k, 199), 200 + np.arange(k)], 1)
    rim = np.stack([200 + np.arange(0, k, 2), 200 + np.arange(1, k, 2)], 1)
    p = np.r_[_path(200), fan, rim]
    w = np.r_[np.full(199, 3), rng.integers(3000, 30000, k), np.full(k // 2, 7)]
    yield "far_overflow", 200 + k, p, w, 0


@pytest.mark.parametrize("name,n,pairs,weights,src", list(_cases()),
                         ids=[c[0] for c in _cases()])
def test_sssp_narrow_shapes(grus, oracle_mod, name, n, pairs, weights, src):
    offs, cols, wts = _csr(n, pairs, weights)
    ref = oracle_mod.sssp(oracle_mod.CSR(offs, cols, wts), src)
    g = grus.Graph.from_csr(offs, cols, wts, symmetric=True)
    for delta in (0, 1, 50):
        if delta == 1 and n > 4000:
            continue  # as many threshold steps as distances
        g.set_tuning(sssp_delta=delta)
        got, st = grus.sssp(g, src, stats=True)
        assert np.array_equal(got, ref), (name, delta)
        reached = ref != grus.INFINIT
        assert st["vertices_reached"] == int(reached.sum())
        assert st["edges_reached"] == int(np.diff(offs)[reached].sum())
    g.free()


@pytest.mark.parametrize("name,n,pairs,weights,src", list(_cases()),
                         ids=[c[0] for c in _cases()])
def test_bfs_narrow_shapes(grus, oracle_mod, name, n, pairs, weights, src):
    """The same shapes without weights: depths, reach counts and the level
    count (one more than the largest depth), and the trace's vertices."""
    offs, cols, _ = _csr(n, pairs, weights)
    ref = oracle_mod.bfs(oracle_mod.CSR(offs, cols), src)
    g = grus.Graph.from_csr(offs, cols, symmetric=True)
    reached = ref != grus.INFINIT
    for tail in (0, 2):
        g.set_tuning(tail_cluster=tail)
        got, st = grus.bfs(g, src, stats=True)
        assert np.array_equal(got, ref), (name, tail)
        assert st["levels"] == int(ref[reached].max()) + 1
        assert st["vertices_reached"] == int(reached.sum())
        assert st["edges_reached"] == int(np.diff(offs)[reached].sum())
        for i, t in enumerate(grus.bfs_trace(g, 100)):
            assert t["vertices"] == int((ref == i + 1).sum()), (name, tail, i)
    g.free()


@pytest.mark.parametrize("make", [
    lambda g: g.Graph.grid2d(400, 500, 5, weighted=True),    # handed over, 2^19 edges and more
    lambda g: g.Graph.grid2d(700, 31, 6, weighted=True),     # whole
    lambda g: g.Graph.rmat(12, 16, 3, weighted=True),        # whole, hubs of many pieces
    lambda g: g.Graph.rmat(15, 8, 4, weighted=True),         # hubs, handed over near the end
    lambda g: g.Graph.rmat(13, 4, 4, weighted=True, symmetric=False),
])
def test_narrow_matches_persistent(grus, make):
    """The same distances with and without the cluster kernel, from several
    sources, synchronous and queued back to back on a stream."""
    torch = pytest.importorskip("torch")
    g = make(grus)
    deg = np.diff(g.copy_offsets())
    srcs = [int(g.max_degree_vertex)] + [int(v) for v in np.flatnonzero(deg > 0)[[0, 7, -1]]]
    g.set_tuning(tail_cluster=2)
    refs = [grus.sssp(g, s, stats=True) for s in srcs]
    g.set_tuning(tail_cluster=0)
    outs = [torch.full((int(g.n),), -7, dtype=torch.int32, device="cuda") for _ in srcs]
    stream = torch.cuda.Stream()
    for s, o in zip(srcs, outs):
        grus.sssp(g, s, out=o, stream=stream)
    stream.synchronize()
    for s, o, (ref, rst) in zip(srcs, outs, refs):
        assert np.array_equal(o.cpu().numpy().view(np.uint32), ref)
        got, st = grus.sssp(g, s, stats=True)
        assert np.array_equal(got, ref)
        assert st["vertices_reached"] == rst["vertices_reached"]
        assert st["edges_reached"] == rst["edges_reached"]
        b0, s0 = grus.bfs(g, s, stats=True)
        g.set_tuning(tail_cluster=2)
        b2, s2 = grus.bfs(g, s, stats=True)
        g.set_tuning(tail_cluster=0)
        assert np.array_equal(b0, b2)
        for k in ("levels", "vertices_reached", "edges_reached"):
            assert s0[k] == s2[k], k
    g.free()
