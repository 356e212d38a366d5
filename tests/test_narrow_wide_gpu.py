"""GPU: vertices whose out-edges do not fit the one-cluster kernel's lists
(16 x 2,048 entries of 64 edges): one of more than 2,097,152 out-edges, and
several smaller ones that fill the lists together, reached after the hand-over.
Expected values follow from the construction."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PATH = 20


def _hubs(count, leaves):
    """A path whose last vertex is joined to `count` hubs of `leaves` leaves."""
    n = PATH + count + count * leaves
    deg = np.ones(n, np.int64)
    deg[1:PATH - 1] = 2
    deg[PATH - 1] = 1 + count
    deg[PATH:PATH + count] = 1 + leaves
    offs = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint32)
    leaf = np.arange(PATH + count, n, dtype=np.uint32).reshape(count, leaves)
    path = [1] + [x for i in range(1, PATH - 1) for x in (i - 1, i + 1)] + [PATH - 2]
    hub_ids = np.arange(PATH, PATH + count, dtype=np.uint32)
    hub_adj = np.concatenate([np.full((count, 1), PATH - 1, np.uint32), leaf], 1)
    cols = np.concatenate([np.array(path, np.uint32), hub_ids, hub_adj.ravel(),
                           np.repeat(hub_ids, leaves)])
    depth = np.concatenate([np.arange(PATH), np.full(count, PATH),
                            np.full(count * leaves, PATH + 1)]).astype(np.uint32)
    assert len(cols) == offs[-1]
    return offs, cols, depth


# pieces: 46,876; 40 x 1,876 = 75,040; 200 x 313 = 62,600 (more hubs spill than
# one step takes)
@pytest.mark.parametrize("count,leaves", [(1, 3000000), (40, 120000), (200, 20000)])
def test_bfs_hubs_past_the_lists(grus, count, leaves):
    offs, cols, depth = _hubs(count, leaves)
    g = grus.Graph.from_csr(offs, cols, symmetric=True)
    got, st = grus.bfs(g, 0, stats=True)
    assert np.array_equal(got, depth)
    assert st["levels"] == PATH + 2
    assert st["vertices_reached"] == len(depth) and st["edges_reached"] == len(cols)
    g.free()


@pytest.mark.parametrize("count,leaves", [(1, 2300000), (40, 70000)])
def test_sssp_settled_hubs_improved_in_the_cluster(grus, count, leaves):
    """A heavy edge reaches the hubs first, so they are settled when the cluster
    takes over; the path then lowers them.  Leaves have no out-edges."""
    path = 60
    n = path + count + count * leaves
    deg = np.zeros(n, np.int64)
    deg[:path - 1] = 1
    deg[0] += count
    deg[path - 1] = count
    deg[path:path + count] = leaves
    offs = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint32)
    hub_ids = np.arange(path, path + count, dtype=np.uint32)
    cols = np.concatenate([[1], hub_ids, np.arange(2, path), hub_ids,
                           np.arange(path + count, n)]).astype(np.uint32)
    lw = np.random.default_rng(3).integers(1, 200, count * leaves).astype(np.uint32)
    wts = np.concatenate([[1], np.full(count, 600), np.ones(path - 2), np.ones(count),
                          lw]).astype(np.uint32)
    assert len(cols) == len(wts) == offs[-1]
    ref = np.concatenate([np.arange(path), np.full(count, path), path + lw]).astype(np.uint32)
    g = grus.Graph.from_csr(offs, cols, wts, symmetric=False)
    g.set_tuning(tail_cluster=2)
    got, st2 = grus.sssp(g, 0, stats=True)
    assert np.array_equal(got, ref)
    g.set_tuning(tail_cluster=0)
    got, st = grus.sssp(g, 0, stats=True)
    assert np.array_equal(got, ref)
    assert st["vertices_reached"] == n and st["edges_reached"] == len(cols)
    assert st["levels"] < st2["levels"]  # the cluster's steps are several levels each
    g.free()


def _tree(path, depth):
    """A path into the root of a binary tree numbered in preorder: few
    neighbours, near by id, and a frontier that doubles."""
    size = (1 << depth) - 1
    left, right, stack = [], [], [(0, depth)]
    while stack:
        v, d = stack.pop()
        if d == 1:
            continue
        half = (1 << (d - 1)) - 1
        left += [v, v]
        right += [v + 1, v + 1 + half]
        stack += [(v + 1, d - 1), (v + 1 + half, d - 1)]
    u = np.concatenate([np.arange(path), np.array(left) + path])
    v = np.concatenate([np.arange(1, path + 1), np.array(right) + path])
    n = path + size
    src, dst = np.concatenate([u, v]), np.concatenate([v, u])
    order = np.lexsort((dst, src))
    w = (np.minimum(u, v) * 40503 + np.maximum(u, v) * 9973) % 255 + 1
    offs = np.zeros(n + 1, np.uint32)
    offs[1:] = np.cumsum(np.bincount(src, minlength=n))
    return offs, dst[order].astype(np.uint32), np.concatenate([w, w])[order].astype(np.uint32)


@pytest.mark.parametrize("path,depth", [(40, 18), (100, 19)])
def test_frontier_wider_than_the_lists(grus, oracle_mod, path, depth):
    offs, cols, wts = _tree(path, depth)
    csr = oracle_mod.CSR(offs, cols, wts)
    g = grus.Graph.from_csr(offs, cols, wts, symmetric=True)
    for call, ref in ((grus.bfs, oracle_mod.bfs(csr, 0)), (grus.sssp, oracle_mod.sssp(csr, 0))):
        for tail in (0, 2):
            g.set_tuning(tail_cluster=tail)
            got, st = call(g, 0, stats=True)
            assert np.array_equal(got, ref), (call.__name__, tail)
            assert st["vertices_reached"] == int(g.n) and st["edges_reached"] == int(g.m)
            if call is grus.bfs:
                assert st["levels"] == path + depth
                for i, t in enumerate(grus.bfs_trace(g, 200)):
                    assert t["vertices"] == int((ref == i + 1).sum()), (tail, i)
    g.free()
