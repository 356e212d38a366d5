"""GPU: more far vertices than the one-cluster kernel's far lists hold (16 x 4,096,
BFS 16 x 1,024): what does not fit waits in the far bitmap until the split."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fan(path, leaves):
    """A path, a fan of `leaves` from its last vertex, and the leaves in pairs;
    the last leaf goes on into a second path and fan."""
    def one(first):
        hub = first + path - 1
        leaf = first + path + np.arange(leaves)
        return hub, leaf, np.concatenate([
            np.stack([np.arange(first, hub), np.arange(first + 1, hub + 1)], 1),
            np.stack([np.full(leaves, hub), leaf], 1),
            np.stack([leaf[0:-1:2], leaf[1::2]], 1)])
    _, leaf, a = one(0)
    _, _, b = one(path + leaves)
    return 2 * (path + leaves), np.concatenate([a, b, [[leaf[-1], path + leaves]]])


def _csr(n, pairs, w):
    u, v = pairs.T
    src, dst, wt = np.r_[u, v], np.r_[v, u], np.r_[w, w]
    order = np.lexsort((dst, src))
    offs = np.zeros(n + 1, np.uint32)
    offs[1:] = np.cumsum(np.bincount(src, minlength=n))
    return offs, dst[order].astype(np.uint32), wt[order].astype(np.uint32)


def test_bfs_far_lists_overflow(grus, oracle_mod):
    """The whole traversal in the cluster (at most 2^17 edges), thresholds at
    multiples of 32: the leaves of both fans lie on one."""
    n, pairs = _fan(32, 20800)
    offs, cols, _ = _csr(n, pairs, np.ones(len(pairs), np.int64))
    assert len(cols) <= 1 << 17
    ref = oracle_mod.bfs(oracle_mod.CSR(offs, cols), 0)
    assert (ref == 32).sum() == 20800 > 16 * 1024
    g = grus.Graph.from_csr(offs, cols, symmetric=True)
    got, st = grus.bfs(g, 0, stats=True)
    assert np.array_equal(got, ref)
    assert st["kernel_launches"] == 1  # the cluster's
    g.free()


def test_sssp_far_lists_overflow(grus, oracle_mod):
    """Handed over (at most 2^19 edges), the fans' leaves far beyond Delta."""
    n, pairs = _fan(40, 70000)
    w = np.full(len(pairs), 3)
    fan = pairs[:, 1] - pairs[:, 0] > 1
    w[fan] = np.random.default_rng(4).integers(3000, 30000, int(fan.sum()))
    n1 = n // 2  # the first half alone: 70,000 leaves > 16 x 4,096
    first = (pairs < n1).all(1)
    offs, cols, wts = _csr(n1, pairs[first], w[first])
    ref = oracle_mod.sssp(oracle_mod.CSR(offs, cols, wts), 0)
    g = grus.Graph.from_csr(offs, cols, wts, symmetric=True)
    g.set_tuning(tail_cluster=2)
    got, st2 = grus.sssp(g, 0, stats=True)
    assert np.array_equal(got, ref)
    g.set_tuning(tail_cluster=0)
    got, st = grus.sssp(g, 0, stats=True)
    assert np.array_equal(got, ref)
    assert st["levels"] < st2["levels"]  # the cluster took over
    g.free()
