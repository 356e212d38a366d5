"""GPU: traversals on graphs around the sizes where the persistent kernels'
grids change, with and without hubs and in-edges.  Equal to the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(n, m, hub, symmetric, seed):
    rng = np.random.default_rng(seed)
    src, dst = rng.integers(0, n, m), rng.integers(0, n, m)
    if hub:
        src, dst = np.r_[src, np.zeros(hub, np.int64)], np.r_[dst, rng.integers(0, n, hub)]
    if symmetric:
        src, dst = np.r_[src, dst], np.r_[dst, src]
    key = np.unique(src * n + dst)
    src, dst = key // n, key % n
    offs = np.zeros(n + 1, np.uint32)
    offs[1:] = np.cumsum(np.bincount(src, minlength=n))
    wts = (np.minimum(src, dst) * 7919 + np.maximum(src, dst) * 104729) % 255 + 1
    return offs, dst.astype(np.uint32), wts.astype(np.uint32)


@pytest.mark.parametrize("hub", [0, 3000])
@pytest.mark.parametrize("n", [1 << 15, (1 << 15) + 1, 1 << 17, (1 << 17) + 1, 1 << 18, (1 << 18) + 1,
                               (1 << 20) + 1])
def test_symmetric(grus, oracle_mod, n, hub):
    offs, cols, wts = _csr(n, 2 * n, hub, True, n)
    g = grus.Graph.from_csr(offs, cols, wts, symmetric=True)
    csr = oracle_mod.CSR(offs, cols, wts)
    srcs = np.array([0, n // 2, n - 1], np.uint32)
    ref = oracle_mod.bfs_multi(csr, srcs)
    assert np.array_equal(grus.bfs(g, 0), ref[0])
    assert np.array_equal(grus.bfs_multi(g, srcs), ref)
    assert np.array_equal(grus.sssp(g, n // 2), oracle_mod.sssp(csr, n // 2))
    g.free()


@pytest.mark.parametrize("csc", [False, True])
@pytest.mark.parametrize("n", [1 << 17, (1 << 18) + 1])
def test_directed(grus, oracle_mod, n, csc):
    offs, cols, wts = _csr(n, 4 * n, 2000, False, n)
    g = grus.Graph.from_csr(offs, cols, wts)
    if csc:
        g.build_csc()
    csr = oracle_mod.CSR(offs, cols, wts)
    srcs = np.array([0, 5], np.uint32)
    ref = oracle_mod.bfs_multi(csr, srcs)
    assert np.array_equal(grus.bfs(g, 0), ref[0])
    assert np.array_equal(grus.bfs_multi(g, srcs), ref)
    g.free()
