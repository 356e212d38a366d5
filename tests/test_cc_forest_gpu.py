"""GPU: connected components where the first forest can go wrong: sizes around
a block and around the size from which roots are hooked twice, paths in and
out of order (long chains of parents), ties in degree, stars, cliques joined by
one edge, and one-way edges.  Equal to the oracle's labels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(grus, oracle_mod, n, src, dst, symmetric):
    src, dst = np.asarray(src, np.int64), np.asarray(dst, np.int64)
    if symmetric:
        src, dst = np.r_[src, dst], np.r_[dst, src]
    key = np.unique(src * n + dst)
    src, dst = key // n, key % n
    offs = np.zeros(n + 1, np.uint32)
    offs[1:] = np.cumsum(np.bincount(src, minlength=n))
    cols = dst.astype(np.uint32)
    ref = oracle_mod.cc(oracle_mod.CSR(offs, cols))
    g = grus.Graph.from_csr(offs, cols, symmetric=symmetric)
    for _ in range(3):
        assert np.array_equal(grus.cc(g), ref)
    g.free()


@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 257, 5000, 1 << 17, (1 << 17) + 1, 700001])
def test_sizes(grus, oracle_mod, n, symmetric):
    """Sparse random edges: many components and, in the larger, a giant one."""
    rng = np.random.default_rng(n)
    m = n * 2 // 3
    _check(grus, oracle_mod, n, rng.integers(0, n, m), rng.integers(0, n, m), symmetric)


@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("n", [3000, 300000])
@pytest.mark.parametrize("kind", ["path", "shuffled", "ring", "star", "caterpillar", "cliques", "pairs", "ladder"])
def test_shapes(grus, oracle_mod, kind, n, symmetric):
    rng = np.random.default_rng(n)
    v = np.arange(n)
    if kind == "path":
        src, dst = v[:-1], v[1:]
    elif kind == "shuffled":
        p = rng.permutation(n)
        src, dst = p[:-1], p[1:]
    elif kind == "ring":
        src, dst = v, (v + 1) % n
    elif kind == "star":
        src, dst = np.full(n - 1, n // 2), np.delete(v, n // 2)
    elif kind == "caterpillar":  # degrees rise along a path: parents form one chain
        k = int(np.sqrt(2 * n)) - 2
        legs = np.repeat(np.arange(k), np.arange(k))
        src, dst = np.r_[np.arange(k - 1), legs], np.r_[np.arange(1, k), k + np.arange(len(legs))]
    elif kind == "cliques":
        a = rng.integers(0, n // 2, 3 * n)
        b = rng.integers(0, n // 2, 3 * n)
        src, dst = np.r_[a, a + n // 2, 0], np.r_[b, b + n // 2, n - 1]
    elif kind == "pairs":
        src, dst = v[:n // 2], n - 1 - v[:n // 2]
    else:  # two rails, rungs at every tenth
        h = n // 2
        src = np.r_[v[:h - 1], v[h:2 * h - 1], v[:h:10]]
        dst = np.r_[v[1:h], v[h + 1:2 * h], v[h:2 * h:10]]
    _check(grus, oracle_mod, n, src, dst, symmetric)
