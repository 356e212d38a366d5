"""GPU: PageRank where its work split can go wrong, against the FP64 oracle
within the package's bars (maximum relative error 1e-4, L1 1e-6): graphs at the
size that still fits shared memory, in-lists around the length that warps may
share, one list shared by many warps, vertices without in- or out-edges, few
iterations (no relabelled columns) and more on the same graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(n, src, dst):
    key = np.unique(src.astype(np.int64) * n + dst)
    src, dst = key // n, key % n
    offs = np.zeros(n + 1, np.uint32)
    offs[1:] = np.cumsum(np.bincount(src, minlength=n))
    return offs, dst.astype(np.uint32)


def _check(grus, oracle_mod, offs, cols, iters=(1, 2, 3, 20, 1)):
    csr = oracle_mod.CSR(offs, cols)
    g = grus.Graph.from_csr(offs, cols)
    for it in iters:
        ref = oracle_mod.pagerank(csr, 0.85, it)
        got = grus.pagerank(g, 0.85, it).astype(np.float64)
        err = np.abs(got - ref)
        assert (err / ref).max() <= 1e-4 and err.sum() <= 1e-6, it
    g.free()


@pytest.mark.parametrize("n", [1, 2, 31, 33, 1000, 47999, 48000, 48001, 70001])
def test_sizes(grus, oracle_mod, n):
    rng = np.random.default_rng(n)
    m = 3 * n
    # sources skewed towards small ids, so that the larger sizes get a plan
    src = (n * rng.random(m) ** 4).astype(np.int64)
    _check(grus, oracle_mod, *_csr(n, src, rng.integers(0, n, m)))


@pytest.mark.parametrize("n", [3000, 90000])
@pytest.mark.parametrize("deg", [15, 16, 63, 64, 65, 255, 256, 257])
def test_list_lengths(grus, oracle_mod, n, deg):
    """Every tenth vertex has `deg` in-edges, the others none or one."""
    rng = np.random.default_rng(deg)
    hubs = np.arange(0, n, 10)
    src = (n * rng.random(len(hubs) * deg) ** 3).astype(np.int64)
    dst = np.repeat(hubs, deg)
    some = rng.integers(0, n, n // 3)
    _check(grus, oracle_mod, *_csr(n, np.r_[src, some], np.r_[dst, (some * 7 + 1) % n]), iters=(3, 20))


@pytest.mark.parametrize("n", [40000, 400000])
def test_one_list_shared_by_many_warps(grus, oracle_mod, n):
    """Half of all vertices point at one, a quarter at another, and the first
    vertices point at everything in a stretch: lists and shares of all mixes."""
    rng = np.random.default_rng(1)
    a = np.arange(n // 2)
    b = np.arange(n // 4)
    c = np.repeat(np.arange(20), n // 10)
    src = np.r_[a, b, c, rng.integers(0, n, n)]
    dst = np.r_[np.full(n // 2, n - 1), np.full(n // 4, n // 3),
                rng.integers(n // 2, n, len(c)), rng.integers(0, n, n)]
    _check(grus, oracle_mod, *_csr(n, src, dst), iters=(1, 20))


def test_equal_degrees_at_the_cut(grus, oracle_mod):
    """All vertices have the same out-degree: which of them get the places in
    shared memory is arbitrary, and a quarter of the edges does not pass."""
    for n in (60000, 150000):
        i = np.arange(n)
        src = np.repeat(i, 4)
        dst = (src * 31 + np.tile([1, 77, 4001, 30011], n)) % n
        _check(grus, oracle_mod, *_csr(n, src, dst), iters=(20,))
