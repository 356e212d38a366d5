"""GPU: multi-source SSSP where the dealing of entries and lanes can go wrong:
out-degrees around the lanes of an entry and the edges of a piece, source
counts around the widths of a row, mean degrees around each width of an
entry's lanes, and enough entries of a skewed graph that warps take them in
turn.  Bit-exact against the oracle's single-source runs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(n, src, dst, seed):
    key = np.unique(src.astype(np.int64) * n + dst)
    src, dst = key // n, key % n
    offs = np.zeros(n + 1, np.uint32)
    offs[1:] = np.cumsum(np.bincount(src, minlength=n))
    w = np.random.default_rng(seed).integers(1, 256, len(dst)).astype(np.uint32)
    return offs, dst.astype(np.uint32), w


def _check(grus, oracle_mod, csr, srcs, rows=None, delta=0):
    offs, cols, wts = csr
    g = grus.Graph.from_csr(offs, cols, wts)
    if delta:
        g.set_tuning(sssp_delta=delta)
    got, st = grus.sssp_multi(g, srcs, stats=True)
    h = oracle_mod.CSR(offs, cols, wts)
    for i in range(len(srcs)) if rows is None else rows:
        assert np.array_equal(got[i], oracle_mod.sssp(h, int(srcs[i]))), i
    assert st["vertices_reached"] == int(np.count_nonzero(got != 4294967294))
    g.free()


@pytest.mark.parametrize("k", [1, 8, 9, 16, 17, 31, 32])
@pytest.mark.parametrize("deg", [1, 4, 5, 31, 32, 33, 127, 128, 129, 511, 512, 513])
def test_degrees(grus, oracle_mod, k, deg):
    """A tenth of the vertices have `deg` out-edges, the others one or two;
    the sources are of both kinds, some of them repeated."""
    n = 3000
    rng = np.random.default_rng(deg)
    some = np.arange(0, n, 10)
    src = np.r_[np.repeat(some, deg), np.arange(n), rng.integers(0, n, n)]
    csr = _graph(n, src, rng.integers(0, n, len(src)), deg)
    srcs = rng.integers(0, n, k).astype(np.uint32)
    srcs[k // 2] = srcs[0]
    _check(grus, oracle_mod, csr, srcs, rows=range(0, k, 3), delta=(0, 64)[deg % 2])


@pytest.mark.parametrize("k", [8, 16, 32])
@pytest.mark.parametrize("mean", [1, 4, 5, 8, 16, 17, 33])
def test_mean_degrees(grus, oracle_mod, k, mean):
    n = 5000
    rng = np.random.default_rng(mean)
    src = np.repeat(np.arange(n), mean)
    csr = _graph(n, src, rng.integers(0, n, len(src)), mean)
    _check(grus, oracle_mod, csr, rng.integers(0, n, k).astype(np.uint32), rows=range(0, k, 5))


@pytest.mark.parametrize("hub", [511, 512, 60000])
def test_entries_taken_in_turn(grus, oracle_mod, hub):
    """More than eight entries a warp, with and without long lists."""
    n = 200000
    rng = np.random.default_rng(hub)
    src = np.r_[np.repeat(np.arange(n), 3), np.full(hub - 3, 7)]
    dst = rng.integers(0, n, len(src))
    dst[-(hub - 3):] = rng.choice(n, hub - 3, replace=False)
    srcs = np.r_[7, rng.integers(0, n, 31)].astype(np.uint32)
    _check(grus, oracle_mod, _graph(n, src, dst, hub), srcs, rows=(0, 1, 16, 31))
