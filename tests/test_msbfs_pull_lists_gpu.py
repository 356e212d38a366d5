"""GPU: multi-source BFS with every level a pull level, on hubs whose in-lists
end around the lengths that lanes, warps and all warps share.  Bit-exact
against the oracle; the pull levels are counted."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LANE, FIRST, SPLIT = 32, 16 * 1024, 32 * 1024


@pytest.mark.parametrize("where", ["first", "last"])
@pytest.mark.parametrize("length", [LANE + 1, LANE + 129, LANE + FIRST, LANE + SPLIT - 1, LANE + SPLIT,
                                    LANE + SPLIT + 1, 3 * SPLIT + 7])
def test_hub_lists_pulled(grus, oracle_mod, where, length):
    """Four hubs of `length` leaves; a hub misses the other hubs' bits until the
    one leaf that they share, the first or the last of its list."""
    hubs, priv = 4, length - 1
    base = hubs + 1 if where == "first" else hubs
    shared = hubs if where == "first" else hubs + hubs * priv
    n = hubs + hubs * priv + 1
    src = np.concatenate([np.r_[base + h * priv + np.arange(priv), shared] for h in range(hubs)])
    dst = np.repeat(np.arange(hubs), priv + 1)
    e = np.unique(np.r_[src * n + dst, dst * n + src])
    src, dst = e // n, e % n
    offs = np.zeros(n + 1, np.uint32)
    offs[1:] = np.cumsum(np.bincount(src, minlength=n))
    g = grus.Graph.from_csr(offs, dst.astype(np.uint32), symmetric=True)
    srcs = np.array([0, 1, 2, 3, n - 1, n - 2, 0], np.uint32)
    ref = oracle_mod.bfs_multi(oracle_mod.CSR(offs, dst.astype(np.uint32)), srcs)
    g.set_tuning(multi_alpha=1e9)
    got, st = grus.bfs_multi(g, srcs, stats=True)
    assert np.array_equal(got, ref)
    assert st["bottom_up_levels"] >= 2
    g.free()
