"""GPU: 64-source BFS where a pull level searches long in-lists: hubs whose
lists end around the lengths that lanes, warps and all warps share, with the
bit that a hub misses in its last, its first or no in-edge.  Bit-exact against
the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LANE, FIRST, SPLIT = 32, 16 * 1024, 32 * 1024


@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("where", ["first", "last", "none"])
@pytest.mark.parametrize("length", [LANE + 1, LANE + 128, LANE + 129, LANE + FIRST, LANE + SPLIT - 1, LANE + SPLIT,
                                    LANE + SPLIT + 1, LANE + SPLIT + 1024, 3 * SPLIT + 7])
def test_hub_lists(grus, oracle_mod, symmetric, where, length):
    """Four hubs of `length` leaves each; every hub is a source, so the level
    after theirs has all leaves in the frontier.  The hubs share one leaf: the
    first or the last of their lists, or none (a chain joins them instead)."""
    hubs, priv = 4, length - 1
    base = hubs + 1 if where == "first" else hubs
    shared = hubs if where == "first" else hubs + hubs * priv
    n = hubs + hubs * priv + 1
    src, dst = [], []
    for h in range(hubs):
        leaves = base + h * priv + np.arange(priv)
        src.append(np.r_[leaves, shared] if where != "none" else leaves)
        dst.append(np.full(len(src[-1]), h))
    src, dst = np.concatenate(src), np.concatenate(dst)
    if where == "none":
        chain = base + np.arange(hubs) * priv
        src, dst = np.r_[src, chain[:-1]], np.r_[dst, chain[1:]]
    e = np.unique(np.r_[src * n + dst, dst * n + src])
    src, dst = e // n, e % n
    if not symmetric:  # one direction of some of the leaves' edges only
        keep = (src < hubs) | (dst < hubs - 1) | (src % 3 != 0)
        src, dst = src[keep], dst[keep]
    offs = np.zeros(n + 1, np.uint32)
    offs[1:] = np.cumsum(np.bincount(src, minlength=n))
    g = grus.Graph.from_csr(offs, dst.astype(np.uint32), symmetric=symmetric)
    if not symmetric:
        g.build_csc()
    csr = oracle_mod.CSR(offs, dst.astype(np.uint32))
    srcs = np.array([0, 1, 2, 3, n - 1, n - 2, 0], np.uint32)
    ref = oracle_mod.bfs_multi(csr, srcs)
    for alpha in (0, 1e6):  # the default rule, and pull levels from the start on
        g.set_tuning(multi_alpha=1 / alpha if alpha else 0)
        got, st = grus.bfs_multi(g, srcs, stats=True)
        assert np.array_equal(got, ref)
        assert st["vertices_reached"] == int(np.count_nonzero(ref != 4294967294))
    g.free()
