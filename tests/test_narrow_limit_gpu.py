"""GPU: the time limit of the one-cluster kernel.  A step that takes longer than
`timeout_ms` ends the traversal with the timeout status, and the graph's
workspace serves the next call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_long_step_ends_with_the_timeout_status(grus):
    """A settled hub of 12 M leaves is improved after the hand-over: one step of
    several milliseconds in the cluster (the grid's waits are well below one)."""
    path, leaves = 60, 12000000
    n = path + 1 + leaves
    deg = np.zeros(n, np.int64)
    deg[:path] = 1
    deg[0] = 2
    deg[path] = leaves
    offs = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint32)
    cols = np.concatenate([[1, path], np.arange(2, path + 1), np.arange(path + 1, n)]).astype(np.uint32)
    wts = np.concatenate([[1, 600], np.ones(path - 1), np.full(leaves, 5)]).astype(np.uint32)
    ref = np.concatenate([np.arange(path + 1), np.full(leaves, path + 5)]).astype(np.uint32)
    g = grus.Graph.from_csr(offs, cols, wts, symmetric=False)
    g.set_tuning(tail_cluster=2, timeout_ms=1)
    assert np.array_equal(grus.sssp(g, 0), ref)  # the grid alone keeps the limit
    g.set_tuning(tail_cluster=0, timeout_ms=1)
    with pytest.raises(grus.GrusError) as e:
        grus.sssp(g, 0, stats=True)
    assert e.value.status == grus.ETIMEDOUT
    g.set_tuning(tail_cluster=0, timeout_ms=0)
    for _ in range(2):
        assert np.array_equal(grus.sssp(g, 0), ref)
    g.free()
