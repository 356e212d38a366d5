"""GPU: single BFS launches of a batch beside one another."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_one_handle_at_two_indices(grus):
    """Both indices' launches use the one handle's workspace."""
    torch = pytest.importorskip("torch")
    gs = [grus.Graph.rmat(17, 16, i, symmetric=True, weighted=True) for i in range(2)]
    b = grus.Batch([gs[0], gs[1], gs[0], gs[0]])
    rng = np.random.default_rng(5)
    queries = [(i, grus.ALGO_BFS, int(rng.integers(gs[0].n))) for i in (0, 1, 2, 3, 2, 0, 1)]
    offs, total = b.layout(queries)
    refs = [grus.bfs(gs[0] if i != 1 else gs[1], src) for i, _, src in queries]
    for _ in range(5):
        out = torch.full((total,), -7, dtype=torch.int32, device="cuda")
        b.run(queries, out, offs)
        torch.cuda.synchronize()
        res = out.cpu().numpy().view(np.uint32)
        for q, o, ref in zip(queries, offs, refs):
            assert np.array_equal(res[o:o + len(ref)], ref), q
    b.free()
    for g in gs:
        g.free()


@pytest.mark.parametrize("small,per", [(1, 1), (3, 3), (4, 9)])
def test_beside_the_workers(grus, small, per):
    """Three, two and no side streams beside the workers' kernel (9, 36 and 72
    tasks on the small graphs), replayed and not."""
    torch = pytest.importorskip("torch")
    gs = [grus.Graph.rmat(17, 16, i, symmetric=True) for i in range(4)]
    gs += [grus.Graph.rmat(12, 16, 10 + i, symmetric=True) for i in range(small)]
    b = grus.Batch(gs)
    rng = np.random.default_rng(per)
    queries = [(i, grus.ALGO_BFS, int(rng.integers(g.n))) for i, g in enumerate(gs)
               for _ in range(2 if i < 4 else per * (2 if small > 3 else 4 if small > 1 else 9))]
    offs, total = b.layout(queries)
    refs = [grus.bfs(gs[i], src) for i, _, src in queries]
    for replay in (False, True, True):
        out = torch.full((total,), -7, dtype=torch.int32, device="cuda")
        b.run(queries, out, offs, use_graph=replay)
        torch.cuda.synchronize()
        res = out.cpu().numpy().view(np.uint32)
        for q, o, ref in zip(queries, offs, refs):
            assert np.array_equal(res[o:o + len(ref)], ref), (q, replay)
    b.free()
    for g in gs:
        g.free()
