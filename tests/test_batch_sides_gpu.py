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
