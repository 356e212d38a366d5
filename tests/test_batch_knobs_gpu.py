"""GPU: every setting of the workers keeps small graphs' SSSP queries with them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("setting", [{}, {"cluster_size": 8}, {"workers": 20}, {"huge_degree": 64},
                                     {"sssp_delta": 100}, {"group_sources": 4}, {"big_edges": 1 << 21}])
def test_settings_of_the_workers_reach_the_queries(grus, setting):
    torch = pytest.importorskip("torch")
    gs = [grus.Graph.rmat(10 + i % 5, 16, i, symmetric=True, weighted=True) for i in range(8)]
    rng = np.random.default_rng(0)
    # 70 sources on one graph are three packs, the workers' kernel is one
    queries = [(i, grus.ALGO_SSSP, int(rng.integers(g.n))) for i, g in enumerate(gs)
               for _ in range(70 if i == 0 else 8)]
    b = grus.Batch(gs, **setting)
    offs, total = b.layout(queries)
    out = torch.full((total,), -7, dtype=torch.int32, device="cuda")
    st = b.run(queries, out, offs, stats=True)
    assert st["kernel_launches"] == (1 if setting else 3), setting
    res = out.cpu().numpy().view(np.uint32)
    for (gi, _, src), o in zip(queries, offs):
        ref = grus.sssp(gs[gi], src)
        assert np.array_equal(res[o:o + len(ref)], ref), (gi, src)
    b.free()
    for g in gs:
        g.free()
