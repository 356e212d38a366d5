"""GPU: batches whose SSSP queries on small graphs may join whole-GPU
multi-graph launches: one graph alone, several with and without big graphs and
BFS queries, sources past a pack, and graphs that have to stay with the
workers.  Every result equals the single query's, with and without replay."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graphs(grus, kind):
    rmat = lambda scale, seed: grus.Graph.rmat(scale, 16, seed, symmetric=True, weighted=True)
    return {
        "one": lambda: [rmat(14, 1)],
        "several": lambda: [rmat(10 + i % 5, i) for i in range(8)],
        "big": lambda: [rmat(13, 1), rmat(17, 2), rmat(14, 3)],
        "grids": lambda: [grus.Graph.grid2d(30, 40, seed=i, weighted=True) for i in range(3)] + [rmat(14, 5)],
        "many": lambda: [rmat(8, i) for i in range(70)],
    }[kind]()


@pytest.mark.parametrize("kind,sssp,bfs", [("one", 1, 0), ("one", 8, 1), ("one", 33, 0), ("several", 1, 0),
                                           ("several", 9, 2), ("big", 6, 2), ("grids", 4, 1), ("many", 2, 0)])
def test_packs(grus, kind, sssp, bfs):
    torch = pytest.importorskip("torch")
    gs = _graphs(grus, kind)
    rng = np.random.default_rng(sssp)
    queries = [(i, grus.ALGO_SSSP, int(rng.integers(g.n))) for i, g in enumerate(gs) for _ in range(sssp)]
    queries += [(i, grus.ALGO_BFS, int(rng.integers(g.n))) for i, g in enumerate(gs) for _ in range(bfs)]
    queries = [queries[i] for i in rng.permutation(len(queries))]
    b = grus.Batch(gs)
    offs, total = b.layout(queries)
    refs = [(grus.sssp if algo == grus.ALGO_SSSP else grus.bfs)(gs[gi], src) for gi, algo, src in queries]
    for replay in (False, True, True):
        out = torch.full((total,), -7, dtype=torch.int32, device="cuda")
        st = b.run(queries, out, offs, use_graph=replay, stats=not replay)
        torch.cuda.synchronize()
        res = out.cpu().numpy().view(np.uint32)
        for q, o, ref in zip(queries, offs, refs):
            assert np.array_equal(res[o:o + len(ref)], ref), q
        assert replay or st["kernel_launches"] >= 1
    # the queries take the workers when the caller sets their sizes
    w = grus.Batch(gs, cluster_size=8)
    out = torch.full((total,), -7, dtype=torch.int32, device="cuda")
    w.run(queries, out, offs, stats=True)
    res = out.cpu().numpy().view(np.uint32)
    assert all(np.array_equal(res[o:o + len(ref)], ref) for o, ref in zip(offs, refs))
    w.free()
    b.free()
    for g in gs:
        g.free()


def test_big_bfs_side_by_side(grus):
    """BFS queries on several big graphs, several on each, beside packs and
    workers' tasks: two runs of one batch follow each other on the caller's
    stream, and each output is complete when that stream reaches its copy."""
    torch = pytest.importorskip("torch")
    gs = [grus.Graph.rmat(17, 16, i, symmetric=True, weighted=True) for i in range(5)]
    gs.append(grus.Graph.rmat(13, 8, 9, symmetric=True, weighted=True))
    rng = np.random.default_rng(3)
    b = grus.Batch(gs)
    sets = []
    for k in (1, 3):
        q = [(i, grus.ALGO_BFS, int(rng.integers(g.n))) for i, g in enumerate(gs) for _ in range(k)]
        q += [(i, grus.ALGO_SSSP, int(rng.integers(gs[i].n))) for i in (0, 5)]
        sets.append([q[i] for i in rng.permutation(len(q))])
    stream = torch.cuda.Stream()
    copies = []
    with torch.cuda.stream(stream):
        for q in sets + sets:
            offs, total = b.layout(q)
            out = torch.full((total,), -7, dtype=torch.int32, device="cuda")
            b.run(q, out, offs, use_graph=len(copies) % 2 == 1, stream=stream)
            copies.append((q, offs, out.clone()))
            out.fill_(-9)
    stream.synchronize()
    for q, offs, out in copies:
        res = out.cpu().numpy().view(np.uint32)
        for (gi, algo, src), o in zip(q, offs):
            ref = (grus.sssp if algo == grus.ALGO_SSSP else grus.bfs)(gs[gi], src)
            assert np.array_equal(res[o:o + len(ref)], ref), (gi, algo, src)
    b.free()
    for g in gs:
        g.free()
