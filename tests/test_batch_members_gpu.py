"""GPU: multi-source groups whose staging grows between runs that also have
whole-GPU launches, whose error words must stay where they are."""
import numpy as np
import pytest


@pytest.mark.gpu
def test_group_staging_grows_beside_big_graphs(grus):
    torch = pytest.importorskip("torch")
    gs = [grus.Graph.rmat(13, 16, 1, symmetric=True, weighted=True),
          grus.Graph.rmat(9, 8, 2, symmetric=True, weighted=True)]
    b = grus.Batch(gs, group_sources=8, big_edges=1 << 16)
    rng = np.random.default_rng(1)
    for small in (4, 40, 200, 3):
        queries = [(0, a, int(rng.integers(gs[0].n))) for a in (grus.ALGO_SSSP, grus.ALGO_BFS) for _ in range(3)]
        queries += [(1, grus.ALGO_SSSP, int(rng.integers(gs[1].n))) for _ in range(small)]
        offs, total = b.layout(queries)
        out = torch.full((total,), -7, dtype=torch.int32, device="cuda")
        # stats: the error words of the big graph's launches are read back
        assert b.run(queries, out, offs, stats=True)["kernel_launches"] >= 2
        res = out.cpu().numpy().view(np.uint32)
        for (gi, algo, src), o in zip(queries, offs):
            ref = (grus.sssp if algo == grus.ALGO_SSSP else grus.bfs)(gs[gi], src)
            assert np.array_equal(res[o:o + len(ref)], ref), (small, gi, algo, src)
    b.free()
    torch.cuda.synchronize()
    for g in gs:
        g.free()


def test_growing_the_staging_frees_only_the_staging():
    """The function that grows the members' staging touches no other buffer."""
    from pathlib import Path
    text = (Path(__file__).resolve().parents[1] / "grus_framework_gb300/csrc/batch.cu").read_text()
    body = text[text.index("static int ensure_members("):]
    body = body[:body.index("\n}\n")]
    freed = {line.split("(b->")[1].split(")")[0] for line in body.splitlines() if "cudaFree" in line}
    assert freed == {"d_msrc", "d_moff", "h_msrc", "h_moff"}
