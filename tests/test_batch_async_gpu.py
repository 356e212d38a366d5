"""GPU: runs of a default batch on small graphs only queue work, also where
their SSSP queries join multi-graph launches and a later run needs more room."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_runs_do_not_wait_for_the_device(grus):
    torch = pytest.importorskip("torch")
    gs = [grus.Graph.rmat(10 + i % 5, 16, i, symmetric=True, weighted=True) for i in range(8)]
    b = grus.Batch(gs)
    rng = np.random.default_rng(0)
    stream = torch.cuda.Stream()
    runs = []
    for count in (1, 8, 33):
        queries = [(i, grus.ALGO_SSSP, int(rng.integers(g.n))) for i, g in enumerate(gs) for _ in range(count)]
        offs, total = b.layout(queries)
        runs.append((queries, offs, torch.full((total,), -7, dtype=torch.int32, device="cuda")))
    torch.cuda.synchronize()
    for queries, offs, out in runs:
        done = torch.cuda.Event()
        with torch.cuda.stream(stream):
            torch.cuda._sleep(1 << 30)  # about half a second of the stream
        b.run(queries, out, offs, stream=stream)
        done.record(stream)
        assert not done.query(), len(queries)
        stream.synchronize()
        res = out.cpu().numpy().view(np.uint32)
        for (gi, _, src), o in zip(queries, offs):
            ref = grus.sssp(gs[gi], src)
            assert np.array_equal(res[o:o + len(ref)], ref), (gi, src)
    # packed, not left to the workers: one query each is one multi-graph launch
    assert b.run(*[runs[0][i] for i in (0, 2, 1)], stats=True)["kernel_launches"] == 1
    b.free()
    for g in gs:
        g.free()
