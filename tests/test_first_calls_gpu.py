"""GPU: a first call's workspace is cleared before its kernels run, on whatever
stream they run, and the call does not wait for other streams' work: here the
default stream is busy while each algorithm's first call runs on another."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _calls(grus, g, stream, torch):
    n = int(g.n)
    u32 = lambda *shape: torch.full(shape, -7, dtype=torch.int32, device="cuda")
    srcs = np.array([1, 2, 3], np.uint32)
    f32 = torch.full((n,), -7.0, dtype=torch.float32, device="cuda")
    return [
        ("bfs", lambda o: grus.bfs(g, 1, out=o, stream=stream), lambda: grus.bfs(g, 1), u32(n)),
        ("sssp", lambda o: grus.sssp(g, 1, out=o, stream=stream), lambda: grus.sssp(g, 1), u32(n)),
        ("cc", lambda o: grus.cc(g, out=o, stream=stream), lambda: grus.cc(g), u32(n)),
        ("pagerank", lambda o: grus.pagerank(g, 0.85, 5, out=o, stream=stream),
         lambda: grus.pagerank(g, 0.85, 5), f32),
        ("bfs_multi", lambda o: grus.bfs_multi(g, srcs, out=o, stream=stream),
         lambda: grus.bfs_multi(g, srcs), u32(3, n)),
        ("sssp_multi", lambda o: grus.sssp_multi(g, srcs, out=o, stream=stream),
         lambda: grus.sssp_multi(g, srcs), u32(3, n)),
    ]


@pytest.mark.parametrize("which", range(6))
def test_first_call_beside_a_busy_default_stream(grus, which):
    torch = pytest.importorskip("torch")
    stream = torch.cuda.Stream()
    graphs = []
    for seed in (4, 3):  # the first graph's call loads the kernels, which waits
        g = grus.Graph.rmat(17, 16, seed, symmetric=True, weighted=True)
        graphs.append(g)
        g.build_index()
        g.build_csc()
        name, call, again, out = _calls(grus, g, stream, torch)[which]
        if seed == 4:
            call(out)
        torch.cuda.synchronize()
    busy = torch.cuda.Event()
    torch.cuda._sleep(1 << 30)  # about half a second of the default stream
    busy.record()
    call(out)
    stream.synchronize()
    # (PageRank needs all SMs for itself, the multi-source calls copy their sources
    # on the default stream first)
    if name in ("bfs", "sssp", "cc"):
        assert not busy.query(), name
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    ref = np.asarray(again())
    assert np.array_equal(got.view(ref.dtype), ref)
    for g in graphs:
        g.free()
