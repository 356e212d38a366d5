"""GPU: PageRank calls with device outputs only queue work, the first ones on a
graph too (its column ids are relabelled in the first), and a program that has
made one call can capture the next."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _skewed(grus, n=200000, m=2000000, seed=2):
    rng = np.random.default_rng(seed)
    src = (n * rng.random(m) ** 4).astype(np.int64)
    key = np.unique(src * n + rng.integers(0, n, m))
    offs = np.zeros(n + 1, np.uint32)
    offs[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    g = grus.Graph.from_csr(offs, (key % n).astype(np.uint32), symmetric=False)
    g.build_csc()
    return g


@pytest.mark.parametrize("scale", [0, 18, 20])
def test_calls_do_not_wait_for_the_stream(grus, scale):
    torch = pytest.importorskip("torch")
    g = grus.Graph.rmat(scale, 16, 3, symmetric=False) if scale else _skewed(grus)
    g.build_csc()
    outs = [torch.zeros(int(g.n), dtype=torch.float32, device="cuda") for _ in range(4)]
    warm = grus.Graph.rmat(10, 4, 1, symmetric=False)
    grus.pagerank(warm, 0.85, 3)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    for i, out in enumerate(outs[:3]):
        done = torch.cuda.Event()
        with torch.cuda.stream(stream):
            torch.cuda._sleep(1 << 30)  # about half a second of the stream
        t0 = time.perf_counter()
        grus.pagerank(g, 0.85, 20, out=out, stream=stream)
        dt = time.perf_counter() - t0
        done.record(stream)
        assert not done.query(), (i, dt)
        stream.synchronize()
    grus.pagerank(g, 0.85, 20, out=outs[3])
    torch.cuda.synchronize()
    for out in outs[:3]:
        assert torch.equal(out, outs[3])
    g.free()
    warm.free()


@pytest.mark.parametrize("first", [1, 20])
def test_capture_after_one_call(grus, oracle_mod, first):
    torch = pytest.importorskip("torch")
    g = _skewed(grus)
    offs, cols, _ = g.copy_csr()
    out = torch.zeros(int(g.n), dtype=torch.float32, device="cuda")
    grus.pagerank(g, 0.85, first, out=out)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    stream = torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=stream):
        grus.pagerank(g, 0.85, 20, out=out, stream=stream)
    ref = oracle_mod.pagerank(oracle_mod.CSR(offs, cols), 0.85, 20)
    for _ in range(3):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        got = out.cpu().numpy().astype(np.float64)
        assert (np.abs(got - ref) / ref).max() <= 1e-4
    direct = torch.empty_like(out)
    grus.pagerank(g, 0.85, 20, out=direct)
    torch.cuda.synchronize()
    assert torch.equal(direct, out)
    g.free()
