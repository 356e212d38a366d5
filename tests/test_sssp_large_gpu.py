"""GPU: single-source SSSP on graphs around the size from which the CTAs take a
level's tiles in turn, against the multi-source kernel's row (another kernel,
itself compared with the oracle) and for the properties of distances."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,ef", [(21, 15), (21, 20), (22, 16)])
def test_taken_tiles(grus, scale, ef):
    torch = pytest.importorskip("torch")
    g = grus.Graph.rmat(scale, ef, 5, symmetric=True, weighted=True)
    assert (g.m >= 1 << 26) == (ef > 15)
    rng = np.random.default_rng(scale)
    srcs = np.array([g.max_degree_vertex, rng.integers(g.n), 0], np.uint32)
    rows = torch.empty((len(srcs), g.n), dtype=torch.int32, device="cuda")
    grus.sssp_multi(g, srcs, out=rows)
    for i, s in enumerate(srcs):
        for _ in range(2):
            out = torch.full((g.n,), -3, dtype=torch.int32, device="cuda")
            grus.sssp(g, int(s), out=out)
            torch.cuda.synchronize()
            assert torch.equal(out, rows[i])
        assert int(out[int(s)]) == 0
    g.free()
