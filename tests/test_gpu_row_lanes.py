"""The CSR sweep at the edges of its rule for lanes per side (mean rows of 4, 10
and 48 edges), through solve() and through solve_noalloc, which reads the mean on
the device and walks the sides with a fixed grid, against a float64 iteration."""
import ctypes as C

import numpy as np
import pytest

from streamsim_gb300 import facetcu
from tests.gpu_helpers import require_gpu
from tests.test_gpu_one_column import SKY, _graph, _jacobi, _model, _optics, _tolerance

pytestmark = pytest.mark.gpu


# 4 and 62 sides: less than a block; 160,000 of 16 lanes: more than the fixed grid
@pytest.mark.parametrize("S", [4, 62, 5002, 160002])
@pytest.mark.parametrize("mean", [0, 1, 3, 4, 9, 10, 47, 48])
def test_lanes(S, mean):
    require_gpu()
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(S + mean)
    deg = np.full(S, mean)
    deg[: S // 2], deg[S // 2:] = mean + mean // 2, mean - mean // 2  # sums to S * mean
    graph = _graph(S, deg, rng, counts=[255, 70000] if mean else None)
    assert int(graph[0][-1]) == S * mean
    o = _optics(S, rng)
    m = _model(S, graph)
    got = m.solve(o, SKY, 5, 0.75)["radiosity"]
    m.close()
    rows, nb, cnt, den, sky = graph
    edges = np.empty(2 * len(nb) + 2, np.uint32)
    edges[0:2 * len(nb):2], edges[1:2 * len(nb):2] = nb, cnt
    d = [torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda()
         for a in (rows, edges, den, sky, o)]
    out = torch.full((S,), -1.0, device="cuda")
    torch.cuda.synchronize()
    p = [C.c_void_p(a.data_ptr()) for a in d]
    md = C.c_float()
    assert facetcu.load().facetcu_solve_noalloc(
        p[0], p[1], p[2], p[3], S, p[4], SKY, 5, 0.75, C.c_void_p(out.data_ptr()), C.byref(md),
        None) == facetcu.OK
    want = _jacobi(graph, o[:, 3].astype(np.float64), o[:, 2].astype(np.float64), 5, 0.75)
    for b in (got, out.cpu().numpy()):
        assert np.max(np.abs(b - want) / want) < _tolerance(graph)
    if S > 4096:  # one sweep kernel for both: the same order of additions
        assert np.array_equal(got, out.cpu().numpy())


@pytest.mark.parametrize("mean", [63, 64, 65])
def test_rows_around_the_cluster_limit(mean):
    """Small graphs whose rows are too long for the cluster go to the sweeps."""
    require_gpu()
    S = 250
    rng = np.random.default_rng(mean)
    graph = _graph(S, np.full(S, mean), rng, counts=[255, 256, 65535])
    o = _optics(S, rng)
    m = _model(S, graph)
    got = m.solve(o, SKY, 16, 0.75)["radiosity"]
    m.close()
    want = _jacobi(graph, o[:, 3].astype(np.float64), o[:, 2].astype(np.float64), 16, 0.75)
    assert np.max(np.abs(got - want) / want) < _tolerance(graph)
