"""A solve that fits into the device's memory without what an earlier call left
behind for speed (here the column plan) is not refused because of it."""
import numpy as np
import pytest

from streamsim_gb300 import facetcu
from tests.gpu_helpers import require_gpu

pytestmark = pytest.mark.gpu


def test_solve_with_the_plan_in_the_way():
    require_gpu()
    torch = pytest.importorskip("torch")
    S, degree, bands = 40960, 272, 64
    rng = np.random.default_rng(8)
    F = S // 2
    v = np.zeros((3 * F, 6), np.float32)
    v[:, :3] = np.repeat(rng.uniform(-20, 20, (F, 3)), 3, 0) + np.tile(
        [[0, 0, 0], [0.1, 0, 0], [0, 0, -0.1]], (F, 1))
    v[:, 4] = 1.0
    nb = rng.integers(0, S, S * degree).astype(np.uint32)
    cnt = rng.integers(1, 4, S * degree).astype(np.uint32)
    sky = rng.integers(0, 50, S).astype(np.uint32)
    graph = ((np.arange(S + 1) * degree).astype(np.uint32), nb, cnt,
             cnt.reshape(S, degree).sum(1).astype(np.uint32) + sky, sky)
    rho = np.full((bands, S), 0.35, np.float32)
    tau = np.full((bands, S), 0.15, np.float32)
    dgeo = rng.uniform(0, 1, (1, S)).astype(np.float32)
    one = np.ones(bands, np.float32)

    def model():
        m = facetcu.FacetrtCuda()
        m.initialize(64, 64, 64)
        m.setGeometry(v)
        m.setGraph(*graph)
        return m

    def solve(m, n):
        out, res = m.solveBatched(rho[:n], tau[:n], 100.0 * one[:n], 500.0 * one[:n], dgeo,
                                  tolerance=1e-5)
        assert res["converged"]
        return out

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    m = model()
    before = free()
    want = solve(m, bands)
    need = before - free()  # of the 64 columns without a plan
    m.close()
    m = model()
    before = free()
    solve(m, 1)
    plan = before - free()
    assert plan > 40 << 20
    left = need - plan // 2
    rest = torch.empty(free() - left, dtype=torch.uint8, device="cuda")
    try:
        got = solve(m, bands)
    finally:
        del rest
        torch.cuda.empty_cache()
    m.close()
    assert np.array_equal(got, want)


def test_geometry_without_room_for_two():
    """Both geometries don't fit: the new one is checked in pieces (more than five
    here) and takes the old one's place; a refused one leaves the old one."""
    require_gpu()
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(2)
    F = 300_001

    def geometry(seed):
        g = np.random.default_rng(seed)
        v = np.zeros((F, 3, 6), np.float32)
        v[:, :, :3] = g.uniform(-8, 8, (F, 1, 3)) + g.uniform(-0.1, 0.1, (F, 3, 3))
        v[:, :, 4] = 1.0
        return v.reshape(-1, 6)

    a, b = geometry(1), geometry(2)
    b[rng.integers(0, len(b)), 0] = 9.5  # the bounds come from one vertex
    b[len(b) - 1, 2] = -9.75
    sun = np.float32([0.3, 0.9, 0.1])

    def model(v):
        m = facetcu.FacetrtCuda()
        m.initialize(64, 64, 1024)
        m.setGeometry(v)
        return m

    m = model(b)
    want = m.computeSunlitFraction(sun)
    m.close()
    m = model(a)
    torch.cuda.synchronize()
    rest = torch.empty(torch.cuda.mem_get_info()[0] - (12 << 20), dtype=torch.uint8, device="cuda")
    try:
        for at, value, match in ((len(b) - 1, np.nan, "non-finite"), (200_000, np.inf, "non-finite")):
            bad = b.copy()
            bad[at, 1] = value
            with pytest.raises(ValueError, match=match):
                m.setGeometry(bad)
        bad = b.copy()
        bad[300_000, 4], bad[800_000, 0] = 2.0, np.nan
        with pytest.raises(ValueError, match="normalized"):  # the earlier vertex
            m.setGeometry(bad)
        m.setGeometry(b)
    finally:
        del rest
        torch.cuda.empty_cache()
    got = m.computeSunlitFraction(sun)
    m.close()
    assert np.array_equal(got, want)


def test_graph_that_does_not_fit_leaves_none():
    """setGraph gives the old graph up before it allocates: where there is no room
    for the new one, solves are refused until a graph is set."""
    require_gpu()
    torch = pytest.importorskip("torch")
    S = 4096
    rng = np.random.default_rng(1)
    v = np.zeros((3 * S // 2, 6), np.float32)
    v[:, :3] = rng.uniform(-5, 5, (3 * S // 2, 3))
    v[:, 4] = 1.0

    def graph(degree):
        cnt = np.ones(S * degree, np.uint32)
        return ((np.arange(S + 1) * degree).astype(np.uint32),
                rng.integers(0, S, S * degree).astype(np.uint32), cnt,
                np.full(S, degree, np.uint32), np.zeros(S, np.uint32))

    small, large = graph(4), graph(2000)  # 64 MB of edges
    o = np.zeros((S, 4), np.float32)
    o[:, 0], o[:, 3] = 0.4, 1.0
    m = facetcu.FacetrtCuda()
    m.initialize(64, 64, 64)
    m.setGeometry(v)
    m.setGraph(*small)
    want = m.solve(o, 0.0, 20)["radiosity"]
    torch.cuda.synchronize()
    rest = torch.empty(torch.cuda.mem_get_info()[0] - (16 << 20), dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(facetcu.FacetcuError):
            m.setGraph(*large)
    finally:
        del rest
        torch.cuda.empty_cache()
    with pytest.raises(RuntimeError, match="buildVisibilityGraph"):
        m.solve(o, 0.0, 20)
    m.setGraph(*small)
    assert np.array_equal(m.solve(o, 0.0, 20)["radiosity"], want)
    m.close()
