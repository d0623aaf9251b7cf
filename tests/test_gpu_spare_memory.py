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
