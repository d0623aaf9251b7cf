"""One-column sweeps on the device against a float64 Jacobi iteration in numpy:
the CSR kernel (k_jacobi_rows) at the edges of its lane groups.

Tolerance: a sweep adds at most `deg` products in FP32, so a row's relative
error per sweep is below (deg + 8) 2^-24, and the iteration (rho + tau = c)
multiplies it by at most 1 / (1 - c)."""
import numpy as np
import pytest

from streamsim_gb300 import facetcu
from tests.gpu_helpers import require_gpu

pytestmark = pytest.mark.gpu

RHO, TAU, SKY = 0.35, 0.15, 100.0


def _graph(S, degrees, rng, counts=None):
    """Rows of the given lengths with unsorted neighbours (some repeated)."""
    rows = np.zeros(S + 1, np.int64)
    rows[1:] = np.cumsum(degrees)
    n = int(rows[-1])
    nb = rng.integers(0, S, n).astype(np.uint32)
    cnt = rng.integers(1, 4, n).astype(np.uint32)
    if counts is not None and n:
        cnt[rng.choice(n, len(counts) * 20)] = np.tile(counts, 20)
    sky = rng.integers(0, 50, S).astype(np.uint32)
    sums = np.add.reduceat(np.append(cnt, 0).astype(np.int64), np.minimum(rows[:-1], n))
    sums[degrees == 0] = 0
    den = (sums + sky).astype(np.uint32)
    return rows.astype(np.uint32), nb, cnt, den, sky


def _model(S, graph):
    rng = np.random.default_rng(5)
    F = S // 2
    v = np.zeros((3 * F, 6), np.float32)
    c = np.repeat(rng.uniform(-20, 20, (F, 3)), 3, 0)
    v[:, :3] = c + np.tile([[0, 0, 0], [0.1, 0, 0], [0, 0, -0.1]], (F, 1))
    v[:, 4] = 1.0
    m = facetcu.FacetrtCuda()
    m.initialize(64, 64, 64)
    m.setGeometry(v)
    m.setGraph(*graph)
    return m


def _incident(graph, B):
    import scipy.sparse as sp
    rows, nb, cnt, den, sky = graph
    S = len(den)
    A = sp.csr_matrix((cnt.astype(np.float64), nb.astype(np.int64), rows.astype(np.int64)), (S, S))
    d = np.maximum(den, 1)
    return np.where(den > 0, (sky * SKY + A @ B) / d, SKY)


def _jacobi(graph, direct, emis, sweeps, relax=1.0):
    B = np.zeros(len(direct))
    for _ in range(sweeps):
        H = _incident(graph, B) + direct
        T = emis + RHO * H + TAU * H.reshape(-1, 2)[:, ::-1].ravel()
        B = B * (1 - relax) + T * relax
    return B


def _optics(S, rng):
    o = np.zeros((S, 4), np.float32)
    o[:, 0], o[:, 1] = RHO, TAU
    o[:, 2] = rng.uniform(0, 5, S)
    o[:, 3] = rng.uniform(0, 800, S)
    return o


def _tolerance(graph):
    deg = int(np.diff(graph[0].astype(np.int64)).max())
    return (deg + 8) * 2.0 ** -24 / (1 - np.float32(RHO) - np.float32(TAU)) + 1e-7


@pytest.mark.parametrize("mean", [2, 20, 90])  # 4, 8 and 16 lanes per side
@pytest.mark.parametrize("S", [2, 62, 1030])
def test_csr_sweep_lane_groups(S, mean):
    require_gpu()
    rng = np.random.default_rng(S + mean)
    edge = np.array([0, 1, mean, 2 * mean, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 129])
    deg = np.resize(edge[edge <= max(4, 3 * mean)], S)
    graph = _graph(S, deg, rng, counts=[70000, 255, 256, 300])
    o = _optics(S, rng)
    m = _model(S, graph)
    got = m.solve(o, SKY, 9, 0.75)["radiosity"]
    m.close()
    want = _jacobi(graph, o[:, 3].astype(np.float64), o[:, 2].astype(np.float64), 9, 0.75)
    assert np.max(np.abs(got - want) / want) < _tolerance(graph)
