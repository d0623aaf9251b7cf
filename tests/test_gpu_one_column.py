"""Sweeps of one and of a few columns on the device against a float64 Jacobi iteration in numpy:
the CSR kernel (k_jacobi_rows) at the edges of its lane groups, and the
shared-memory plan (column.cu) at the edges of its tiles, windows and groups,
and the 8- and 16-column panels (k_sweep_mid) at the edges of their rounds.

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


# sides: one tile less 2, exactly one tile, a second tile of 2 sides, and a
# ragged last window; row lengths with empty rows and one far above the rest
@pytest.fixture(scope="module", params=[49150, 49152, 49154, 102402])
def planned(request):
    require_gpu()
    S = request.param
    rng = np.random.default_rng(S)
    deg = rng.integers(150, 330, S)
    deg[rng.choice(S, S // 50)] = 0
    deg[rng.choice(S, 200)] = np.arange(1, 201) % 40
    deg[7] = 3000
    graph = _graph(S, deg, rng, counts=[255, 256, 257, 511, 512, 4097, 65535])
    assert int(graph[0][-1]) >= 10 << 20  # large enough for the plan
    m = _model(S, graph)
    yield dict(S=S, graph=graph, model=m, optics=_optics(S, rng))
    m.close()


def test_planned_sweep(planned):
    o = planned["optics"]
    got = planned["model"].solve(o, SKY, 12, 0.75)["radiosity"]
    want = _jacobi(planned["graph"], o[:, 3].astype(np.float64), o[:, 2].astype(np.float64), 12,
                   0.75)
    assert np.max(np.abs(got - want) / want) < _tolerance(planned["graph"])
    again = planned["model"].solve(o, SKY, 12, 0.75)["radiosity"]
    assert np.array_equal(got, again)


@pytest.mark.parametrize("precision", [facetcu.PRECISION_FP32, facetcu.PRECISION_MIXED])
def test_planned_panel(planned, precision):
    S, o = planned["S"], planned["optics"]
    col = lambda k: o[:, k][None, :]  # noqa: E731
    out, res = planned["model"].solveBatched(
        col(0), col(1), np.float32([SKY]), np.float32([1.0]), col(3), emission=col(2),
        precision=precision, tolerance=1e-6)
    want = _jacobi(planned["graph"], o[:, 3].astype(np.float64), o[:, 2].astype(np.float64), 60)
    assert res["converged"]
    # the stop rule leaves at most tolerance / (1 - c)
    assert np.max(np.abs(out[0] - want) / want) < _tolerance(planned["graph"]) + 1e-6 / (1 - RHO - TAU)


def test_planned_incident_in_a_node(planned):
    """The node's net radiation of object facets is the sum over both sides of
    eps H - E with the longwave radiosity it returns."""
    S, graph = planned["S"], planned["graph"]
    F = S // 2
    rng = np.random.default_rng(1)
    p, keep = facetcu.energy_parameters(
        F, [facetcu.EnergySurface([0.1], [0.0], 0.3, 0.1, vegetation=False)], np.zeros(F, np.uint32),
        coupling_iterations=1, solver_tolerance=1e-6)
    T0 = rng.uniform(285, 305, F).astype(np.float32).repeat(2)
    meteo = dict(air_temperature=20.0, vapor_pressure=12.0, pressure=1000.0, wind_speed=2.0,
                 shortwave=0.0, longwave=SKY)
    out, _ = planned["model"].facetebNode(p, meteo, np.float32([0, 1, 0]), np.zeros(S, np.float32),
                                          None, T0, fields=("longwave_radiosity", "net_radiation"))
    eps = 1.0 - np.float64(np.float32(0.3)) - np.float64(np.float32(0.1))
    H = _incident(graph, out["longwave_radiosity"].astype(np.float64))
    # the emitted part from the final temperature the node returns
    E = eps * 5.670374419e-8 * out["temperature"].astype(np.float64) ** 4
    want = (eps * H - E).reshape(-1, 2).sum(1).repeat(2)
    # H is rounded once to float and the two products and sums are floats
    scale = 2 * (eps * H.max() + E.max())
    assert np.max(np.abs(out["net_radiation"] - want)) < 12 * 2.0 ** -24 * scale + 1e-6 * scale


@pytest.mark.parametrize("bands", [5, 8, 11, 16])  # panels of 8 and 16 columns
@pytest.mark.parametrize("S", [2, 6, 1030])
def test_few_columns(S, bands):
    """Rows around 64 and 128 edges (one round of 16 and 8 columns), empty rows
    before, between and after others, an odd number of facets."""
    require_gpu()
    rng = np.random.default_rng(S + bands)
    edge = np.array([0, 1, 63, 64, 65, 0, 0, 127, 128, 129, 255, 256, 257, 3, 0, 500])
    graph = _graph(S, np.resize(edge, S), rng, counts=[255, 256, 257, 1000])
    m = _model(S, graph)
    scale = np.linspace(0.5, 2.0, bands, dtype=np.float32)
    o = _optics(S, rng)
    rep = lambda v: np.repeat(v[None, :], bands, 0)  # noqa: E731
    out, res = m.solveBatched(rep(o[:, 0]), rep(o[:, 1]), np.full(bands, SKY, np.float32), scale,
                              o[:, 3][None, :], emission=rep(o[:, 2]), tolerance=1e-7)
    m.close()
    tol = _tolerance(graph) + 1e-7 / (1 - RHO - TAU)
    for b in range(bands):
        direct = (o[:, 3] * scale[b]).astype(np.float64)
        want = _jacobi(graph, direct, o[:, 2].astype(np.float64), 60)
        assert np.max(np.abs(out[b] - want) / want) < tol
