"""Whether a solve runs through the graph's column plan is decided by the call's
own arguments: the plan adds in another order, and a call's bits must not depend
on what was solved before it."""
import numpy as np
import pytest

from streamsim_gb300 import facetcu
from tests.gpu_helpers import require_gpu
from tests.test_gpu_one_column import _graph, _jacobi, _model, _optics, _tolerance

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def planned_graph():
    """A graph large enough for the plan (10 M edges) and its optics."""
    require_gpu()
    S, degree = 40960, 272
    rng = np.random.default_rng(3)
    F = S // 2
    v = np.zeros((3 * F, 6), np.float32)
    v[:, :3] = np.repeat(rng.uniform(-20, 20, (F, 3)), 3, 0) + np.tile(
        [[0, 0, 0], [0.1, 0, 0], [0, 0, -0.1]], (F, 1))
    v[:, 4] = 1.0
    nb = rng.integers(0, S, S * degree).astype(np.uint32)
    cnt = rng.integers(1, 4, S * degree).astype(np.uint32)
    sky = rng.integers(0, 50, S).astype(np.uint32)
    den = cnt.reshape(S, degree).sum(1).astype(np.uint32) + sky
    o = np.zeros((S, 4), np.float32)
    o[:, 0], o[:, 1] = 0.35, 0.15
    o[:, 2] = rng.uniform(0, 5, S)
    o[:, 3] = rng.uniform(0, 800, S)
    return v, ((np.arange(S + 1) * degree).astype(np.uint32), nb, cnt, den, sky), o


def test_short_solves_before_and_after_the_plan(planned_graph):
    v, graph, o = planned_graph
    m = facetcu.FacetrtCuda()
    m.initialize(64, 64, 64)
    m.setGeometry(v)
    m.setGraph(*graph)

    def short():
        return [m.solve(o, 100.0, 4, 0.75)["radiosity"],
                m.solveAccelerated(o, 100.0, maximum_iterations=4, batch_iterations=2, tolerance=0.0)[
                    "radiosity"]]

    before = short()
    m.solve(o, 100.0, 128)
    after = short()
    m.close()
    for a, b in zip(before, after):
        assert np.array_equal(a, b)


def test_few_sweeps_use_the_csr(planned_graph):
    """12 sweeps of 11 M edges don't pay for a plan (0.5 ms against some 9 us
    saved a sweep): they give the bits of three calls of 4 sweeps, each from the
    one before, which are too short for one by any rule.  128 sweeps do."""
    v, graph, o = planned_graph
    m = facetcu.FacetrtCuda()
    m.initialize(64, 64, 64)
    m.setGeometry(v)
    m.setGraph(*graph)

    def chained(calls):
        b = np.zeros(len(o), np.float32)
        for _ in range(calls):
            b = m.solveAccelerated(o, 100.0, initial=b, maximum_iterations=4, batch_iterations=4,
                                   tolerance=0.0)["radiosity"]
        return b

    assert np.array_equal(m.solve(o, 100.0, 12)["radiosity"], chained(3))
    assert not np.array_equal(m.solve(o, 100.0, 128)["radiosity"], chained(32))
    m.close()


# sides: one tile less 2, exactly one tile, a second tile of 2 sides, and a
# ragged last window; row lengths with empty rows and one far above the rest
@pytest.mark.parametrize("S", [49150, 49152, 49154, 102402])
def test_long_solves_use_the_plan(S):
    require_gpu()
    rng = np.random.default_rng(S)
    deg = rng.integers(150, 330, S)
    deg[rng.choice(S, S // 50)] = 0
    deg[rng.choice(S, 200)] = np.arange(1, 201) % 40
    deg[7] = 3000
    graph = _graph(S, deg, rng, counts=[255, 256, 257, 511, 512, 4097, 65535])
    o = _optics(S, rng)
    m = _model(S, graph)
    got = m.solve(o, 100.0, 80, 0.75)["radiosity"]
    m.close()
    want = _jacobi(graph, o[:, 3].astype(np.float64), o[:, 2].astype(np.float64), 80, 0.75)
    assert np.max(np.abs(got - want) / want) < _tolerance(graph)
