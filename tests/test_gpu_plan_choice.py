"""Whether a solve runs through the graph's column plan is decided by the call's
own arguments: the plan adds in another order, and a call's bits must not depend
on what was solved before it."""
import numpy as np
import pytest

from streamsim_gb300 import facetcu
from tests.gpu_helpers import require_gpu

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
