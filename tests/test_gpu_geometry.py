"""setGeometry's checks on the device: which error is raised, and that a
refused geometry leaves the old one and its graph as they were; builds of
changing size on one context, whose scratch blocks are lent again."""
import numpy as np
import pytest

from streamsim_gb300 import facetcu, scenes
from tests.gpu_helpers import model_for, require_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("facets", [1, 85, 86, 5000])  # around one block of vertices
def test_first_bad_vertex_decides(facets):
    require_gpu()
    rng = np.random.default_rng(facets)
    v = np.zeros((3 * facets, 6), np.float32)
    v[:, :3] = rng.uniform(-5, 5, (3 * facets, 3))
    v[:, 4] = 1.0
    m = facetcu.FacetrtCuda()
    m.initialize(64, 64, 64)
    m.setGeometry(v)
    last = 3 * facets - 1

    def refused(edits, match):
        w = v.copy()
        for i, k, x in edits:
            w[i, k] = x
        with pytest.raises(ValueError, match=match):
            m.setGeometry(w)

    for x in (np.nan, np.inf, -np.inf):
        refused([(last, 1, x)], "non-finite position")
    refused([(last, 4, 0.98)], "normalized")
    refused([(0, 3, np.nan)], "normalized")
    refused([(last, 5, np.inf)], "normalized")
    refused([(0, 4, 2.0), (last, 0, np.nan)], "normalized")  # the earlier vertex
    refused([(0, 0, np.nan), (last, 4, 2.0)], "non-finite position")
    refused([(last, 4, 2.0), (last, 0, np.nan)], "non-finite position")  # the same vertex
    ok = v.copy()
    ok[last, 4] = 1.009
    m.setGeometry(ok)
    m.close()


def test_refused_geometry_changes_nothing():
    require_gpu()
    sc = scenes.config1(seed=3, leaves=60, grid=4)
    m = model_for(sc.vertices, 128, 64)
    m.buildVisibilityGraph(scenes.hemisphere_directions())
    before = m.graph()
    bad = sc.vertices[:30].copy()
    bad[7, 2] = np.nan
    with pytest.raises(ValueError):
        m.facet_count, keep = len(bad) // 3, m.facet_count
        try:
            m.setGeometry(bad)
        finally:
            m.facet_count = keep
    for a, b in zip(before, m.graph()):
        assert np.array_equal(a, b)
    m.buildVisibilityGraph(scenes.hemisphere_directions())
    for a, b in zip(before, m.graph()):
        assert np.array_equal(a, b)
    m.close()


def test_builds_of_changing_size_on_one_context():
    require_gpu()
    one = facetcu.FacetrtCuda()
    one.initialize(128, 128, 256)
    uv, dirs = scenes.hemisphere_samples(48, 4, seed=3)
    sun = scenes.sun_direction(30, 135)
    for leaves in (40, 2500, 3, 900, 40):
        sc = scenes.config1(seed=leaves, leaves=leaves, grid=5)
        fresh = model_for(sc.vertices, 128, 256)
        got = []
        for m in (one, fresh):
            m.setGeometry(sc.vertices)
            m.buildVisibilityGraph(scenes.hemisphere_directions())
            raster = m.graph() + (m.computeSunlitFraction(sun),)
            m.buildHemisphereGraph(uv, dirs, 48, 20, 4)
            got.append(raster + m.graph() + (m.hemisphereSunlit(sun, uv, 48, 4),))
        fresh.close()
        for a, b in zip(*got):
            assert np.array_equal(a, b)
    one.close()
