"""setGeometry's checks where the host makes them (up to 1,200 facets) and where
the device does, around the limit and around whole blocks of vertices: the same
errors, and bounds that give the same raster."""
import numpy as np
import pytest

from oracle.pyoracle import raster_config
from streamsim_gb300 import scenes
from tests.gpu_helpers import graphs_equal, model_for, require_gpu
from tests.test_gpu_geometry import test_first_bad_vertex_decides as first_bad_vertex

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("facets", [1199, 1200, 1201, 1365, 1366])
def test_first_bad_vertex(facets):
    first_bad_vertex(facets)


@pytest.mark.parametrize("facets", [1, 1200, 1201, 2048])
def test_bounds(oracle, facets):
    """One far vertex decides each side of the frame."""
    require_gpu()
    rng = np.random.default_rng(facets)
    v = np.zeros((facets, 3, 6), np.float32)
    v[:, :, :3] = rng.uniform(-2, 2, (facets, 1, 3)) + rng.uniform(-0.4, 0.4, (facets, 3, 3))
    v[:, :, 4] = 1.0
    v = v.reshape(-1, 6)
    v[-1, :3] = [5.5, 3.25, -4.75]
    v[len(v) // 2, :3] = [-3.5, -2.5, 6.0]
    m = model_for(v, 48, 512)
    dirs = scenes.hemisphere_directions()[::8]
    m.buildVisibilityGraph(dirs)
    p = v[:, :3]
    cfg = raster_config(48, 512, p.min(0), p.max(0), 0, 1.0, 1.0)
    assert graphs_equal(m.graph(), oracle.build_graph(v, cfg, dirs)) is None
    m.close()
