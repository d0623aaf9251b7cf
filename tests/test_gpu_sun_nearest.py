"""The sun pass keeps a pixel's nearest fragment and their number instead of a
list.  Against the CPU oracle, equal: depths from 1 to 900, equal depths (append
order decides), boxes for a thread, 8 lanes and the grid, and the limit per pixel.
The same buffers hold a graph build's lists in between."""
import numpy as np
import pytest

from streamsim_gb300 import scenes
from tests.gpu_helpers import graphs_equal, model_for, oracle_cfg, require_gpu

pytestmark = pytest.mark.gpu

UP = np.array([[0.0, 1.0, 0.0]], np.float32)
FRAME = (np.float32([-1.0, -1.0, -1.0]), np.float32([1.0, 1.0, 1.0]))


def _sheets(depth, ties):
    rng = np.random.default_rng(depth)
    v = np.zeros((depth, 3, 6), np.float32)
    v[:, :, [0, 2]] = np.float32([[-3, -3], [3.5, -3], [-3, 3.5]])
    level = rng.permutation(depth)
    level = {"none": level, "threes": level // 3, "all": 0 * level}[ties]
    v[:, :, 1] = (level[:, None] - depth / 2) / depth
    v[:, :, 4] = rng.choice([-1.0, 1.0], depth)[:, None]
    return v.reshape(-1, 6)


@pytest.mark.parametrize("depth", [1, 2, 33, 257, 900])
@pytest.mark.parametrize("ties", ["none", "threes", "all"])
@pytest.mark.parametrize("raster", [5, 33])
def test_sheets(oracle, depth, ties, raster):
    require_gpu()
    v = _sheets(depth, ties)
    m = model_for(v, raster, 1024, FRAME)
    cfg = oracle_cfg(v, raster, 1024, FRAME)
    for sun in (UP[0], scenes.sun_direction(20.0, 65.0)):
        want = oracle.sunlit(v, cfg, sun)[0]
        assert np.array_equal(m.computeSunlitFraction(sun), want)
        m.buildVisibilityGraph(UP)
        assert graphs_equal(m.graph(), oracle.build_graph(v, cfg, UP)) is None
        assert np.array_equal(m.computeSunlitFraction(sun), want)
    m.close()


@pytest.mark.parametrize("facets,size", [(700, 0.02), (700, 0.2), (300, 0.9)])
@pytest.mark.parametrize("neighbours", [0, 4])
def test_mixed_boxes(oracle, facets, size, neighbours):
    """Every fifth facet twice: equal depths from two sides of a list."""
    require_gpu()
    rng = np.random.default_rng(facets)
    v = np.zeros((facets, 3, 6), np.float32)
    v[:, :, :3] = rng.uniform(-0.8, 0.8, (facets, 1, 3)) + rng.uniform(-size, size, (facets, 3, 3))
    v[:, :, 4] = rng.choice([-1.0, 1.0], facets)[:, None]
    v[-(facets // 5):] = v[:facets // 5]
    v = v.reshape(-1, 6)
    frame, periodic = (FRAME[0] * 1.5, FRAME[1] * 1.5), (neighbours, 1.5, 1.5)
    m = model_for(v, 97, 1024, frame, periodic)
    cfg = oracle_cfg(v, 97, 1024, frame, periodic)
    for sun in (UP[0], scenes.sun_direction(55.0, 200.0)):
        assert np.array_equal(m.computeSunlitFraction(sun), oracle.sunlit(v, cfg, sun)[0])
    m.close()


def test_limit_per_pixel():
    """As many fragments as the limit pass, one more is refused."""
    require_gpu()
    m = model_for(_sheets(40, "none"), 16, 40, FRAME)
    m.computeSunlitFraction(UP[0])
    m.setGeometry(_sheets(41, "none"))
    m.setRasterBounds(*FRAME)
    with pytest.raises(RuntimeError, match="Direct-light A-buffer overflow"):
        m.computeSunlitFraction(UP[0])
    m.close()
