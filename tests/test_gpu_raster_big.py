"""Triangles whose boxes whole blocks or warps take (above 1,024 pixels), from one in
the frame to more than the grid has warps, against the CPU oracle: one alone, as
many as blocks, a few to a block, and a warp each.  Whole numbers, equal."""
import numpy as np
import pytest

from streamsim_gb300 import scenes
from tests.gpu_helpers import graphs_equal, model_for, oracle_cfg, require_gpu

pytestmark = pytest.mark.gpu

FRAME = (np.float32([-1.0, -1.0, -1.0]), np.float32([1.0, 1.0, 1.0]))


# the grid has 8 blocks of 8 warps an SM: 1,216 and 9,728 on 152 SMs
@pytest.mark.parametrize("facets,directions", [(1, 1), (3, 1), (40, 30), (700, 2), (330, 40)])
def test_large_boxes(oracle, facets, directions):
    require_gpu()
    rng = np.random.default_rng(facets)
    v = np.zeros((facets, 3, 6), np.float32)
    v[:, :, [0, 2]] = rng.uniform(-0.3, 0.3, (facets, 1, 2)) + rng.uniform(0.2, 0.6, (facets, 3, 1)) * (
        np.float32([[-1, -1], [1, -0.8], [-0.2, 1]]) + rng.uniform(-0.3, 0.3, (facets, 3, 2)))
    v[:, :, 1] = (rng.permutation(facets) / facets - 0.5)[:, None] + rng.uniform(-0.02, 0.02, (facets, 3))
    v[:, :, 4] = rng.choice([-1.0, 1.0], facets)[:, None]
    v = v.reshape(-1, 6)
    m = model_for(v, 192, 1024, FRAME)
    cfg = oracle_cfg(v, 192, 1024, FRAME)
    dirs = scenes.hemisphere_directions()[:directions]
    m.buildVisibilityGraph(dirs)
    assert graphs_equal(m.graph(), oracle.build_graph(v, cfg, dirs)) is None
    sun = scenes.sun_direction(20, 30)
    assert np.array_equal(m.computeSunlitFraction(sun), oracle.sunlit(v, cfg, sun)[0])
    m.close()
