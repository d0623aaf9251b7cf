"""Chains of 9 to 64 fragments: up to 16 and 32 are ordered by networks in
registers, those with equal depths among more than 16 and longer ones as std::sort
orders them.  Against the CPU oracle; whole numbers, equal."""
import numpy as np
import pytest

from streamsim_gb300 import scenes
from tests.gpu_helpers import graphs_equal, model_for, oracle_cfg, require_gpu

pytestmark = pytest.mark.gpu

UP = np.array([[0.0, 1.0, 0.0]], np.float32)
FRAME = (np.float32([-1.0, -1.0, -1.0]), np.float32([1.0, 1.0, 1.0]))


def _check(oracle, v, raster, dirs, periodic=(0, 1.0, 1.0), bounds=FRAME):
    m = model_for(v, raster, 1024, bounds, periodic)
    cfg = oracle_cfg(v, raster, 1024, bounds, periodic)
    for _ in range(2):  # the second build starts from the first one's pool
        m.buildVisibilityGraph(dirs)
        g = oracle.build_graph(v, cfg, dirs)
        assert graphs_equal(m.graph(), g) is None
    m.close()
    return g


@pytest.mark.parametrize("depth", [9, 10, 15, 16, 17, 24, 31, 32, 33, 48, 64])
@pytest.mark.parametrize("ties", ["none", "last two", "threes", "all"])
def test_sheets(oracle, depth, ties):
    require_gpu()
    rng = np.random.default_rng(depth)
    v = np.zeros((depth, 3, 6), np.float32)
    v[:, :, [0, 2]] = np.float32([[-3, -3], [3.5, -3], [-3, 3.5]])
    level = rng.permutation(depth)
    level = {"none": level, "last two": np.maximum(level, 1), "threes": level // 3,
             "all": 0 * level}[ties]
    v[:, :, 1] = (level[:, None] - depth / 2) / depth
    v[:, :, 4] = rng.choice([-1.0, 1.0], depth)[:, None]
    g = _check(oracle, v.reshape(-1, 6), 33, UP)
    assert g.max_depth == depth


@pytest.mark.parametrize("facets,size", [(600, 0.5), (1500, 0.35)])
@pytest.mark.parametrize("neighbours", [0, 4])
def test_mixed_lengths(oracle, facets, size, neighbours):
    """All lengths side by side, a fifth of the facets twice (equal depths)."""
    require_gpu()
    rng = np.random.default_rng(facets)
    v = np.zeros((facets, 3, 6), np.float32)
    v[:, :, :3] = rng.uniform(-0.8, 0.8, (facets, 1, 3)) + rng.uniform(-size, size, (facets, 3, 3))
    v[:, :, 4] = rng.choice([-1.0, 1.0], facets)[:, None]
    v[-facets // 5:] = v[:len(v[-facets // 5:])]
    g = _check(oracle, v.reshape(-1, 6), 72, scenes.hemisphere_directions()[::7],
               (neighbours, 1.5, 1.5), (FRAME[0] * 1.5, FRAME[1] * 1.5))
    assert g.max_depth > 32
