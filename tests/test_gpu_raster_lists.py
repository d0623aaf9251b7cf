"""Raster visibility at the edges of its paths: chain lengths around what is
ordered in registers (2, 4, 8), in a thread's memory (64) and beyond, and
triangles around the boxes that a thread, a warp and a block take, against the
CPU oracle.  All results are whole numbers and equal."""
import numpy as np
import pytest

from streamsim_gb300 import scenes
from tests.gpu_helpers import graphs_equal, model_for, oracle_cfg, require_gpu

pytestmark = pytest.mark.gpu

UP = np.array([[0.0, 1.0, 0.0]], np.float32)
FRAME = (np.float32([-1.0, -1.0, -1.0]), np.float32([1.0, 1.0, 1.0]))


def _triangles(rng, n, size, heights, normals):
    """n random triangles of about the given size in the frame's square."""
    v = np.zeros((n, 3, 6), np.float32)
    centre = rng.uniform(-0.7, 0.7, (n, 1, 2))
    v[:, :, [0, 2]] = centre + rng.uniform(-size, size, (n, 3, 2))
    v[:, :, 1] = heights[:, None]
    v[:, :, 4] = normals[:, None]
    return v.reshape(-1, 6)


def _check(oracle, v, raster, layers, dirs, sun):
    m = model_for(v, raster, layers, FRAME)
    cfg = oracle_cfg(v, raster, layers, FRAME)
    m.buildVisibilityGraph(dirs)
    g = oracle.build_graph(v, cfg, dirs)
    assert graphs_equal(m.graph(), g) is None
    assert np.array_equal(m.computeSunlitFraction(sun), oracle.sunlit(v, cfg, sun)[0])
    m.close()
    return g


@pytest.mark.parametrize("depth", [1, 2, 3, 4, 5, 7, 8, 9, 16, 17, 63, 64, 65, 300])
@pytest.mark.parametrize("ties", [False, True])
def test_chain_lengths(oracle, depth, ties):
    """`depth` sheets over the whole frame, facing up or down, in shuffled order;
    with ties, groups of sheets share a height and the append order decides."""
    require_gpu()
    rng = np.random.default_rng(depth)
    v = np.zeros((depth, 3, 6), np.float32)
    v[:, :, [0, 2]] = np.float32([[-3, -3], [3.5, -3], [-3, 3.5]])
    level = rng.permutation(depth)
    v[:, :, 1] = ((level // 3 if ties else level)[:, None] - depth / 2) / depth
    v[:, :, 4] = rng.choice([-1.0, 1.0], depth)[:, None]
    g = _check(oracle, v.reshape(-1, 6), 33, 512, UP, UP[0])
    assert g.max_depth == depth


# 64 pixels per unit at raster 128: boxes of 1-9, around 16, some hundred and
# around and above 1,024 pixels, mixed in every warp
@pytest.mark.parametrize("size", [0.01, 0.03, 0.05, 0.15, 0.25, 0.8, None])
def test_triangle_sizes(oracle, size):
    require_gpu()
    rng = np.random.default_rng(7)
    n = 301  # a remainder in the last warp
    s = rng.choice([0.01, 0.04, 0.2, 0.7], (n, 1, 1)) if size is None else size
    v = _triangles(rng, n, s, rng.uniform(-0.9, 0.9, n), rng.choice([-1.0, 1.0], n))
    dirs = scenes.hemisphere_directions()[::9]
    _check(oracle, v, 128, 512, dirs, scenes.sun_direction(30, 135))


@pytest.mark.parametrize("raster,sheets", [(32, 3), (1024, 3), (1024, 6)])
def test_pair_sort_tiles(oracle, raster, sheets):
    """2,048 pairs (one tile of the sort), 2 M, and 5.2 M: more tiles than a
    digit's scan takes at once.  No facet lies below or above all others, so that
    sides have mirrored entries, forward entries, both or none."""
    require_gpu()
    rng = np.random.default_rng(sheets)
    v = np.zeros((sheets, 3, 6), np.float32)
    v[:, :, [0, 2]] = np.float32([[-20, -20], [30, -20], [-20, 30]])  # the whole frame
    v[:, :, 1] = (rng.permutation(sheets)[:, None] - sheets / 2) / sheets
    v[:, :, 4] = rng.choice([-1.0, 1.0], sheets)[:, None]
    g = _check(oracle, v.reshape(-1, 6), raster, 64, UP, UP[0])
    assert int(g.counts.astype(np.int64).sum()) == 2 * raster * raster * (sheets - 1)
