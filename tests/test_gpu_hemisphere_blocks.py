"""The ray caster's blocks of several facets where a facet has few rays: 2 to 64
facets a block, with a ragged last block, against the CPU oracle (whole numbers,
equal)."""
import pytest

from streamsim_gb300 import facetcu, scenes
from tests.gpu_helpers import graphs_equal, require_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaves,grid,rays", [
    (150, 8, 16), (350, 13, 33), (900, 22, 16), (1700, 8, 32), (1700, 8, 5), (900, 22, 65)])
def test_blocks_of_several_facets(oracle, leaves, grid, rays):
    require_gpu()
    sc = scenes.config1(seed=leaves + rays, leaves=leaves, grid=grid)
    uv, dirs = scenes.hemisphere_samples(rays, 3, seed=rays)
    m = facetcu.FacetrtCuda()
    m.initialize(64, 64, 64)
    m.setGeometry(sc.vertices)
    _, dropped = m.buildHemisphereGraph(uv, dirs, rays, rays, 3)
    g, dropped_o = oracle.hemisphere_graph(sc.vertices, uv, dirs, rays, 3, rays)
    assert graphs_equal(m.graph(), g) is None
    assert dropped == dropped_o
    m.close()
