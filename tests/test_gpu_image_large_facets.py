"""Sensor images where the facets' boxes go to different kernels: a lane up to 16
pixels, a warp up to 1,024, the large-box kernel above, alone (its blocks share a
facet), a few, and more than it has blocks; from one facet to 32 a warp.  The side
images equal the oracle's."""
import numpy as np
import pytest

from oracle import image_oracle as io
from streamsim_gb300 import facetcu
from tests.gpu_helpers import model_for, require_gpu

pytestmark = pytest.mark.gpu

SIZE, SCENE = 72, 12.0  # 6 pixels a metre


def _facets(rng, n, edge):
    """Random triangles of about the given edge (m), many of them tilted."""
    t = rng.uniform(-5, 5, (n, 1, 3)) * [1.0, 0.2, 1.0] + [0.0, 2.0, 0.0]
    t = t + rng.uniform(-edge, edge, (n, 3, 3)) * [1.0, 0.3, 1.0]
    nrm = np.cross(t[:, 1] - t[:, 0], t[:, 2] - t[:, 0])
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    return np.concatenate([t, np.repeat(nrm[:, None], 3, 1)], 2)


@pytest.mark.parametrize("small,medium,large", [
    (0, 0, 1), (0, 0, 3), (0, 300, 0), (0, 0, 1300), (5000, 40, 8), (30000, 60, 40), (78000, 33, 5)])
def test_large_facets(small, medium, large):
    require_gpu()
    rng = np.random.default_rng(small + medium + large)
    v = np.concatenate([_facets(rng, small, 0.1), _facets(rng, medium, 1.2), _facets(rng, large, 6.0)])
    # neighbours in a warp: large ones side by side and scattered
    v = v[rng.permutation(len(v))] if medium else v
    v = np.ascontiguousarray(v.reshape(-1, 6), np.float32)
    m = model_for(v, 64, 64)
    for perspective, zenith in ((False, 0.0), (False, 40.0), (True, 15.0)):
        where = (6.0, 6.0, 14.0) if perspective else (np.nan,) * 3
        s = facetcu.sensor(SIZE, SIZE, perspective, zenith, 30.0, 50.0, SCENE, SCENE, where)
        _, idx, _ = m.renderSensorImage(s, [], [])
        cam = io.Camera(width=SIZE, height=SIZE, perspective=perspective, vza=zenith, vaa=30.0,
                        fov=50.0, scene_x=SCENE, scene_y=SCENE, position=where)
        want = io.side_image(cam, v.reshape(-1, 3, 6)[:, :, :3])[0]
        assert np.array_equal(idx, want), f"{np.sum(idx != want)} pixels differ"
    m.close()
