"""The mean squared error is summed in doubles: squares that a float does not hold
leave a loss that it does."""
import numpy as np
import pytest

from streamsim_gb300 import facetcu
from tests.gpu_helpers import require_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,far", [(1, 1.0e19), (300, 3.0e19), (65536, 1.0e21)])
def test_squares_above_the_float_range(rows, far):
    require_gpu()
    m = facetcu.FacetrtCuda()
    m.initialize(16, 16, 8)
    m.mlpReset(1)
    m.mlpSetParameters(np.zeros(facetcu.MLP_PARAMETERS, np.float32))  # outputs are 0
    rng = np.random.default_rng(rows)
    t = rng.normal(size=(rows, 64)).astype(np.float32)
    t[rows // 2, 5], t[0, 63] = far, -0.25 * far
    loss, g = m.mlpLossAndGradient(np.zeros((rows, 12), np.float32), t)
    m.close()
    want = np.mean(t.astype(np.float64) ** 2)
    assert want < np.finfo(np.float32).max
    assert abs(loss - want) <= 2.0 ** -23 * want  # one rounding to float
    assert np.all(np.isfinite(g))
