"""A graph without edges needs no edge array: setGraph reads as many edges as the
row offsets name, and every side sees only the sky."""
import ctypes as C

import numpy as np
import pytest

from streamsim_gb300 import facetcu
from tests.gpu_helpers import require_gpu

pytestmark = pytest.mark.gpu


def test_null_edges():
    require_gpu()
    S = 6
    v = np.zeros((3 * S // 2, 6), np.float32)
    v[:, :3] = np.random.default_rng(0).uniform(-1, 1, (3 * S // 2, 3))
    v[:, 4] = 1.0
    m = facetcu.FacetrtCuda()
    m.initialize(64, 64, 64)
    m.setGeometry(v)
    rows, den = np.zeros(S + 1, np.uint32), np.full(S, 4, np.uint32)
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    assert m.lib.facetcu_set_graph(m.h, S, p(rows), None, p(den), p(den)) == facetcu.OK
    o = np.zeros((S, 4), np.float32)
    o[:, 0] = 0.5
    got = m.solve(o, 8.0, 4)["radiosity"]
    m.close()
    assert np.array_equal(got, np.full(S, 4.0, np.float32))
