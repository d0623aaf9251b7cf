"""Incident radiation of the shortwave windows (two windows per lane, groups of
lanes over the edges) for window counts around its groups and rows.

The node returns sums over the windows, and the exchange is linear: with A the
counts, den the denominators and sky the sky counts of the graph,
    sum_w H_w = (sky sum_w L_w + A sum_w B_w) / den + dgeo sum_w dni_w
holds for the returned sums but for their roundings, W + 1 of them on either
side and a few in the direct term, of 2^-24 each (all terms are positive)."""
import numpy as np
import pytest

from streamsim_gb300 import facetcu
from tests.gpu_helpers import require_gpu
from tests.test_gpu_one_column import _graph, _model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W", [1, 2, 3, 8, 9, 16, 17, 20, 31, 32, 33, 63, 64, 65, 70])
def test_sum_over_windows(W):
    require_gpu()
    rng = np.random.default_rng(W)
    S = 1030
    deg = np.resize([0, 1, 2, 3, 4, 5, 11, 12, 13, 40, 41, 200], S)
    rows, nb, cnt, den, sky = _graph(S, deg, rng, counts=[1 << 20, 255])
    for s in (8, 9, 500):  # denominators that floats don't hold
        den[s] += (1 << 25) + 1 - sky[s]
        sky[s] = (1 << 25) + 1
    graph = (rows, nb, cnt, den, sky)
    m = _model(S, graph)
    F = S // 2
    surface = facetcu.EnergySurface([0.2], [0.1], 0.05, 0.02,
                                    energy_reflectance=np.full(2001, 0.3, np.float32),
                                    energy_transmittance=np.full(2001, 0.2, np.float32))
    p, keep = facetcu.energy_parameters(F, [surface], np.zeros(F, np.uint32), None, 0.0, [],
                                        coupling_iterations=1)
    windows = (facetcu.ShortwaveWindow * W)()
    dni, L = rng.uniform(0, 60, W).astype(np.float32), rng.uniform(0, 30, W).astype(np.float32)
    for w in range(W):
        windows[w].direct_normal, windows[w].diffuse = float(dni[w]), float(L[w])
        windows[w].energy_band = int(rng.integers(0, 2001))
    sun = np.float32([0.6, 0.8, 0.0])
    lit = rng.uniform(0, 1, S).astype(np.float32)
    out, _ = m.facetebNode(p, dict(air_temperature=20.0, vapor_pressure=10.0, pressure=1000.0,
                                   wind_speed=1.0, shortwave=500.0, longwave=300.0),
                           sun, lit, windows, np.full(S, 293.0, np.float32))
    m.close()
    import scipy.sparse as sp
    A = sp.csr_matrix((cnt.astype(float), nb.astype(np.int64), rows.astype(np.int64)), (S, S))
    B = out["shortwave_radiosity"].astype(float)
    dgeo = lit.astype(float) * np.where(np.arange(S) % 2 == 0, float(sun[1]), 0.0)
    mean = (sky * L.astype(float).sum() + A @ B) / np.maximum(den, 1)
    want = np.where(den > 0, mean, L.astype(float).sum()) + dgeo * dni.astype(float).sum()
    tol = (2 * (W + 1) + 6) * 2.0 ** -24
    assert np.max(np.abs(out["incident_shortwave"] - want) / want) <= tol
    assert np.all(B > 0)
