"""How a panel begins, for widths of every path: from zero (the first sweep's
result becomes the residual) and from given values, with and without emission,
and arrays that are not 16-byte aligned, against the FP64 solve of the same
library."""
import numpy as np
import pytest

from streamsim_gb300 import facetcu
from tests.gpu_helpers import require_gpu
from tests.test_gpu_one_column import _graph, _model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bands", [1, 3, 8, 31, 32, 33, 64, 67, 128, 131])
@pytest.mark.parametrize("precision", [facetcu.PRECISION_FP32, facetcu.PRECISION_MIXED])
def test_zero_and_given_start(bands, precision):
    require_gpu()
    rng = np.random.default_rng(bands)
    S = 1022  # whole tiles of 32 sides and a part of one
    m = _model(S, _graph(S, rng.integers(0, 40, S), rng))
    rho = rng.uniform(0.05, 0.4, (bands, S)).astype(np.float32)
    tau = rng.uniform(0.0, 0.2, (bands, S)).astype(np.float32)
    emis = rng.uniform(0.0, 3.0, (bands, S)).astype(np.float32)
    sky, beam = rng.uniform(10, 90, bands), rng.uniform(100, 900, bands)
    geo = rng.uniform(0, 1, (1, S)).astype(np.float32)
    for e in (None, emis):
        want, _ = m.solveBatched(rho, tau, sky, beam, geo, e, facetcu.PRECISION_FP64, 1e-9)
        got, _ = m.solveBatched(rho, tau, sky, beam, geo, e, precision, 1e-6)
        again, _ = m.solveBatched(rho, tau, sky, beam, geo, e, precision, 1e-6, initial=0.5 * want)
        # the last sweep changes no side by more than 1e-6 of its column's largest
        # value M, and its own rounding is at most (deg + 8) 2^-24 M; the error is
        # the sum of what further sweeps would add, 1 / (1 - c), c = rho + tau <= 0.6
        top = want.max(axis=1, keepdims=True)
        for x in (got, again):
            assert np.max(np.abs(x - want) / top) <= (1e-6 + 48 * 2.0 ** -24) / 0.4
    m.close()


def test_bad_values_at_any_place():
    require_gpu()
    rng = np.random.default_rng(1)
    S, bands = 30, 5
    m = _model(S, _graph(S, rng.integers(0, 9, S), rng))
    good = np.full((bands, S), 0.25, np.float32)
    geo, k = np.ones((1, S), np.float32), np.full(bands, 10.0)
    for i in (0, 1, 2, 3, S * bands - 3, S * bands - 2, S * bands - 1):
        for name, value in (("rho", np.nan), ("tau", -0.5), ("rho", 0.9), ("emis", np.inf)):
            a = {"rho": good.copy(), "tau": good.copy(), "emis": good.copy()}
            a[name].reshape(-1)[i] = value
            with pytest.raises(ValueError):
                m.solveBatched(a["rho"], a["tau"], k, k, geo, a["emis"], facetcu.PRECISION_FP32)
    m.close()
