"""One sweep through the column plan whose sums a float holds exactly: every word of
the plan has to be there, in its row, with its count.  Radiosities are small whole
numbers, row sums stay below 2^24 and denominators are a power of two, so the
results equal the integers' quotients bit for bit.  (A tolerance from the longest
row lets a lost low byte of a large count pass.)"""
import numpy as np
import pytest

from streamsim_gb300 import facetcu
from tests.gpu_helpers import require_gpu
from tests.test_gpu_one_column import _model

pytestmark = pytest.mark.gpu

DENOMINATOR = 1 << 20


# one tile less 2 sides, exactly one tile, a second tile of 2, three tiles with a
# ragged last window; counts of one word, and of two (more than 8 significant bits)
@pytest.mark.parametrize("S", [49150, 49152, 49154, 102402])
@pytest.mark.parametrize("counts", [[1, 2, 255, 256, 65280], [257, 511, 513, 4097, 65535], None])
def test_every_word_counts(S, counts):
    require_gpu()
    rng = np.random.default_rng(S)
    deg = rng.integers(170, 330, S)
    deg[rng.choice(S, S // 50)] = 0
    deg[rng.choice(S, 200)] = np.arange(1, 201) % 40
    deg[7] = 3000
    rows = np.zeros(S + 1, np.int64)
    rows[1:] = np.cumsum(deg)
    n = int(rows[-1])
    assert n >= 10 << 20  # large enough for the plan
    nb = rng.integers(0, S, n).astype(np.uint32)
    cnt = rng.integers(1, 4, n).astype(np.int64)
    if counts is None:
        cnt = rng.integers(1, 1 << 11, n)
    else:  # in a fiftieth of the rows' places, a few a row
        at = rng.choice(n, n // 100, replace=False)
        cnt[at] = np.resize(counts, len(at))
    B = rng.integers(0, 4, S).astype(np.int64)
    sums = np.add.reduceat(np.append(cnt * B[nb], 0), np.minimum(rows[:-1], n))
    sums[deg == 0] = 0
    assert sums.max() < 1 << 24
    one = np.ones((1, S), np.float32)
    m = _model(S, (rows.astype(np.uint32), nb, cnt.astype(np.uint32),
                   np.full(S, DENOMINATOR, np.uint32), np.zeros(S, np.uint32)))
    for precision in (facetcu.PRECISION_FP32, facetcu.PRECISION_MIXED):
        got, res = m.solveBatched(one, 0.0 * one, np.zeros(1, np.float32), np.zeros(1, np.float32),
                                  precision=precision, tolerance=1e-6, maximum_iterations=1,
                                  initial=B.astype(np.float32)[None], raise_on_nonconvergence=False)
        assert np.array_equal(got[0], (sums / DENOMINATOR).astype(np.float32))
    m.close()
