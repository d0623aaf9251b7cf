"""All sweeps of a small graph in one launch (a cluster of 16 blocks that own
the sides in groups of 16) at its edges: fewer sides than blocks, part groups,
sweep counts around the deltas that leave together, shares of edges that do not
fit, and sizes and sweep counts on both sides of its limits, against a float64 Jacobi iteration.  The
largest change that is reported is compared as well.

Tolerance: as in test_gpu_one_column (derived there); the change of the last
sweep is a difference of two such values, so twice that, of the largest value."""
import numpy as np
import pytest

from tests.gpu_helpers import require_gpu
from tests.test_gpu_one_column import SKY, _graph, _jacobi, _model, _optics, _tolerance

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,sweeps", [(2, 11), (2, 12), (30, 13), (256, 63), (258, 64), (510, 65),
                                      (4096, 64), (4094, 130), (4098, 64), (20000, 12)])
def test_sizes_and_sweep_counts(S, sweeps):
    require_gpu()
    rng = np.random.default_rng(S)
    deg = rng.integers(0, 20, S)
    deg[rng.choice(S, S // 2, replace=False)] = 0
    _check(_graph(S, deg, rng, counts=[65535]), S, rng, sweeps)


@pytest.mark.parametrize("case", ["one_block_heavy", "limit", "above_limit", "count_above"])
def test_uneven_shares_and_limits(case):
    """`one_block_heavy`: nearly all edges are those of the first group."""
    require_gpu()
    rng = np.random.default_rng(3)
    S, counts = 4096, None
    deg = np.full(S, 24)
    if case == "one_block_heavy":
        deg = np.full(S, 1)
        deg[:16] = 5000
    elif case == "limit":
        deg[:100000 - deg.sum()] += 1
    elif case == "above_limit":
        deg[:100001 - deg.sum()] += 1
    else:
        counts = [65536]
    _check(_graph(S, deg, rng, counts=counts), S, rng, 13)


def _check(graph, S, rng, sweeps):
    m = _model(S, graph)
    o = _optics(S, rng)
    for relax in (1.0, 0.6):
        result = m.solve(o, SKY, sweeps, relax)
        got = result["radiosity"]
        want = _jacobi(graph, o[:, 3].astype(float), o[:, 2].astype(float), sweeps, relax)
        tol = _tolerance(graph)
        assert np.max(np.abs(got - want) / np.maximum(np.abs(want), 1e-30)) <= tol
        before = _jacobi(graph, o[:, 3].astype(float), o[:, 2].astype(float), sweeps - 1, relax)
        assert abs(result["maxDelta"] - np.max(np.abs(want - before))) <= (
            2 * tol * np.max(np.abs(want)))
    m.close()
