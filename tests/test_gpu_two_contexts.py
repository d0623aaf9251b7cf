"""Two contexts on one GPU, each used by a thread of its own: what one of them
does must not show in the other's results.  Whole numbers and fixed orders of
addition, so the results are the same as alone, bit for bit."""
import threading

import numpy as np
import pytest

from streamsim_gb300 import scenes
from tests.gpu_helpers import model_for, require_gpu

pytestmark = pytest.mark.gpu


def _together(jobs, rounds):
    """Runs the jobs, a thread each, `rounds` times side by side; every result
    is compared with the job's result alone."""
    alone = [job() for job in jobs]
    gate = threading.Barrier(len(jobs))
    wrong = []

    def work(i):
        try:
            gate.wait()
            for k in range(rounds):
                got = jobs[i]()
                if not all(np.array_equal(a, b) for a, b in zip(got, alone[i])):
                    wrong.append((i, k))
        except Exception as e:  # noqa: BLE001 - shown by the assertion below
            wrong.append((i, repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def _soup(n, seed):
    rng = np.random.default_rng(seed)
    v = np.zeros((n, 3, 6), np.float32)
    v[:, :, :3] = rng.uniform(-8, 8, (n, 1, 3)) + rng.uniform(-1, 1, (n, 3, 3))
    v[:, :, 4] = rng.choice([-1.0, 1.0], n)[:, None]
    return v.reshape(-1, 6)


def test_raster_builds_of_two_sizes():
    """Different facets, tiles and frame sizes: with one frame for both contexts
    a kernel would take the other's facet count, width and tiles."""
    require_gpu()
    dirs = scenes.hemisphere_directions()[::4]
    sun = scenes.sun_direction(30, 135)
    models = [model_for(_soup(400, 1), 96, 512), model_for(_soup(3000, 2), 160, 512, None, (4, 20.0, 20.0))]

    def job(m):
        def run():
            m.buildVisibilityGraph(dirs)
            return (*m.graph(), m.computeSunlitFraction(sun))
        return run

    _together([job(m) for m in models], 40)
    for m in models:
        m.close()
