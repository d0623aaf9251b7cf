"""Two contexts on one GPU, each used by a thread of its own: what one of them
does must not show in the other's results.  Whole numbers and fixed orders of
addition, so the results are the same as alone, bit for bit."""
import threading

import numpy as np
import pytest

from streamsim_gb300 import facetcu, scenes
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


def test_hemisphere_builds_of_two_sizes():
    """The caster's block takes 32 KB of shared memory for 40,000 facets and 256
    rays and a few hundred bytes for 300 facets and 32."""
    require_gpu()
    jobs, models = [], []
    for n, rays, seed in ((40000, 256, 3), (300, 32, 4)):
        v = _soup(n, seed)
        v[:, :3] *= np.float32(n / 300) ** np.float32(1 / 3)  # as dense
        m = facetcu.FacetrtCuda()
        m.initialize(64, 64, 64)
        m.setGeometry(v)
        models.append(m)
        uv, d = scenes.hemisphere_samples(rays, 2, seed=5)

        def run(m=m, uv=uv, d=d, rays=rays):
            m.buildHemisphereGraph(uv, d, rays, 32, 2)
            return m.graph()
        jobs.append(run)
    _together(jobs, 30)
    for m in models:
        m.close()


def test_small_solves_of_two_sizes():
    """Graphs that one cluster launch solves; the largest's edges want ten times the
    smallest's shared memory.  (Several threads each: the calls meet more often.)"""
    require_gpu()
    jobs, models = [], []
    for S, degree, seed in ((3200, 28, 1), (64, 4, 2), (64, 4, 3), (64, 4, 4), (3200, 28, 5), (64, 4, 6)):
        rng = np.random.default_rng(seed)
        v = _soup(S // 2, seed)
        rows = (np.arange(S + 1) * degree).astype(np.uint32)
        nb = rng.integers(0, S, S * degree).astype(np.uint32)
        cnt = rng.integers(1, 4, S * degree).astype(np.uint32)
        sky = rng.integers(0, 50, S).astype(np.uint32)
        den = cnt.reshape(S, degree).sum(1).astype(np.uint32) + sky
        m = facetcu.FacetrtCuda()
        m.initialize(64, 64, 64)
        m.setGeometry(v)
        m.setGraph(rows, nb, cnt, den, sky)
        models.append(m)
        o = np.zeros((S, 4), np.float32)
        o[:, 0], o[:, 1] = 0.35, 0.15
        o[:, 3] = rng.uniform(0, 800, S)
        jobs.append(lambda m=m, o=o: (m.solve(o, 100.0, 16, 1.0)["radiosity"],))
    _together(jobs, 400)
    for m in models:
        m.close()
