"""The work that is timed when the framework's speed is looked at.

Each case is one call, or the few calls that belong together, that a user of
the library makes: the two view-factor builds with the sun's pass, the
reference-semantics solve, the batched solve of one scene and of a batch of
scenes, the band loop behind `facetcu eFacetRT`, a FacetEB time node, a
gradient of the warm-start network and a sensor image.  The scenes are the
sizes of the repository's workloads (scenes.py): 4,096 facets (soil and
scattered leaves) and forests of up to 203,000 facets (60 trees of 3,000
leaves).

`listed`, `draw`, `prepare`, `run`, `work` and `exact` are explained at their
definitions.  Everything is made from the seed alone.  Solves run on
exchange graphs made here (`exchange_graph`), so that `exact` can solve the
same system in 64 bits without the library.
"""
import ctypes
import math

import numpy as np
import torch

from streamsim_gb300 import facetcu as fc
from streamsim_gb300 import scenes

LEAVES = 3000  # leaves of a crown, as in the forest workload
SUN = (30.0, 135.0)
SKY, BEAM = 100.0, 800.0


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


# ---- the cases ----------------------------------------------------------------
def listed():
    small = {"trees": 0, "grid": 32}      # 2,048 leaves over 2,048 soil triangles
    forest = {"trees": 60, "grid": 100}   # 180,000 leaves over 20,000 soil triangles
    return [
        # the eFacetRT default: 40 directions on a 1,024 x 1,024 raster, on the
        # smallest scene the repository names and on the forest
        {"name": "raster_graph_small", "kind": "raster", **small, "raster": 1024, "directions": 40},
        {"name": "raster_graph_forest", "kind": "raster", **forest, "raster": 1024,
         "directions": 40},
        # hemisphere view factors: 256 rays on the small scene, 512 on the forest
        {"name": "hemisphere_graph_small", "kind": "hemisphere", **small, "rays": 256,
         "top_k": 256, "sun_samples": 256},
        {"name": "hemisphere_graph_forest", "kind": "hemisphere", **forest, "rays": 512,
         "top_k": 256, "sun_samples": 256},
        # the drop-in solver, 64 sweeps of one band: launches count at 4,096
        # facets, the gather at 200,000
        {"name": "solve_small", "kind": "solve", **small, "rays": 24, "accelerated": False},
        {"name": "solve_forest", "kind": "solve", **forest, "rays": 512, "accelerated": False},
        # the headline: 64 bands of one sun, inputs and outputs on the device
        {"name": "batched_mixed_64", "kind": "batched", **forest, "rays": 512, "bands": 64,
         "suns": 1, "thermal": False, "precision": "mixed", "host": False},
        # six scenes of uneven size in one batch, 64 bands and one thermal band
        # (a 64-column and a 1-column panel)
        {"name": "scene_batch_mixed", "kind": "scene_batch", "scenes": 6, "lo": 4000, "hi": 60000,
         "rays": 256, "bands": 64},
        # the band loop of an eFacetRT project: 9 sensor bands, two of them
        # thermal, host arrays in and out, 64 sweeps each
        {"name": "band_loop", "kind": "band_loop", "trees": 20, "grid": 50, "rays": 256},
        # one FacetEB time node on the forest: 20 shortwave windows, the
        # longwave coupling rounds and 8 sensor bands
        {"name": "energy_node", "kind": "energy_node", **forest, "rays": 512, "top_k": 256},
        # loss and gradient of the warm-start network on its training batch
        {"name": "mlp_gradient", "kind": "mlp_gradient", "rows": 65536},
        # three bands of the forest seen by an oblique sensor
        {"name": "sensor_image", "kind": "image", **forest, "width": 1024, "height": 1024,
         "perspective": False, "zenith": 35.0, "bands": 3},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges: any kind, sizes spread over the
    logarithm of their range, odd ones among them."""
    kind = rng.choice(["raster", "hemisphere", "solve", "solve", "batched", "batched", "batched",
                       "scene_batch", "band_loop", "energy_node", "mlp_gradient", "image"])
    trees = _log(rng, 1, 50) if rng.random() < 0.8 else 0
    scene = {"trees": trees, "grid": _log(rng, 12, 99)}
    if kind == "raster":
        return {"kind": kind, **scene, "raster": rng.choice([256, 384, 500, 777, 1024]),
                "directions": rng.choice([17, 40])}
    if kind == "hemisphere":
        return {"kind": kind, **scene, "rays": rng.randint(48, 511), "top_k": rng.randint(40, 256),
                "sun_samples": rng.randint(16, 256)}
    if kind == "solve":
        return {"kind": kind, **scene, "rays": rng.randint(16, 511),
                "accelerated": rng.random() < 0.5}
    if kind == "batched":
        suns = rng.choice([1, 1, 2, 3])
        return {"kind": kind, **scene, "rays": rng.randint(64, 511),
                "bands": _log(rng, 1, 130 // suns), "suns": suns,
                "thermal": rng.random() < 0.3, "precision": rng.choice(["mixed", "fp32"]),
                "host": rng.random() < 0.5}
    if kind == "scene_batch":
        return {"kind": kind, "scenes": rng.randint(2, 6), "lo": _log(rng, 1000, 4000),
                "hi": _log(rng, 8000, 60000), "rays": rng.randint(64, 256),
                "bands": rng.randint(3, 96)}
    if kind == "band_loop":
        return {"kind": kind, **scene, "rays": rng.randint(32, 400)}
    if kind == "energy_node":
        return {"kind": kind, "trees": _log(rng, 1, 20), "grid": _log(rng, 12, 99),
                "rays": rng.randint(64, 400), "top_k": 256}
    if kind == "mlp_gradient":
        return {"kind": kind, "rows": _log(rng, 500, 65000)}
    return {"kind": kind, **scene, "width": rng.randint(200, 1024), "height": rng.randint(200, 1024),
            "perspective": rng.random() < 0.5, "zenith": rng.uniform(0.0, 60.0),
            "bands": rng.randint(1, 6)}


def work(case):
    """Bytes each input and output takes once, and the operations the path
    cannot do without (an edge's multiply-add per column and sweep; a ray's
    descent to one leaf; a triangle's projection per direction)."""
    kind = case["kind"]
    if kind == "mlp_gradient":
        n = case["rows"]
        weights = 128 * 12 + 128 * 128 + 64 * 128
        return {"bytes": 4.0 * n * (12 + 64) + 8.0 * 26432, "flops": 6.0 * n * weights}
    if kind == "scene_batch":
        facets = sum(_batch_facets(case))
        cols, sweeps = case["bands"] + 1, 16
        S = 2.0 * facets
        edges = S * 0.4 * case["rays"]
        return {"bytes": 4 * edges + S * cols * 12 + S * 4, "flops": 2 * edges * cols * sweeps}
    F = _facets(case)
    S = 2.0 * F
    if kind == "raster":
        return {"bytes": 72.0 * F + S * 12 + 8 * 6.0 * S, "flops": 100.0 * F * case["directions"]}
    if kind == "hemisphere":
        rays = S * case["rays"] + S / 2 * case["sun_samples"]
        edges = S * min(case["top_k"], 0.36 * case["rays"])
        return {"bytes": 72.0 * F + 8 * edges + S * 16,
                "flops": rays * (40.0 * math.log2(2 * F) + 60)}
    if kind == "image":
        px = case["width"] * case["height"]
        return {"bytes": 72.0 * F + 4 * S * case["bands"] + px * (4.0 + 4 * case["bands"]),
                "flops": 200.0 * F}
    edges = S * 0.4 * case["rays"]
    if kind == "solve":
        return {"bytes": 8 * edges + S * (12 + 16 + 4), "flops": 2 * edges * 64}
    if kind == "batched":
        cols = (case["bands"] + (1 if case["thermal"] else 0)) * case["suns"]
        return {"bytes": 4 * edges + S * (8.0 * (case["bands"]) + 4 * cols + 4 * case["suns"]),
                "flops": 2 * edges * cols * 16}
    if kind == "band_loop":
        return {"bytes": 8 * edges + S * (4 + 4 * 9 + 4) + 80.0 * F,
                "flops": 2 * edges * 10 * 64}
    # the node's 58 single-column solves, about 16 sweeps each, and 2 x 20 + 10 gathers
    return {"bytes": 8 * edges + S * 4 * (2 + 12 + 8) + 80.0 * F, "flops": 2 * edges * 58 * 16}


# ---- scenes -------------------------------------------------------------------
def _leaf_count(case):
    return case["trees"] * LEAVES if case["trees"] else 2 * case["grid"] * case["grid"]


def _facets(case):
    return _leaf_count(case) + 2 * case["grid"] * case["grid"]


def scene_vertices(case, seed):
    """(3F, 6) float32 vertices: leaves (crown by crown, or scattered over the
    plot when there are no trees), then the soil's triangles."""
    rng = np.random.default_rng([seed, 11])
    n, trees, grid = _leaf_count(case), case["trees"], case["grid"]
    half = 5.0 if not trees else 4.0 + 2.75 * math.sqrt(trees)
    if trees:
        h = rng.uniform(4.0, 8.0, trees)
        r = rng.uniform(1.5, 3.0, trees)
        xz = rng.uniform(-half + 3, half - 3, (trees, 2))
        d = rng.normal(size=(n, 3))
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        tree = np.repeat(np.arange(trees), LEAVES)
        rad = r[tree] * rng.uniform(0, 1, n) ** (1.0 / 3.0)
        c = np.stack([xz[tree, 0], h[tree], xz[tree, 1]], 1) + d * rad[:, None]
        c[:, 1] = np.maximum(c[:, 1], 0.3)
        edge = 0.08
    else:
        c = np.stack([rng.uniform(-5, 5, n), rng.uniform(0.2, 1.5, n), rng.uniform(-5, 5, n)], 1)
        edge = 0.05
    nrm = rng.normal(size=(n, 3))
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    if not trees:
        nrm[:, 1] = np.abs(nrm[:, 1])
    helper = np.where(np.abs(nrm[:, 1:2]) < 0.9, [[0.0, 1.0, 0.0]], [[1.0, 0.0, 0.0]])
    t = np.cross(helper, nrm)
    t /= np.linalg.norm(t, axis=1, keepdims=True)
    b = np.cross(nrm, t)
    a0 = rng.uniform(0, 2 * np.pi, n)
    tri = np.stack([c + edge / math.sqrt(3.0) * (np.cos(a0 + k * 2.0944)[:, None] * t +
                                                 np.sin(a0 + k * 2.0944)[:, None] * b)
                    for k in range(3)], 1)
    leaf = np.concatenate([tri, np.repeat(nrm[:, None, :], 3, 1)], 2)
    x = np.linspace(-half, half, grid + 1)
    i, k = (q.ravel() for q in np.meshgrid(np.arange(grid), np.arange(grid), indexing="ij"))
    y = np.zeros(grid * grid)
    p00, p01 = np.stack([x[i], y, x[k]], 1), np.stack([x[i], y, x[k + 1]], 1)
    p11, p10 = np.stack([x[i + 1], y, x[k + 1]], 1), np.stack([x[i + 1], y, x[k]], 1)
    soil = np.concatenate([np.stack([p00, p01, p11], 1), np.stack([p00, p11, p10], 1)])
    up = np.broadcast_to(np.array([0.0, 1.0, 0.0]), soil.shape)
    v = np.concatenate([leaf, np.concatenate([soil, up], 2)])
    return np.ascontiguousarray(v.reshape(-1, 6), np.float32)


def sun_vector():
    z, a = math.radians(SUN[0]), math.radians(SUN[1])
    return np.array([math.sin(z) * math.cos(a), math.cos(z), math.sin(z) * math.sin(a)], np.float32)


def exchange_graph(case, seed):
    """A count-form exchange graph with the statistics of the hemisphere view
    factors of these scenes: each side sends `rays` rays, to sky (10-60 %),
    to its own crown (nearer leaves more often), to soil around its crown and
    to other crowns.  (rows (S + 1), neighbours, counts, denominators, sky
    counts) as int64/int32 tensors on the device, rows sorted by neighbour."""
    dev = _device()
    g = torch.Generator(device=dev)
    g.manual_seed(1000003 * seed + 17)
    F, leaves, rays = _facets(case), _leaf_count(case), case["rays"]
    S = 2 * F
    crown = LEAVES if case["trees"] else leaves
    soil_tris = F - leaves
    step = max(1, (1 << 25) // rays)
    nb, cnt, lens, skies = [], [], [], []
    for s0 in range(0, S, step):
        side = torch.arange(s0, min(S, s0 + step), device=dev, dtype=torch.int32)[:, None]
        n = side.shape[0]
        own = side >> 1
        is_leaf = own < leaves
        rand = lambda *shape: torch.rand(*shape, device=dev, generator=g)  # noqa: E731
        cat = rand(n, rays)
        sky_f = 0.1 + 0.5 * rand(n, 1)
        # own crown (soil sides take a crown drawn per row)
        base = torch.where(is_leaf, own // crown, (rand(n, 1) * (leaves // crown)).int()) * crown
        near = (crown * 2 * rand(n, rays).pow(7)).int()
        to = 2 * base + (2 * (own - base).clamp(min=0) + near) % (2 * crown)
        # soil near the crown: a window of a two-hundredth of the soil, upper sides
        win = max(1, soil_tris // 200)
        at = (base.long() * 2654435761 % soil_tris).int()
        soil = 2 * (leaves + (at + (win * rand(n, rays)).int()) % soil_tris)
        far = (2 * leaves * rand(n, rays)).int().clamp(max=2 * leaves - 1)
        rest = (cat - sky_f) / (1 - sky_f)
        t = torch.where(rest < 0.6, to, torch.where(rest < 0.92, soil, far))
        t = torch.where((cat < sky_f) | ((t >> 1) == own), torch.full_like(t, S), t)
        t = torch.sort(t, dim=1).values
        head = torch.ones_like(t, dtype=torch.bool)
        head[:, 1:] = t[:, 1:] != t[:, :-1]
        pos = head.reshape(-1).nonzero().reshape(-1)
        val = t.reshape(-1)[pos]
        length = torch.diff(pos, append=pos.new_tensor([n * rays])).int()
        keep = val != S
        row = pos // rays
        nb.append(val[keep])
        cnt.append(length[keep])
        lens.append(torch.bincount(row[keep], minlength=n))
        sky = torch.zeros(n, dtype=torch.int32, device=dev)
        sky[row[~keep]] = length[~keep]
        skies.append(sky)
    rows = torch.zeros(S + 1, dtype=torch.int64, device=dev)
    rows[1:] = torch.cumsum(torch.cat(lens), 0)
    denom = torch.full((S,), rays, dtype=torch.int32, device=dev)
    return rows, torch.cat(nb), torch.cat(cnt), denom, torch.cat(skies)


def band_tables(case, seed, bands):
    """Per-band reflectance and transmittance (bands, S) float32: leaves ramp
    0.04 -> 0.48 with tau = 0.4 rho, soil 0.12 -> 0.30, each side a few per
    cent off its material."""
    dev = _device()
    g = torch.Generator(device=dev)
    g.manual_seed(1000003 * seed + 29)
    S, leaves = 2 * _facets(case), _leaf_count(case)
    t = torch.linspace(0, 1, bands, device=dev)[:, None] if bands > 1 else torch.zeros(1, 1, device=dev)
    leaf = torch.arange(S, device=dev)[None, :] < 2 * leaves
    vary = 0.95 + 0.1 * torch.rand(1, S, device=dev, generator=g)
    rho = torch.where(leaf, 0.04 + 0.44 * t, 0.12 + 0.18 * t) * vary
    tau = torch.where(leaf, 0.4 * rho, torch.zeros_like(rho))
    return rho.float().contiguous(), tau.float().contiguous()


def thermal_band(case, seed):
    """One thermal band: emissivity 0.97 leaf / 0.95 soil and the emitted
    radiance at 11 um of facets at 280-320 K."""
    dev = _device()
    g = torch.Generator(device=dev)
    g.manual_seed(1000003 * seed + 31)
    F, leaves = _facets(case), _leaf_count(case)
    eps = torch.where(torch.arange(F, device=dev) < leaves, 0.97, 0.95).repeat_interleave(2)
    T = 280 + 40 * torch.rand(F, device=dev, generator=g, dtype=torch.float64)
    planck = 1.1910439340652e8 / (11.0 ** 5 * torch.expm1(14388.291040407 / (T * 11.0)))
    return (1 - eps).float(), (eps * planck.repeat_interleave(2)).float()


def sun_geometry(case, seed, suns):
    """sunlit fraction times the sun's cosine, (suns, S) float32."""
    dev = _device()
    g = torch.Generator(device=dev)
    g.manual_seed(1000003 * seed + 37)
    S = 2 * _facets(case)
    lit = torch.rand(suns, S, device=dev, generator=g)
    return torch.where(lit < 0.5, torch.zeros_like(lit), (lit - 0.5) * 1.9).float().contiguous()


def sunlit_fractions(case, seed):
    return (sun_geometry(case, seed, 1)[0] / 0.95).clamp(max=1.0).cpu().numpy()


# ---- models -------------------------------------------------------------------
def _model(raster=1024):
    m = fc.FacetrtCuda()
    m.initialize(raster, raster, 1024)
    return m


def _solver_model(case, seed):
    """A model with its geometry and exchange graph: the handle a program
    keeps while it solves."""
    m = _model()
    m.setGeometry(scene_vertices(case, seed))
    m.setGraph(*(a.cpu().numpy() for a in exchange_graph(case, seed)))
    return m


def _batch_facets(case):
    lo, hi, n = math.log(case["lo"]), math.log(case["hi"]), case["scenes"]
    return [_facets(c) for c in (_batch_scene(case, i) for i in range(n))]


def _batch_scene(case, i):
    lo, hi, n = math.log(case["lo"]), math.log(case["hi"]), case["scenes"]
    size = math.exp(lo + (hi - lo) * i / max(1, n - 1))
    trees = int(size * 0.9 / LEAVES)
    leaves = trees * LEAVES
    grid = max(8, int(math.sqrt((size - leaves) / 2))) if trees else max(8, int(math.sqrt(size / 4)))
    return {"trees": trees, "grid": grid, "rays": case["rays"]}


MATERIALS = ([0.05, 0.08, 0.45, 0.30, 0.22], [0.04, 0.06, 0.40], 0.02, 0.01)
BANDS = [450.0, 550.0, 650.0, 865.0, 1240.0, 1610.0, 2200.0, 10000.0, 11000.0]


def _numpy(a):
    return a.cpu().numpy()


def prepare(case, seed):
    """What a program holds before the call: scenes, tables, models."""
    kind = case["kind"]
    if kind == "raster":
        room = np.zeros((2 * _facets(case) * 3 * case["directions"] // 4, 2), np.int32)
        return {"case": case, "model": _model(case["raster"]), "vertices": scene_vertices(case, seed),
                "directions": fc.hemisphere_directions(case["directions"]), "sun": sun_vector(),
                "edges": room}
    if kind == "hemisphere":
        uv, dirs = scenes.hemisphere_samples(case["rays"], 32, seed=7 + seed % 1000)
        suv, _ = scenes.hemisphere_samples(case["sun_samples"], 32, seed=8)
        room = np.zeros((2 * _facets(case) * min(case["top_k"], case["rays"]), 2), np.int32)
        return {"case": case, "model": _model(), "vertices": scene_vertices(case, seed), "uv": uv,
                "dirs": dirs, "sun_uv": suv, "sun": sun_vector(), "edges": room}
    if kind == "solve":
        rho, tau = band_tables(case, seed, 3)
        optics = torch.zeros(rho.shape[1], 4, device=rho.device)
        optics[:, 0], optics[:, 1] = rho[1], tau[1]
        optics[:, 3] = BEAM * sun_geometry(case, seed, 1)[0]
        return {"case": case, "model": _solver_model(case, seed), "optics": _numpy(optics)}
    if kind == "batched":
        rho, tau, emis, sky, beam, dgeo = _batch_inputs(case, seed)
        state = {"case": case, "model": _solver_model(case, seed)}
        given = {"rho": rho, "tau": tau, "emis": emis, "sky": sky, "beam": beam, "dgeo": dgeo}
        if case["host"]:
            return {**state, **{k: None if v is None else _numpy(v) for k, v in given.items()}}
        out = torch.empty(rho.shape[0] * case["suns"], rho.shape[1], device=rho.device)
        return {**state, **given, "out": out}
    if kind == "scene_batch":
        parts, models = [], []
        for i in range(case["scenes"]):
            sc = _batch_scene(case, i)
            models.append(_solver_model(sc, seed + 7919 * i))
            parts.append(_batch_inputs({**sc, "bands": case["bands"], "suns": 1, "thermal": True},
                                       seed + 7919 * i))
        m = _model()
        m.sceneBatch(models)
        for one in models:
            one.close()
        cat = [torch.cat([p[k] for p in parts], 1).contiguous() for k in (0, 1, 2)]
        out = torch.empty_like(cat[0])
        return {"case": {**case, "host": False, "precision": "mixed", "suns": 1}, "model": m,
                "rho": cat[0], "tau": cat[1], "emis": cat[2], "sky": parts[0][3],
                "beam": parts[0][4], "dgeo": torch.cat([p[5] for p in parts], 1).contiguous(),
                "out": out}
    if kind == "band_loop":
        F, leaves = _facets(case), _leaf_count(case)
        mi, tex = _band_materials(case, seed)
        p, keep = fc.spectral_parameters(
            BANDS, leaves, ground=fc.Surface([0.20, 0.22, 0.25], [0.0], 0.05, 0.0, 305.0, 295.0),
            materials=[fc.Surface(*MATERIALS, 301.0, 297.0), fc.Surface([0.15], [0.0], 0.05, 0.0,
                                                                        310.0, 300.0)],
            material_indices=mi, texture_factors=tex, sky_temperature=250.0)
        return {"case": case, "model": _solver_model(case, seed), "parameters": p, "keep": keep,
                "lit": sunlit_fractions(case, seed), "sun": sun_vector()}
    if kind == "energy_node":
        m = _model()
        m.setGeometry(scene_vertices(case, seed))
        uv, dirs = scenes.hemisphere_samples(case["rays"], 32, seed=7)
        m.buildHemisphereGraph(uv, dirs, case["rays"], case["top_k"], 32)
        F, leaves = _facets(case), _leaf_count(case)
        mi = np.where(np.arange(F) < leaves, 0, 1).astype(np.uint32)
        red_edge = np.where(np.arange(2001) < 300, 0.06, 0.46).astype(np.float32)
        surfaces = [fc.EnergySurface(*MATERIALS, energy_reflectance=red_edge,
                                     energy_transmittance=0.8 * red_edge, surface_resistance=150.0,
                                     heat_capacity_per_area=1500.0),
                    fc.EnergySurface([0.15], [0.0], 0.05, 0.0, soil_moisture=0.22)]
        nm = np.arange(2001, dtype=np.float64)
        bands = [450.0, 550.0, 650.0, 865.0, 1610.0, 2200.0, 10000.0, 11000.0]
        rng = np.random.default_rng([seed, 13])
        meteo = dict(air_temperature=24.0 + float(rng.uniform(-2, 2)), vapor_pressure=15.0,
                     pressure=1000.0, wind_speed=2.0, shortwave=750.0, longwave=330.0)
        sun = sun_vector()
        _, windows, bd, bf = fc.shortwave_windows(
            meteo["shortwave"], float(sun[1]), np.exp(-((nm - 150.0) / 600.0) ** 2),
            0.35 * np.exp(-((nm - 20.0) / 300.0) ** 2), 0.8, 100, bands)
        p, keep = fc.energy_parameters(leaves, surfaces, mi, None, 0.0, bands,
                                       solver_tolerance=1e-6)
        T0 = np.full(2 * F, meteo["air_temperature"] + 273.15, np.float32)
        return {"case": case, "model": m, "parameters": p, "keep": keep, "meteo": meteo, "sun": sun,
                "lit": sunlit_fractions(case, seed), "windows": windows, "T0": T0, "bd": bd,
                "bf": bf}
    if kind == "mlp_gradient":
        m = _model(64)
        x, target, params = _network(case, seed)
        m.mlpSetParameters(params)
        return {"case": case, "model": m, "x": x, "target": target}
    # a sensor image
    m = _model()
    v = scene_vertices(case, seed)
    m.setGeometry(v)
    half = float(np.abs(v[:, 0]).max())
    rng = np.random.default_rng([seed, 19])
    position = (half, half, 25.0) if case["perspective"] else (float("nan"),) * 3
    s = fc.sensor(case["width"], case["height"], case["perspective"], case["zenith"], 45.0,
                  50.0 if case["perspective"] else 0.0, 2 * half, 2 * half, position)
    values = rng.uniform(0.02, 0.6, (case["bands"], 2 * _facets(case))).astype(np.float32)
    return {"case": case, "model": m, "sensor": s, "values": values,
            "wavelengths": [450.0 + 100 * b for b in range(case["bands"])]}


def _batch_inputs(case, seed):
    rho, tau = band_tables(case, seed, case["bands"])
    dev = rho.device
    sky = torch.full((case["bands"],), SKY, device=dev)
    beam = torch.full((case["bands"],), BEAM, device=dev)
    emis = None
    if case["thermal"]:  # the last band is thermal: no beam, its own emission
        r, e = thermal_band(case, seed)
        rho = torch.cat([rho, r[None]])
        tau = torch.cat([tau, torch.zeros_like(r)[None]])
        emis = torch.zeros_like(rho)
        emis[-1] = e
        sky = torch.cat([sky, sky.new_tensor([2.0])])
        beam = torch.cat([beam, beam.new_tensor([0.0])])
    return rho, tau, emis, sky, beam, sun_geometry(case, seed, case["suns"])


def _band_materials(case, seed):
    F, leaves = _facets(case), _leaf_count(case)
    rng = np.random.default_rng([seed, 23])
    mi = np.where(np.arange(F) < leaves, rng.choice([0, 0, 0, 1], F), 9).astype(np.uint32)
    return mi, rng.uniform(0.8, 1.2, F).astype(np.float32)


def _network(case, seed):
    rng = np.random.default_rng([seed, 29])
    x = rng.uniform(0.0, 1.0, (case["rows"], 12)).astype(np.float32)
    x[:, 11] = 2 * x[:, 11] - 1
    target = (0.2 * rng.uniform(0.0, 1.0, (case["rows"], 64)) ** 2).astype(np.float32)
    params = np.concatenate(
        [rng.uniform(-1, 1, n) * lim for n, lim in
         ((128 * 12, 0.2), (128, 0.1), (128 * 128, 0.15), (128, 0.1), (64 * 128, 0.18), (64, 0.1))])
    return x, target, params.astype(np.float32)


# ---- one pass -----------------------------------------------------------------
def _ptr(t):
    return None if t is None else t.data_ptr()


def _graph(model, room):
    """The graph as the library hands it over: rows, edges {neighbour, count}
    at the front of the caller's `room` (the rest of it stays 0), denominators,
    sky counts."""
    S, n = ctypes.c_uint32(), ctypes.c_uint64()
    model._check(model.lib.facetcu_graph_size(model.h, ctypes.byref(S), ctypes.byref(n)))
    rows, den, sky = (np.empty(k, np.int32) for k in (S.value + 1, S.value, S.value))
    if n.value > len(room):
        raise RuntimeError(f"{n.value} edges do not fit a room of {len(room)}")
    model._check(model.lib.facetcu_get_graph(
        model.h, *(ctypes.c_void_p(a.ctypes.data) for a in (rows, room, den, sky))))
    return rows, room, den, sky


def run(state):
    case, m, kind = state["case"], state["model"], state["case"]["kind"]
    if kind == "raster":
        m.setGeometry(state["vertices"])
        m.buildVisibilityGraph(state["directions"])
        lit = m.computeSunlitFraction(state["sun"])
        return [*_graph(m, state["edges"]), lit]
    if kind == "hemisphere":
        m.setGeometry(state["vertices"])
        _, dropped = m.buildHemisphereGraph(state["uv"], state["dirs"], case["rays"],
                                            case["top_k"], 32)
        lit = m.hemisphereSunlit(state["sun"], state["sun_uv"], case["sun_samples"], 32)
        return [*_graph(m, state["edges"]), dropped, lit]
    if kind == "solve":
        if case["accelerated"]:
            return m.solveAccelerated(state["optics"], SKY)["radiosity"]
        return m.solve(state["optics"], SKY, 64)["radiosity"]
    if kind in ("batched", "scene_batch"):
        precision = fc.PRECISION_MIXED if case["precision"] == "mixed" else fc.PRECISION_FP32
        if case["host"]:
            out, _ = m.solveBatched(state["rho"], state["tau"], state["sky"], state["beam"],
                                    state["dgeo"], emission=state["emis"], precision=precision,
                                    tolerance=1e-5, maximum_iterations=2000)
            return out
        cfg = fc.BatchConfig(state["rho"].shape[0], case["suns"], precision, fc.WARM_NONE, 2000,
                             1e-5, 0, 0)
        m.solveBatchedDevice(cfg, _ptr(state["rho"]), _ptr(state["tau"]), _ptr(state["emis"]),
                             _ptr(state["sky"]), _ptr(state["beam"]), _ptr(state["dgeo"]), None,
                             _ptr(state["out"]))
        return state["out"]
    if kind == "band_loop":
        bands, enhancement, _ = m.solveBands(state["parameters"], state["lit"], state["sun"])
        return [bands, enhancement]
    if kind == "energy_node":
        out, _ = m.facetebNode(state["parameters"], state["meteo"], state["sun"], state["lit"],
                               state["windows"], state["T0"], state["bd"], state["bf"])
        return out
    if kind == "mlp_gradient":
        loss, grad = m.mlpLossAndGradient(state["x"], state["target"])
        return [loss, grad]
    image, side, _ = m.renderSensorImage(state["sensor"], state["values"], state["wavelengths"])
    return [image, side]


# ---- the same in 64 bits ------------------------------------------------------
def _exchange(case, seed):
    """H(B) = (sky_s L + sum_n count B_n) / denom as a function of (S, cols)
    float64 panels, without the library."""
    rows, nb, cnt, den, sky = exchange_graph(case, seed)
    S = den.numel()
    A = torch.sparse_csr_tensor(rows.int(), nb.int(), cnt.double(), (S, S))
    den, sky = den.double()[:, None], sky.double()[:, None]
    return lambda B, L: (sky * L + A @ B) / den


def _jacobi(incident, rho, tau, emis, direct, sky, sweeps):
    """B = E + rho H_s + tau H_other from zero; `sweeps`, or to 1e-13."""
    S = rho.shape[0]
    B = torch.zeros_like(rho)
    for _ in range(sweeps or 400):
        H = incident(B, sky) + direct
        new = emis + rho * H + tau * H.view(S // 2, 2, -1).flip(1).reshape(S, -1)
        moved = (new - B).abs().max() / new.abs().max()
        B = new
        if not sweeps and float(moved) < 1e-13:
            break
    return B


def exact(case, seed):
    """run()'s floating outputs in 64 bits.  None for the view-factor builds
    (their counts are whole numbers; the sunlit fractions are ratios of
    counts), for a sensor image (the sides' own values, picked by a whole
    number) and for the FacetEB node (a damped temperature iteration that its
    own tolerance stops, so that its result has no value to converge to)."""
    kind = case["kind"]
    if kind == "mlp_gradient":
        return _network_exact(case, seed)
    if kind == "solve":
        rho, tau = band_tables(case, seed, 3)
        direct = (BEAM * sun_geometry(case, seed, 1)[0]).float().double()[:, None]
        B = _jacobi(_exchange(case, seed), rho[1].double()[:, None], tau[1].double()[:, None], 0.0,
                    direct, SKY, 0 if case["accelerated"] else 64)
        return B[:, 0]
    if kind == "batched":
        return _batched_exact(case, seed)
    if kind == "scene_batch":
        return torch.cat([_batched_exact({**_batch_scene(case, i), "bands": case["bands"],
                                          "suns": 1, "thermal": True}, seed + 7919 * i)
                          for i in range(case["scenes"])], 1)
    if kind == "band_loop":
        return _band_loop_exact(case, seed)
    return None


def _batched_exact(case, seed):
    rho, tau, emis, sky, beam, dgeo = _batch_inputs(case, seed)
    incident = _exchange(case, seed)
    out = []
    for k in range(case["suns"]):
        for b0 in range(0, rho.shape[0], 32):
            b = slice(b0, b0 + 32)
            direct = dgeo[k].double()[:, None] * beam[b].double()[None, :]
            e = 0.0 if emis is None else emis[b].T.double()
            out.append(_jacobi(incident, rho[b].T.double().contiguous(), tau[b].T.double(), e,
                               direct, sky[b].double()[None, :], 0).T)
    return torch.cat(out)


def _band_loop_exact(case, seed):
    """makeSpectralOptics and the 64-sweep solve of each band: optical bands
    as apparent reflectance, and the first band's gain from direct light."""
    dev = _device()
    F, leaves = _facets(case), _leaf_count(case)
    mi, tex = (torch.from_numpy(a.astype(t)).to(dev) for a, t in
               zip(_band_materials(case, seed), (np.int64, np.float64)))
    v = torch.from_numpy(scene_vertices(case, seed)).to(dev).double()
    sun = torch.from_numpy(sun_vector()).to(dev).double()
    cos = (v[::3, 3:] * sun).sum(1)
    cos = torch.stack([cos, -cos], 1).reshape(-1).clamp(min=0)
    lit = torch.from_numpy(sunlit_fractions(case, seed)).to(dev).double()
    incident = _exchange(case, seed)
    f = np.float32
    ground = ([0.20, 0.22, 0.25], [0.0], 0.05, 0.0, 305.0, 295.0)
    surfaces = [MATERIALS + (301.0, 297.0), ([0.15], [0.0], 0.05, 0.0, 310.0, 300.0), ground]
    slot = torch.where(mi < 2, mi, torch.full_like(mi, 2))
    cosz = float(sun_vector()[1])
    ref = 700.0 * cosz + 50.0
    planck = lambda nm, T: 1.1910439340652e8 / (  # noqa: E731
        (nm / 1000) ** 5 * math.expm1(14388.291040407 / (T * nm / 1000)))
    per_band = lambda a, b: float(f(a[min(b, len(a) - 1)]))  # noqa: E731
    out, enhancement = [], None
    for b, nm in enumerate(BANDS):
        thermal = nm > 2500.0
        pick = lambda vals: torch.tensor(vals, dtype=torch.float64, device=dev)[slot]  # noqa: E731
        r = pick([float(f(s[2])) if thermal else per_band(s[0], b) for s in surfaces])
        t = pick([float(f(s[3])) if thermal else per_band(s[1], b) for s in surfaces])
        r = (r if thermal else r * tex).clamp(0, 1)
        t = torch.minimum(t, 1 - r)
        r, t = (q.repeat_interleave(2)[:, None] for q in (r, t))
        if thermal:
            hot, cold = (pick([planck(nm, s[k]) for s in surfaces]).repeat_interleave(2)
                         for k in (4, 5))
            e = ((1 - r - t)[:, 0] * (lit * hot + (1 - lit) * cold))[:, None]
            out.append(_jacobi(incident, r, t, e, 0.0, planck(nm, 250.0), 64)[:, 0])
            continue
        direct = (700.0 * lit * cos)[:, None]
        B = _jacobi(incident, r, t, 0.0, direct, 50.0, 64)[:, 0]
        out.append((B / ref).clamp(0, 1))
        if b == 0:
            diffuse = _jacobi(incident, r, t, 0.0, 0.0 * direct, 50.0, 64)[:, 0]
            enhancement = (out[0] - (diffuse / ref).clamp(0, 1)).clamp(min=0)
    return [torch.stack(out), enhancement]


def _network_exact(case, seed):
    x, target, p = _network(case, seed)
    dev = _device()
    x, target = (torch.from_numpy(a).to(dev).double() for a in (x, target))
    parts, at = [], 0
    for shape in ((128, 12), (128,), (128, 128), (128,), (64, 128), (64,)):
        n = int(np.prod(shape))
        q = torch.from_numpy(p[at:at + n].reshape(shape)).to(dev)
        q = q.bfloat16().double() if len(shape) == 2 else q.double()  # weights are read in BF16
        parts.append(q.requires_grad_())
        at += n
    w1, b1, w2, b2, w3, b3 = parts
    h = torch.nn.functional.gelu(x @ w1.T + b1)
    h = torch.nn.functional.gelu(h @ w2.T + b2)
    loss = ((h @ w3.T + b3 - target) ** 2).mean()
    loss.backward()
    return [float(loss), torch.cat([q.grad.reshape(-1) for q in parts])]
