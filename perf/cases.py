"""Performance cases: the work a user of this renderer has it do, one call (or
one frame) at a time, through the package's public entry points.

Every case is a dict of plain values with a "kind":

  mesh_closest    Scene.mesh_intersect on one triangle soup (the closest-hit
                  query set of the benchmark and smaller ones): collision,
                  picking and baking queries against one mesh. `tuned` passes
                  the launch configuration the benchmark settles on; without
                  it the call takes the library's default.
  scene_closest   Scene.intersect with hit geometry on the museum-like scene:
                  half camera rays in image order, half incoherent rays.
  scene_occluded  Scene.intersectP on the same scene: shadow and
                  ambient-occlusion rays, bounded and unbounded.
  render          Scene.render: fixed or adaptive sampling, the wavefront or
                  the plain integrator, on the museum-like scene or the
                  Cornell box.
  caustic_frame   PhotonMap.emit + build + render_caustics: one frame of the
                  caustics scene from new photons.
  photon_gather   PhotonMap.gather: k-nearest irradiance at given points.
  tonemap         tonemap(): the display transform of one frame.
  serve           Server.submit + wait of a batch of mixed requests.

Sizes are those of the repository's benchmark configurations and tests, or
smaller and ragged ones of the same shapes. Inputs come from the seed alone.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import photorealisticrender4610_b200 as prr
from photorealisticrender4610_b200 import scenes as sc

# The launch configuration bench.py's autotuner picks on the query set.
TUNED = {"block_size": 128, "persistent": 2, "batch": 8, "sort_rays": 5}


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # a picking / collision query: a few thousand rays, latency counts
        dict(name="mesh_closest_small", kind="mesh_closest", tris=10_000, rays=4_099, tuned=False),
        # baking: a mid-size soup with the default call
        dict(name="mesh_closest_default", kind="mesh_closest", tris=300_000, rays=1_500_007,
             tuned=False),
        # the benchmark's closest-hit query set
        dict(name="mesh_closest_query_set", kind="mesh_closest", tris=1_000_000, rays=4_194_304,
             tuned=True),
        # scene-level queries with hit geometry (custom integrators, AOVs)
        dict(name="scene_closest", kind="scene_closest", level=5, rays=2_000_003),
        # scene-level visibility (shadow, ambient occlusion)
        dict(name="scene_occluded", kind="scene_occluded", level=5, rays=2_000_003),
        # a museum-like frame on the wavefront integrator, fixed samples
        dict(name="render_frame", kind="render", scene="museum", level=6, width=960, height=540,
             spp=16, min_spp=16, depth=8, mode="wavefront"),
        # the reference's default mode: adaptive sampling, up to depth 12
        dict(name="render_adaptive", kind="render", scene="museum", level=4, width=320,
             height=180, spp=64, min_spp=1, depth=12, mode="wavefront"),
        # the Cornell box of the plain method (Scene.render's default mode)
        dict(name="render_plain", kind="render", scene="cornell", level=0, width=256, height=256,
             spp=16, min_spp=16, depth=5, mode="plain"),
        # one caustics frame from new photons, 64-nearest gathers
        dict(name="caustic_frame", kind="caustic_frame", photons=2_000_000, width=1024,
             height=1024, spp=32, k=64, radius=0.02, depth=8),
        # irradiance at given points (a lightmap, a final gather)
        dict(name="photon_gather", kind="photon_gather", photons=40_000, points=60_013, k=64,
             radius=0.02),
        # the display transform of a 1920x1080 frame
        dict(name="tonemap_frame", kind="tonemap", width=1920, height=1080, mapper="agx",
             exposure=1.0),
        # a render server with a handful of mixed requests in flight
        dict(name="serve_mix", kind="serve", requests=8, max_side=512, max_spp=32, depth=8),
    ]


def _log_int(rng, lo, hi):
    """An integer in [lo, hi], uniform over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["mesh_closest", "scene_closest", "scene_occluded", "render", "render",
                       "caustic_frame", "photon_gather", "tonemap", "serve"])
    if kind == "mesh_closest":
        return dict(kind=kind, tris=_log_int(rng, 1_000, 1_000_000),
                    rays=_log_int(rng, 1_000, 4_000_000), tuned=rng.random() < 0.5)
    if kind in ("scene_closest", "scene_occluded"):
        return dict(kind=kind, level=rng.randint(2, 6), rays=_log_int(rng, 1_000, 2_000_000))
    if kind == "render":
        museum = rng.random() < 0.7
        spp = _log_int(rng, 1, 16)
        plain = rng.random() < 0.3
        adaptive = rng.random() < 0.3
        if adaptive:
            spp *= 4
        return dict(kind=kind, scene="museum" if museum else "cornell",
                    level=rng.randint(3, 6) if museum else 0,
                    width=_log_int(rng, 33, 640), height=_log_int(rng, 33, 360), spp=spp,
                    min_spp=1 if adaptive else spp, depth=rng.randint(2, 12),
                    mode="plain" if plain else "wavefront")
    if kind == "caustic_frame":
        return dict(kind=kind, photons=2 * _log_int(rng, 50_000, 1_000_000),
                    width=_log_int(rng, 128, 1024), height=_log_int(rng, 128, 1024),
                    spp=_log_int(rng, 1, 32), k=rng.choice([0, 16, 64]),
                    radius=rng.choice([0.01, 0.02]), depth=rng.randint(4, 12))
    if kind == "photon_gather":
        return dict(kind=kind, photons=_log_int(rng, 2_000, 50_000),
                    points=_log_int(rng, 1_000, 100_000), k=rng.choice([0, 8, 32, 64]),
                    radius=rng.choice([0.01, 0.02]))
    if kind == "tonemap":
        return dict(kind=kind, width=_log_int(rng, 64, 3840), height=_log_int(rng, 64, 2160),
                    mapper=rng.choice(["raw", "standard", "agx", "pbrneutral", "aces"]),
                    exposure=rng.choice([0.18, 1.0, 2.5]))
    return dict(kind="serve", requests=rng.randint(2, 8), max_side=rng.choice([128, 256, 512]),
                max_spp=_log_int(rng, 4, 32), depth=rng.randint(4, 8))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 13)
    return g


def _uniform(g, n, lo, hi):
    """(n, 3) float32 uniform in the box [lo, hi]."""
    lo = torch.tensor(lo, dtype=torch.float32, device="cuda")
    hi = torch.tensor(hi, dtype=torch.float32, device="cuda")
    return lo + (hi - lo) * torch.rand(n, 3, generator=g, device="cuda")


def _directions(g, n):
    v = torch.randn(n, 3, generator=g, device="cuda")
    return v / v.norm(dim=1, keepdim=True).clamp_min(1e-12)


@functools.lru_cache(maxsize=2)
def _sky(width, height):
    return sc.procedural_sky(width, height)


def _museum(level, seed, width, height):
    """The museum-like scene at a lower subdivision level (its own sky size)."""
    desc = sc.museum_like(width, height, level=level, seed=1 + int(seed) % 10_000,
                          env_size=(4, 2))
    desc.env = _sky(1024, 512)
    return desc


def _scene_rays(case, seed):
    """Half camera rays in image order, half incoherent rays inside the room."""
    n = case["rays"]
    g = _gen(seed)
    half = n // 2
    eye = torch.tensor([0.0, 2.6, 6.5], device="cuda")
    side = max(1, int(math.ceil(math.sqrt(half))))
    k = torch.arange(half, device="cuda")
    x = ((k % side).float() + torch.rand(half, generator=g, device="cuda")) / side * 6.0 - 3.0
    y = torch.div(k, side, rounding_mode="floor").float() / side * 3.0 - 0.5
    target = torch.stack([x, y, torch.zeros_like(x)], 1)
    d0 = target - eye
    d0 = d0 / d0.norm(dim=1, keepdim=True)
    o0 = eye.expand(half, 3)
    o1 = _uniform(g, n - half, (-3.5, 0.05, -3.0), (3.5, 2.5, 3.0))
    d1 = _directions(g, n - half)
    return torch.cat([o0, o1]).contiguous(), torch.cat([d0, d1]).contiguous(), g


def _photons(n, seed):
    """Caustic photons on a floor: half in a Gaussian focus, half spread over
    a disc, arriving from above with a few percent of power variation."""
    r = np.random.Generator(np.random.PCG64(int(seed) + 101))
    a = n // 2
    xz = np.concatenate([r.normal(0.0, 0.15, (a, 2)), _disc(r, n - a)])
    rec = np.zeros((n, 9), np.float32)
    rec[:, 0] = xz[:, 0]
    rec[:, 1] = r.uniform(-1e-4, 1e-4, n)
    rec[:, 2] = xz[:, 1]
    d = np.stack([r.normal(0, 0.2, n), -np.ones(n), r.normal(0, 0.2, n)], 1)
    rec[:, 3:6] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rec[:, 6:9] = 1e-4 * r.uniform(0.9, 1.1, (n, 3))
    return rec[r.permutation(n)]


def _disc(r, n):
    rad, phi = np.sqrt(r.random(n)), r.uniform(0.0, 2.0 * math.pi, n)
    return np.stack([rad * np.cos(phi), rad * np.sin(phi)], 1)


def _points(n, seed):
    r = np.random.Generator(np.random.PCG64(int(seed) + 202))
    xz = _disc(r, n)
    return np.stack([xz[:, 0], np.zeros(n), xz[:, 1]], 1).astype(np.float32)


def _hdr_frame(case, seed):
    """Linear radiance as a renderer leaves it: log-normal around 0.3 with a
    few bright highlights and black pixels."""
    g = _gen(seed)
    h, w = case["height"], case["width"]
    x = torch.exp(torch.randn(h, w, 3, generator=g, device="cuda") * 1.2 - 1.2)
    u = torch.rand(h, w, 1, generator=g, device="cuda")
    x = torch.where(u > 0.995, x * 300.0, x)
    return torch.where(u < 0.02, torch.zeros_like(x), x).contiguous()


def _soup(n, seed):
    desc = sc.SceneDesc(width=256, height=256, name="soup")
    m = desc.add_material(sc.Material(sc.DIFFUSE, (0.7, 0.6, 0.5), 0.6, 0.0))
    verts, _, _ = sc.query_set(n, 1, seed=int(seed) + 7)
    desc.objects.append(sc.MeshObject(verts, m))
    desc.env = _sky(1024, 512)
    desc.camera = sc.Camera(eye=(2.2, 1.6, 2.4), target=(0.5, 0.5, 0.5), fovv=40, fovh=45)
    return desc


def _requests(case, seed):
    """(scene, width, height, spp): the sizes stand for the case (uniform in
    logarithm); which scene each request renders changes with the seed."""
    r = np.random.Generator(np.random.PCG64(int(seed) * 31 + 5))
    s = np.random.Generator(np.random.PCG64(case["requests"] * 1009 + case["max_side"]))
    out = []
    for _ in range(case["requests"]):
        w = int(round(math.exp(s.uniform(math.log(64), math.log(case["max_side"])))))
        h = int(round(math.exp(s.uniform(math.log(64), math.log(case["max_side"])))))
        spp = int(round(math.exp(s.uniform(math.log(4), math.log(max(4, case["max_spp"]))))))
        out.append((int(r.integers(0, 2)), w, h, spp))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mesh_closest":
        verts, o, d = sc.query_set(case["tris"], case["rays"], seed=int(seed) + 1)
        return dict(case=case, scene=prr.Scene.single_mesh(verts),
                    o=torch.from_numpy(o).cuda(), d=torch.from_numpy(d).cuda(),
                    config=TUNED if case["tuned"] else None)
    if kind in ("scene_closest", "scene_occluded"):
        scene = prr.Scene.from_desc(_museum(case["level"], seed, 960, 540))
        o, d, g = _scene_rays(case, seed)
        state = dict(case=case, scene=scene, o=o, d=d)
        if kind == "scene_occluded":
            n = case["rays"]
            t = torch.rand(n, generator=g, device="cuda") * 4.0 + 0.05
            far = torch.rand(n, generator=g, device="cuda") < 0.5
            state["tmax"] = torch.where(far, torch.full_like(t, math.inf), t)
        return state
    if kind == "render":
        desc = (_museum(case["level"], seed, case["width"], case["height"])
                if case["scene"] == "museum" else sc.cornell_box(case["width"], case["height"]))
        return dict(case=case, scene=prr.Scene.from_desc(desc), seed=1 + int(seed))
    if kind == "caustic_frame":
        desc = sc.caustics(case["width"], case["height"])
        return dict(case=case, scene=prr.Scene.from_desc(desc), pm=prr.PhotonMap(),
                    seed=1 + int(seed))
    if kind == "photon_gather":
        pm = prr.PhotonMap().set(_photons(case["photons"], seed)).build(case["radius"])
        return dict(case=case, pm=pm, points=_points(case["points"], seed))
    if kind == "tonemap":
        return dict(case=case, rgb=_hdr_frame(case, seed))
    srv = prr.Server()
    for desc in (_museum(4, seed, 256, 256), _soup(50_000, seed)):
        srv.add_scene(prr.Scene.from_desc(desc))
    reqs = _requests(case, seed)
    outs = [torch.empty(h, w, 3, dtype=torch.float32, device="cuda") for _, w, h, _ in reqs]
    return dict(case=case, server=srv, reqs=reqs, outs=outs, seed=1 + int(seed) * 100)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "mesh_closest":
        return state["scene"].mesh_intersect(0, state["o"], state["d"], config=state["config"])
    if kind == "scene_closest":
        return state["scene"].intersect(state["o"], state["d"], geo=True)
    if kind == "scene_occluded":
        return state["scene"].intersectP(state["o"], state["d"], state["tmax"])
    if kind == "render":
        return state["scene"].render(case["spp"], case["depth"], seed=state["seed"],
                                     min_spp=case["min_spp"], mode=case["mode"])
    if kind == "caustic_frame":
        pm, scene = state["pm"], state["scene"]
        pm.emit(scene, case["photons"], seed=state["seed"], max_depth=case["depth"])
        pm.build(case["radius"])
        return pm.render_caustics(scene, case["spp"], max_depth=case["depth"],
                                  seed=state["seed"], k_nearest=case["k"])
    if kind == "photon_gather":
        return state["pm"].gather(state["points"], k_nearest=case["k"])
    if kind == "tonemap":
        return prr.tonemap(state["rgb"], case["mapper"], exposure=case["exposure"])
    srv = state["server"]
    ids = [srv.submit(s, spp, case["depth"], seed=state["seed"] + k, size=(w, h), out=out)
           for k, ((s, w, h, spp), out) in enumerate(zip(state["reqs"], state["outs"]))]
    for rid in ids:
        srv.wait(rid)
    return state["outs"]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _tree_work(tris, rays):
    """Flops of `rays` tree walks: the two boxes (24 flops each) of one node
    per level down to a four-triangle leaf, and that leaf's tests (45 each)."""
    levels = max(1.0, math.log2(max(2.0, tris / 4.0)))
    return rays * (48.0 * levels + 4 * 45.0)


def _tree_bytes(tris):
    """A mesh once: 36 bytes a triangle and a 64-byte node for four."""
    return tris * 36 + tris / 4 * 64


def work(case):
    kind = case["kind"]
    if kind == "mesh_closest":
        return {"bytes": _tree_bytes(case["tris"]) + case["rays"] * 32,
                "flops": _tree_work(case["tris"], case["rays"])}
    if kind in ("scene_closest", "scene_occluded"):
        tris = 6 * 20 * 4 ** case["level"]
        per_ray = 24 + (36 if kind == "scene_closest" else 5)
        return {"bytes": _tree_bytes(tris) + case["rays"] * per_ray,
                "flops": _tree_work(tris, case["rays"])}
    if kind == "render":
        tris = 6 * 20 * 4 ** case["level"] if case["scene"] == "museum" else 12
        px = case["width"] * case["height"]
        # an adaptive pixel takes at least two samples; a sample traces about
        # two closest-hit rays and a shadow ray and shades two hits
        samples = px * (case["spp"] if case["min_spp"] == case["spp"] else 2)
        return {"bytes": _tree_bytes(tris) + px * 16,
                "flops": _tree_work(tris, 3 * samples) + samples * 2 * 500.0}
    if kind == "caustic_frame":
        px = case["width"] * case["height"]
        # about one photon in forty is stored; a sample traces one ray and
        # tests the photons of its disc
        stored = case["photons"] / 40
        return {"bytes": stored * 36 + px * 12,
                "flops": _tree_work(1300, case["photons"] + px * case["spp"]) +
                px * case["spp"] * 10 * 8.0}
    if kind == "photon_gather":
        # the focus holds half of the photons in about a tenth of the disc
        inside = case["photons"] * case["radius"] ** 2
        return {"bytes": case["photons"] * 24 + case["points"] * 24,
                "flops": case["points"] * max(1.0, inside) * 12.0}
    if kind == "tonemap":
        px = case["width"] * case["height"]
        return {"bytes": px * 27, "flops": px * 120.0}
    px = sum(w * h for _, w, h, _ in _requests(case, 0))
    samples = sum(w * h * spp for _, w, h, spp in _requests(case, 0))
    return {"bytes": _tree_bytes(50_000 + 30_722) + px * 12,
            "flops": _tree_work(40_000, 3 * samples) + samples * 2 * 500.0}


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------
def _exact_closest(verts, o, d):
    """t of the closest hit by testing every triangle in float64 (inf: none)."""
    v = torch.from_numpy(verts).cuda().double().reshape(-1, 3, 3)
    v0, e1, e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    o, d = torch.from_numpy(o).cuda().double(), torch.from_numpy(d).cuda().double()
    n12 = torch.linalg.cross(e1, e2)
    out = []
    rows = max(1, (1 << 26) // len(v0))
    for a in range(0, len(o), rows):
        oo, dd = o[a:a + rows], d[a:a + rows]
        # scalar triple products, expanded so that each is a matrix product
        det = -(dd @ n12.T)
        m = torch.linalg.cross(oo, dd)
        tn = oo @ n12.T - (v0 * n12).sum(1)
        # u = (o - v0) . (d x e2), v = -(o - v0) . (d x e1), with
        # (o - v0) . (d x e) = m . e - d . (e x v0)
        u = m @ e2.T - dd @ torch.linalg.cross(e2, v0).T
        w = -(m @ e1.T - dd @ torch.linalg.cross(e1, v0).T)
        u, w, t = u / det, w / det, tn / det
        ok = (det.abs() >= 1e-6) & (u >= 0) & (w >= 0) & (u + w <= 1) & (t > 1e-3)
        out.append(torch.where(ok, t, torch.full_like(t, math.inf)).amin(1))
    return torch.cat(out).cpu()


def _exact_gather(rec, q, k, radius):
    rec, q = torch.from_numpy(rec).cuda().double(), torch.from_numpy(q).cuda().double()
    pos, power = rec[:, :3], rec[:, 6:9]
    radius = float(np.float32(radius))
    out = []
    rows = max(1, (1 << 25) // len(pos))
    for a in range(0, len(q), rows):
        p = q[a:a + rows]
        dist = torch.sqrt(((p[:, None, 0] - pos[None, :, 0]) ** 2) +
                          ((p[:, None, 1] - pos[None, :, 1]) ** 2) +
                          ((p[:, None, 2] - pos[None, :, 2]) ** 2))
        rk = torch.full((len(p),), radius, dtype=torch.float64, device="cuda")
        if k > 0 and len(pos) > k:
            kth = torch.topk(dist, k + 1, dim=1, largest=False).values
            dense = kth[:, k] <= radius
            rk = torch.where(dense, kth[:, k - 1], rk)
        e = (dist <= rk[:, None]).double() @ power
        out.append(e / (math.pi * rk * rk)[:, None])
    return torch.cat(out).cpu()


def _oetf64(x):
    x = np.clip(x, 0.0, 1.0)
    return np.where(x < 0.0031308, 12.92 * x, 1.055 * np.power(x, 1 / 2.4) - 0.055)


def _agx64(c):
    inset = np.array([[0.544814746488245, 0.373787398372697, 0.0813978551390581],
                      [0.140416948464053, 0.754137554567394, 0.105445496968552],
                      [0.0888104196149096, 0.178871756420858, 0.732317823964232]])
    outset = np.array([[1.96488741169489, -0.855988495690215, -0.108898916004672],
                       [-0.299313364904742, 1.32639796461980, -0.0270845997150571],
                       [-0.164352742528393, -0.238183969428088, 1.40253671195648]])
    x = np.maximum(np.maximum(c, 0.0) @ inset.T, 0.0)
    cross, contrast = 0.1841865, 1.25
    toe = (1 / cross - 1) * cross ** contrast
    slope = contrast * cross ** (contrast - 1) * toe / (cross ** contrast + toe) ** 2
    top = 1 - cross
    w = (16 - cross) ** 2 / top * slope
    t = np.power(x, contrast)
    s = slope * (x - cross)
    s = s * (1 + (x - cross) / w) / (1 + s / top) + cross
    y = np.minimum(np.where(x < cross, t / (t + toe), s), 1.0)
    return _oetf64(y @ outset.T)


def _neutral64(c):
    start, desat = 0.8 - 0.04, 0.15
    x = c.min(-1, keepdims=True)
    c = c - np.where(x < 0.08, x - 6.25 * x * x, 0.04)
    peak = c.max(-1, keepdims=True)
    d = 1 - start
    new = 1 - d * d / (np.maximum(peak, start) + d - start)
    g = 1 - 1 / (desat * (np.maximum(peak, start) - new) + 1)
    hi = c * (new / np.maximum(peak, start)) * (1 - g) + new * g
    return _oetf64(np.where(peak < start, c, hi))


def exact(case, seed):
    kind = case["kind"]
    if kind == "mesh_closest":
        if case["tris"] * case["rays"] > 400_000_000:
            return None
        verts, o, d = sc.query_set(case["tris"], case["rays"], seed=int(seed) + 1)
        return (None, _exact_closest(verts, o, d))
    if kind == "photon_gather":
        return _exact_gather(_photons(case["photons"], seed), _points(case["points"], seed),
                             case["k"], case["radius"])
    if kind == "tonemap":
        c = _hdr_frame(case, seed).cpu().numpy().astype(np.float64) * case["exposure"]
        f = {"raw": lambda x: np.clip(x, 0.0, 1.0), "standard": _oetf64, "agx": _agx64,
             "pbrneutral": _neutral64,
             "aces": lambda x: _oetf64(np.clip(x * (2.51 * x + 0.03) /
                                               (x * (2.43 * x + 0.59) + 0.14), 0.0, 1.0))}
        return (torch.from_numpy(f[case["mapper"]](c)), None)
    return None
