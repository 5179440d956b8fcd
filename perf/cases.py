"""The work this library is used for, as cases that can be timed and compared.

Each case is a dict of plain values; prepare() makes what a program holds before the call (a
committed scene, rays, a film, a cache), run() is one pass through the public entry points of
pbrt_b200 (scene.py, cache.py, or the C ABI of include/pbrt_b200.h where a program hands over
device buffers), work() what a pass cannot do without, exact() the answers in 64 bits where
they exist (hit distances against few enough primitives, the network and its gradient).

Every call is the plain synchronous one: it returns when its results are there, as it does for
a program that has set no stream of its own. Films, hits and gradients come back whole.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from pbrt_b200 import workloads
from pbrt_b200.cache import PARAMS, RECORD, RadianceCache
from pbrt_b200.scene import Batch, Scene, create_scenes, default_context, render_params

NEAR, FAR = 1e-4, 1e30
LAYERS = ((96, 64), (64, 64), (64, 64), (64, 64), (64, 64), (64, 16))  # (inputs, outputs) of the network, padded
IN, OUT = 82, 3  # of which used


def listed():
    return [
        # A program whose rays live in its own (pageable) memory asks for a few thousand at a
        # time: an integrator that keeps its loop on the host. Launches, copies and waits.
        dict(name="rays_host_small", kind="rays", query="closest", level=5, rays=4099, memory="host", spread=1.5),
        # The headline ray cast: 2^24 incoherent rays, device-resident, a 327,680-triangle mesh.
        dict(name="rays_closest_large", kind="rays", query="closest", level=7, rays=1 << 24, memory="device", spread=3.0),
        # Occlusion answers for a ragged batch of shadow rays around the same mesh.
        dict(name="rays_any_ragged", kind="rays", query="any", level=7, rays=3_000_001, memory="device", spread=1.5),
        # Rays against a scene of many objects (10,000 spheres under transforms), object ids wanted.
        dict(name="rays_many_objects", kind="objects", query="closest", objects=10_000, rays=1_500_000),
        # The small render: closed box of triangles, the first image of anyone's day.
        dict(name="render_box", kind="render", scene="box", size=0, width=256, height=256, spp=16, depth=8, roulette=0),
        # Analytic shapes, a deep top-level tree, glass and metal, sky light, Russian roulette.
        dict(name="render_spheres", kind="render", scene="spheres", size=10_000, width=1024, height=768, spp=64, depth=16,
             roulette=4),
        # A heavy mesh in a closed box at full HD, few samples, long paths.
        dict(name="render_knot", kind="render", scene="knot", size=10_627, width=1920, height=1080, spp=4, depth=32,
             roulette=4),
        # Many small scenes as one batch: thumbnails or training views.
        dict(name="batch_small_scenes", kind="batch", scenes=24, width=128, height=128, spp_max=32, level_max=5),
        # The first frame after a cut with the learned cache: reset, one training round beside
        # the frame, two samples a pixel whose paths end into the network.
        dict(name="cached_frame", kind="cached", size=10_627, width=1920, height=1080, spp=2, depth=32, roulette=4),
        # The network alone, forward: radiance for a frame's worth of surface points.
        dict(name="cache_query", kind="query", records=2_000_003),
        # Forward and backward: the gradient of one training batch of the online trainer.
        dict(name="cache_gradient", kind="gradient", records=1 << 14),
        # Geometry that changes: the mesh's tree built anew on the GPU, then traced.
        dict(name="rebuild_and_trace", kind="rebuild", level=7, bins=16, leaf=4, rays=100_003),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rays", "rays", "objects", "render", "render", "batch", "cached", "query", "gradient", "rebuild"])
    if kind == "rays":
        memory = rng.choice(["device", "device", "host"])
        return dict(kind=kind, query=rng.choice(["closest", "any"]), level=rng.randint(3, 7),
                    rays=_log(rng, 1000, (1 << 24) if memory == "device" else 2_000_000), memory=memory,
                    spread=round(rng.uniform(1.0, 3.0), 2))
    if kind == "objects":
        return dict(kind=kind, query=rng.choice(["closest", "any"]), objects=_log(rng, 30, 10_000),
                    rays=_log(rng, 1000, 1_500_000))
    if kind == "render":
        scene = rng.choice(["box", "spheres", "knot"])
        size = {"box": 0, "spheres": _log(rng, 30, 10_000), "knot": _log(rng, 300, 10_627)}[scene]
        width, height, roulette = _log(rng, 64, 1920), _log(rng, 64, 1080), rng.choice([0, 4])
        spp = min(_log(rng, 1, 64), (8_000_000 if roulette else 2_000_000) // (width * height))
        return dict(kind=kind, scene=scene, size=size, width=width, height=height, spp=max(1, spp),
                    depth=rng.randint(2, 32), roulette=roulette)
    if kind == "batch":
        return dict(kind=kind, scenes=_log(rng, 4, 32), width=_log(rng, 32, 160), height=_log(rng, 32, 160),
                    spp_max=_log(rng, 4, 32), level_max=rng.randint(3, 5))
    if kind == "cached":
        return dict(kind=kind, size=_log(rng, 300, 10_627), width=_log(rng, 128, 1920), height=_log(rng, 128, 1080),
                    spp=rng.randint(1, 2), depth=rng.randint(6, 32), roulette=rng.choice([0, 4]))
    if kind == "query":
        return dict(kind=kind, records=_log(rng, 100, 2_000_003))
    if kind == "gradient":
        return dict(kind=kind, records=_log(rng, 100, 1 << 16))
    bins, leaf = rng.choice([(8, 1), (16, 4)])
    return dict(kind="rebuild", level=rng.randint(3, 7), bins=bins, leaf=leaf, rays=_log(rng, 1000, 1_000_000))


# ---- inputs ----------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _rays(seed, n, lo, hi, spread, shadow):
    """(8, n) float32 planes on the GPU: origins uniform in a cube of `spread` times the box's
    largest side, directions uniform on the sphere; shadow rays end at a point as far away as
    the box is large or nearer."""
    g = _generator(seed)
    u = torch.rand(6, n, generator=g, device="cuda")
    side = float(max(hi[k] - lo[k] for k in range(3)))
    centre = torch.tensor([(lo[k] + hi[k]) / 2 for k in range(3)], dtype=torch.float32, device="cuda")
    rays = torch.empty(8, n, device="cuda")
    rays[0:3] = centre[:, None] + (u[0:3] - 0.5) * (spread * side)
    z, phi = u[3] * 2 - 1, u[4] * (2 * math.pi)
    s = (1 - z * z).clamp_min(0).sqrt()
    d = torch.stack([s * phi.cos(), s * phi.sin(), z])
    rays[3:6] = d * ((d[0] * d[0] + d[1] * d[1]) + d[2] * d[2]).rsqrt()
    rays[6] = NEAR
    rays[7] = NEAR + u[5] * side if shadow else FAR
    return rays


def _mesh_desc(v, f, bins, leaf):
    return dict(meshes=[dict(vertices=v, indices=f)], materials=[dict(kind=0, color=(0.5, 0.5, 0.5))],
                objects=[dict(shape=0, mesh=0, material=0, to_world=None, to_local=None)], lights=[], bvh_bins=bins,
                bvh_max_leaf=leaf)


def _mesh_case(case, seed):
    v, f = workloads.displaced_icosphere(case["level"], seed=seed % 100_003)
    rays = _rays(seed, case["rays"], v.min(0), v.max(0), case.get("spread", 2.0), case.get("query") == "any")
    return v, f, rays.cpu().numpy() if case.get("memory") == "host" else rays


def _objects_case(case, seed):
    desc, _ = workloads.many_spheres(case["objects"], seed=seed % 100_003)
    return desc, _rays(seed, case["rays"], (-10.0,) * 3, (10.0,) * 3, 1.2, case["query"] == "any")


def _render_scene(case, seed):
    if case.get("scene") == "box":
        return workloads.cornell_box(case["width"], case["height"])
    if case.get("scene") == "spheres":
        return workloads.many_spheres(case["size"], seed=seed % 100_003, width=case["width"], height=case["height"])
    return workloads.radiance_cache_scene(case["width"], case["height"], segments=case["size"], seed=seed % 100_003)


def _film(width, height):
    return torch.zeros(height, width, 3, dtype=torch.float64, device="cuda")


def _records(seed, n):
    """Surface points of a unit box: position, roughness, direction, normal, albedo."""
    g = _generator(seed)
    r = torch.zeros(n, RECORD, device="cuda")
    r[:, 0:4] = torch.rand(n, 4, generator=g, device="cuda")
    for at in (4, 8):
        v = torch.randn(n, 3, generator=g, device="cuda")
        r[:, at:at + 3] = v / v.norm(dim=1, keepdim=True)
    r[:, 12:15] = torch.rand(n, 3, generator=g, device="cuda")
    return r


def _targets(seed, n):
    return -torch.log1p(-torch.rand(n, OUT, generator=_generator(seed + 7), device="cuda"))  # radiance: many dim, few bright


def _weights(seed):
    """He-uniform weights of the seed, the padded inputs and outputs zero."""
    g = torch.Generator().manual_seed(seed)
    parts = []
    for k, (i, o) in enumerate(LAYERS):
        used_i, used_o = IN if k == 0 else i, OUT if k == len(LAYERS) - 1 else o
        w = torch.zeros(o, i)
        w[:used_o, :used_i] = (torch.rand(used_o, used_i, generator=g) * 2 - 1) * math.sqrt(6.0 / used_i)
        parts.append(w.reshape(-1))
    return torch.cat(parts)


def _cache(seed, scene_min=(0.0, 0.0, 0.0), scene_max=(1.0, 1.0, 1.0)):
    return RadianceCache(scene_min, scene_max, seed=seed)


def prepare(case, seed):
    kind, s = case["kind"], dict(case=case)
    if kind == "rays":
        v, f, s["rays"] = _mesh_case(case, seed)
        s["scene"] = Scene.from_description(_mesh_desc(v, f, 16, 4)).commit(device_build=True)
    elif kind == "objects":
        desc, s["rays"] = _objects_case(case, seed)
        s["scene"] = Scene.from_description(desc).commit()
    elif kind == "render":
        desc, s["camera"] = _render_scene(case, seed)
        s["scene"], s["seed"] = Scene.from_description(desc).commit(device_build=True), seed
        s["film"] = _film(case["width"], case["height"])
    elif kind == "batch":
        made = workloads.batch_scenes(case["scenes"], seed=seed % 100_003, width=case["width"], height=case["height"],
                                      levels=(3, case["level_max"]), spp=(4, case["spp_max"]))
        scenes = create_scenes([d for d, _, _ in made], device_build=True)
        s["batch"] = Batch(scenes, [render_params(cam, spp, 8, seed=seed + i) for i, (_, cam, spp) in enumerate(made)])
        s["films"] = [_film(case["width"], case["height"]) for _ in made]
    elif kind == "cached":
        desc, s["camera"] = _render_scene(case, seed)
        s["scene"], s["seed"] = Scene.from_description(desc).commit(device_build=True), seed
        s["cache"] = _cache(seed, (-0.5,) * 3, (0.5,) * 3)
        s["film"] = _film(case["width"], case["height"])
    elif kind in ("query", "gradient"):
        s["cache"] = _cache(seed)
        s["cache"].set_weights(_weights(seed).numpy())
        s["records"] = _records(seed, case["records"])
        if kind == "query":
            s["rgb"] = torch.zeros(case["records"], OUT, device="cuda")
        else:
            s["targets"], s["gradient"] = _targets(seed, case["records"]), torch.zeros(PARAMS, device="cuda")
    else:
        v, f, s["rays"] = _mesh_case(case, seed)
        s["desc"] = _mesh_desc(v, f, case["bins"], case["leaf"])
    torch.cuda.synchronize()  # the calls run on the library's own stream
    return s


# ---- one pass --------------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "rays":
        return s["scene"].intersect(s["rays"]) if case["query"] == "closest" else s["scene"].intersect_p(s["rays"])
    if kind == "objects":
        if case["query"] == "closest":
            return s["scene"].intersect(s["rays"], with_object=True)
        return s["scene"].intersect_p(s["rays"])
    if kind == "render":
        return s["scene"].render(s["camera"], case["spp"], case["depth"], seed=s["seed"], rr_start=case["roulette"],
                                 film=s["film"])
    if kind == "batch":
        return s["batch"].render(0, films=s["films"])
    if kind == "cached":
        s["cache"].reset()
        return s["scene"].render_cached(s["cache"], s["camera"], case["spp"], case["depth"], seed=s["seed"],
                                        rr_start=case["roulette"], train_rounds=1, film=s["film"])
    if kind in ("query", "gradient"):
        cache, rec = s["cache"], s["records"]
        ctx = cache.ctx
        if kind == "query":
            ctx.check(ctx.lib.pbrt_cache_query(cache.h, rec.data_ptr(), rec.shape[0], s["rgb"].data_ptr()), "query")
            return s["rgb"]
        loss = C.c_float()
        ctx.check(ctx.lib.pbrt_cache_gradient(cache.h, rec.data_ptr(), s["targets"].data_ptr(), rec.shape[0],
                                              s["gradient"].data_ptr(), C.byref(loss)), "gradient")
        return s["gradient"], loss.value
    scene = Scene.from_description(s["desc"], default_context()).commit(device_build=True)
    info = scene.info()
    return scene.intersect(s["rays"]), [info[k] for k in ("mesh_node_count", "mesh_leaf_count", "mesh_max_depth")]


# ---- what a pass cannot do without -----------------------------------------------------------
def _knot_bytes(case):
    return 2 * case["size"] * 41 * 40


def work(case):
    kind = case["kind"]
    if kind in ("rays", "objects"):
        answer = 1 if case["query"] == "any" else 8 if kind == "rays" else 12
        scene = 20 * 4 ** case["level"] * 36 if kind == "rays" else case["objects"] * 100
        return dict(bytes=case["rays"] * (32 + answer) + scene, flops=case["rays"] * 24)
    if kind in ("render", "cached"):
        scene = {"box": 34 * 36, "spheres": case["size"] * 100}.get(case.get("scene"), _knot_bytes(case))
        pixels = case["width"] * case["height"]
        per_path = 400 + (2 * (IN * 64 + 4 * 64 * 64 + 64 * OUT) if kind == "cached" else 0)
        return dict(bytes=pixels * 24 + scene, flops=pixels * case["spp"] * per_path)
    if kind == "batch":
        pixels = case["scenes"] * case["width"] * case["height"]
        return dict(bytes=pixels * 24, flops=pixels * (4 + case["spp_max"]) / 2 * 400)
    net = 2 * (IN * 64 + 4 * 64 * 64 + 64 * OUT)
    if kind == "query":
        return dict(bytes=case["records"] * (RECORD * 4 + 12), flops=case["records"] * net)
    if kind == "gradient":
        return dict(bytes=case["records"] * (RECORD * 4 + 12) + PARAMS * 8, flops=case["records"] * net * 3)
    triangles = 20 * 4 ** case["level"]
    return dict(bytes=triangles * (12 + 6 + 72) + case["rays"] * 40, flops=triangles * 100)


# ---- the answers in 64 bits ------------------------------------------------------------------
def _mesh_distances(v, f, rays):
    """Nearest hit distance of every ray, every triangle tried (Moller-Trumbore)."""
    tri = torch.from_numpy(v.astype(np.float64)[f.astype(np.int64)]).cuda()
    p0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    r = torch.as_tensor(rays).cuda().double()
    out = torch.full((r.shape[1],), math.inf, dtype=torch.float64, device="cuda")
    step = max(1, 4_000_000 // tri.shape[0])
    for a in range(0, r.shape[1], step):
        o, d = r[0:3, a:a + step].T[:, None], r[3:6, a:a + step].T[:, None]
        q = torch.cross(d.expand(-1, tri.shape[0], -1), e2[None].expand(d.shape[0], -1, -1), dim=2)
        det = (e1 * q).sum(2)
        s = o - p0
        u = (s * q).sum(2) / det
        q = torch.cross(s, e1[None].expand_as(s), dim=2)
        w, t = (d * q).sum(2) / det, (e2 * q).sum(2) / det
        ok = (det.abs() >= 1e-8) & (u >= 0) & (w >= 0) & (u + w <= 1)
        ok &= (t >= r[6, a:a + step, None]) & (t <= r[7, a:a + step, None])
        out[a:a + step] = torch.where(ok, t, math.inf).amin(1)
    return out


def _sphere_distances(desc, rays):
    """Nearest hit distance of every ray, every sphere tried."""
    c = torch.tensor(np.stack([o["to_world"][[3, 7, 11]] for o in desc["objects"]]), dtype=torch.float64, device="cuda")
    r2 = torch.tensor([float(np.float32(o["radius"])) for o in desc["objects"]], dtype=torch.float64, device="cuda") ** 2
    r = rays.double()
    out = torch.full((r.shape[1],), math.inf, dtype=torch.float64, device="cuda")
    step = max(1, 60_000_000 // c.shape[0])
    for a in range(0, r.shape[1], step):
        o, d = r[0:3, a:a + step].T, r[3:6, a:a + step].T
        tca = d @ c.T - (o * d).sum(1, keepdim=True)
        d2 = ((o * o).sum(1, keepdim=True) - 2 * (o @ c.T) + (c * c).sum(1)) - tca * tca
        thc = (r2 - d2).clamp_min(0).sqrt()
        near, far = r[6, a:a + step, None], r[7, a:a + step, None]
        t = torch.where(tca - thc > near, tca - thc, tca + thc)
        out[a:a + step] = torch.where((tca >= 0) & (d2 <= r2) & (t > near) & (t < far), t, math.inf).amin(1)
    return out


def _network(records, weights):
    x = records.double()
    octave = (x[:, 0:3, None] * math.pi) * (2.0 ** torch.arange(12, dtype=torch.float64, device="cuda"))
    bands = torch.stack([octave.sin(), octave.cos()], 3).reshape(-1, 72)
    h = torch.cat([bands, x[:, 4:7], x[:, 8:11], x[:, 12:15], x[:, 3:4]], 1)
    h = torch.nn.functional.pad(h, (0, LAYERS[0][0] - IN))
    at = 0
    for k, (i, o) in enumerate(LAYERS):
        h = h @ weights[at:at + i * o].view(o, i).T
        h = h.relu() if k < len(LAYERS) - 1 else h
        at += i * o
    return h[:, :OUT]


def exact(case, seed):
    kind = case["kind"]
    if kind == "rays" and case["query"] == "closest" and case["rays"] * 20 * 4 ** case["level"] < 2e9:
        v, f, rays = _mesh_case(case, seed)
        return None, _mesh_distances(v, f, rays)
    if kind == "rebuild" and case["rays"] * 20 * 4 ** case["level"] < 2e9:
        v, f, rays = _mesh_case(case, seed)
        return (None, _mesh_distances(v, f, rays)), None
    if kind == "objects" and case["query"] == "closest":
        return None, _sphere_distances(*_objects_case(case, seed)), None
    if kind == "query":
        w, rec = _weights(seed).cuda().double(), _records(seed, case["records"])
        return torch.cat([_network(part, w) for part in rec.split(1 << 18)])
    if kind == "gradient":
        w = _weights(seed).cuda().double().requires_grad_()
        o = _network(_records(seed, case["records"]), w)
        d = o - _targets(seed, case["records"]).double()
        loss = (d * d / (o.detach() ** 2 + 0.01)).sum() / o.numel()  # relative squared error, its denominator held
        return torch.autograd.grad(loss, w)[0], float(loss.detach())
    # Rendered images have no 64-bit value: a path's random decisions follow from FP32 comparisons.
    return None
