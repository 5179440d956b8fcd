"""Scene::intersect over mixed scenes by the walk of the wide tree (scene_walk.cuh) against the
counted queries, which take the binary trees one object at a time: the same objects, primitives and
distances where a walk in another order, or with another far end, could answer differently."""
import numpy as np
import pytest
import torch

import pbrt_b200 as pb
from pbrt_b200 import workloads as W
from pbrt_b200.scene import Batch, render_params

pytestmark = pytest.mark.gpu
TR = pb.Transform


def _rays(rng, n, spread, aim, near=0.0, far=1e30):
    """Unit directions from a cube of side 2 * spread: half of them random, half towards points of `aim`."""
    o = rng.uniform(-spread, spread, (3, n)).astype(np.float32)
    d = rng.normal(size=(3, n))
    tgt = np.asarray(aim)[rng.integers(0, len(aim), n)].T + rng.normal(size=(3, n)) * 0.5
    d[:, ::2] = (tgt - o)[:, ::2]
    r = np.empty((8, n), np.float32)
    r[0:3], r[3:6], r[6], r[7] = o, W.normalize_f32(d.astype(np.float32)), near, far
    return r


def _commit(objects, **kw):
    s = pb.Scene()
    for o in objects:
        s.add_object(o)
    return s.commit(**kw)


def _same(s, rays):
    """Every query of `rays` against the counted form; the hits' mask."""
    r = torch.from_numpy(np.ascontiguousarray(rays)).cuda()
    torch.cuda.synchronize()
    bp, bt, bo, _ = s.intersect_counted(r)
    wp, wt, wo = s.intersect(r, with_object=True)
    hit = (bo != -1).cpu().numpy()
    bad = (wo != bo) | (wt != bt) | ((wp != bp) & (bo != -1))
    assert not bad.any(), f"{int(bad.sum())} of {rays.shape[1]} answers differ"
    bocc, _ = s.intersect_p_counted(r)
    assert torch.equal(s.intersect_p(r), bocc)
    return hit, bt.cpu().numpy()


def _place(rng, shape, at, rigid=True):
    turn = TR.rotation_x(rng.uniform(0, 6)) * TR.rotation_y(rng.uniform(0, 6))
    return pb.Transformed(pb.Simple(shape), TR.translation([float(x) for x in at]) * turn)


def _analytic(rng, n=24):
    """Overlapping spheres, cylinders, boxes, rectangles and solids of them, turned and moved."""
    out, at = [], rng.uniform(-2, 2, (n, 3))
    for k, c in enumerate(at):
        a, b = rng.uniform(0.3, 1.5, 2)
        shape = [pb.Sphere(a), pb.Cylinder(a, b), pb.AABox((a, b, a)), pb.Rectangle(a, b),
                 pb.Csg("subtraction", [(pb.Sphere(a), TR.identity()), (pb.AABox((a, a, 3 * a)), TR.identity())]),
                 pb.Csg("union", [(pb.Cylinder(a, b), TR.identity()), (pb.Sphere(0.8 * a), TR.translation([0, b / 2, 0]))])][k % 6]
        out.append(_place(rng, shape, c))
    out += [pb.Simple(pb.Sphere(1.0)), pb.Simple(pb.AABox((1.0, 2.5, 0.5)))]
    return out, at


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_an_interval_that_ends_at_a_hit(seed):
    """tmax at a hit's own distance, one float below and one above: the exits of a solid shape count
    only strictly inside the interval, whatever end the walk offers the shape."""
    rng = np.random.default_rng(seed)
    objects, at = _analytic(rng)
    for scene in (objects, objects[:1] + [pb.Simple(pb.Sphere(1.0))], [pb.Simple(pb.Sphere(1.0))]):
        s = _commit(scene)
        rays = _rays(rng, 40_000, 3.0, at)
        hit, t = _same(s, rays)
        assert hit.sum() > 1000
        for end in (t[hit], np.nextafter(t[hit], np.float32(0)), np.nextafter(t[hit], np.float32(1e30))):
            again = rays[:, hit].copy()
            again[7] = end
            _same(s, again)


def _scaling(x, y, z):
    return TR(np.diag([x, y, z, 1.0]), np.diag([1 / x, 1 / y, 1 / z, 1.0]))


def _unordered(rng, n=20):
    """Objects whose distances are not the ray's own: scaled placements of every kind, alone, in chains
    and in compounds, and solids that hold a plane or a scaled element; among meshes and spheres."""
    ball = pb.TriangleMesh(*W.displaced_icosphere(3, seed=9))
    out, at = [], rng.uniform(-4, 4, (n, 3))
    for k, c in enumerate(at):
        scale = [_scaling(2, 2, 2), _scaling(0.5, 0.5, 0.5), _scaling(0.5, 2.0, 1.0)][k // 6 % 3]
        move = TR.translation([float(x) for x in c]) * TR.rotation_z(rng.uniform(0, 6))
        shape = [pb.Sphere(0.6), ball, pb.Cylinder(0.4, 0.8), pb.AABox((0.7, 0.7, 0.7))][k % 4]
        if k % 6 == 0:
            o = pb.Transformed(pb.Simple(shape), move * scale)
        elif k % 6 == 1:
            o = pb.Transformed(pb.Transformed(pb.Simple(shape), scale), move)
        elif k % 6 == 2:
            o = pb.Compound([pb.Transformed(pb.Simple(shape), move * scale), pb.Transformed(pb.Simple(pb.Sphere(0.5)), move)])
        elif k % 6 == 3:
            o = pb.Simple(pb.Csg("intersection", [(pb.Sphere(1.0), move), (pb.Plane(), move)]))
        elif k % 6 == 4:
            o = pb.Simple(pb.Csg("subtraction", [(pb.Sphere(0.6), move * scale), (pb.AABox((0.5, 0.5, 3.0)), move)]))
        else:
            o = pb.Transformed(pb.Simple(pb.Sphere(0.9)), move)
        out.append(o)
    return out + [pb.Simple(ball)], at


@pytest.mark.parametrize("seed", [1, 2, 3, 4])
def test_objects_whose_distances_are_not_the_rays(seed):
    rng = np.random.default_rng(seed)
    objects, at = _unordered(rng)
    for scene in (objects, objects[0::6] + objects[-1:], objects[3::6] + objects[5::6], objects[2::6]):
        hit, _ = _same(_commit(scene), _rays(rng, 100_000, 5.0, at))
        assert hit.sum() > 5000


def test_a_scaled_sphere_before_its_box():
    """The layout that decides by the order: the scaled sphere's distance (5.5, its local one) lies before
    the box at 8 and its own entry at 11 behind it."""
    box = pb.AABox((2.0, 2.0, 2.0))
    objects = [pb.Transformed(pb.Simple(box), TR.translation([1.0, -20.0, 0.0])),
               pb.Transformed(pb.Simple(pb.Sphere(1.0)), TR.translation([13.0, -0.1, 0.0]) * _scaling(2, 2, 2)),
               pb.Transformed(pb.Simple(box), TR.translation([9.0, 0.1, 0.0])),
               pb.Transformed(pb.Simple(box), TR.translation([3.0, 20.0, 0.0]))]
    rng = np.random.default_rng(5)
    d = np.concatenate([np.ones((1, 4000)), rng.normal(size=(2, 4000)) * 0.02])
    rays = np.zeros((8, 4000), np.float32)
    rays[3:6], rays[7] = W.normalize_f32(d.astype(np.float32)), 1e30
    hit, t = _same(_commit(objects), rays)
    assert (t[hit] < 7).any()


@pytest.mark.parametrize("scale", [0.25, 0.9, 1.1, 8.0])
def test_directions_that_are_not_unit_vectors(scale):
    rng = np.random.default_rng(7)
    objects, at = _analytic(rng)
    rays = _rays(rng, 100_000, 3.0, at)
    rays[3:6] *= np.float32(scale)
    _same(_commit(objects + [pb.Simple(pb.TriangleMesh(*W.displaced_icosphere(3, seed=9)))]), rays)


def _towards(rng, tgt, dist):
    """Rays of a set length from random directions to the points `tgt` (n, 3)."""
    o = rng.normal(size=tgt.shape)
    o = tgt + o / np.linalg.norm(o, axis=1, keepdims=True) * dist
    r = np.empty((8, len(tgt)), np.float32)
    r[0:3] = o.T.astype(np.float32)
    r[3:6], r[6], r[7] = W.normalize_f32((tgt.T - r[0:3].astype(np.float64)).astype(np.float32)), 0.0, 1e30
    return r


@pytest.mark.parametrize("ratio", [1e-3, 1e-4, 1e-5])
def test_small_spheres_far_away(ratio):
    """A sphere's distance loses as many digits as the sphere is far in its radii: hits before their boxes."""
    rng = np.random.default_rng(11)
    c, r = rng.normal(size=(400, 3)) * 8 * ratio, ratio * 10 ** rng.uniform(-0.5, 0.5, 400)
    s = _commit([pb.Transformed(pb.Simple(pb.Sphere(float(q))), TR.translation([float(x) for x in p])) for p, q in zip(c, r)])
    n = 2_000_000
    tgt = c[rng.integers(0, 400, n)] + rng.normal(size=(n, 3)) * ratio
    hit, _ = _same(s, _towards(rng, tgt, rng.uniform(0.5, 1.5, (n, 1))))
    assert hit.mean() > 0.5


def _sheet(n, half, turn, lift):
    g = np.linspace(-half, half, n + 1)
    x, z = np.meshgrid(g, g, indexing="ij")
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    a = (i * (n + 1) + j).reshape(-1)
    f = np.stack([a, a + n + 1, a + n + 2, a, a + n + 2, a + 1], -1).reshape(-1, 3)
    v = np.stack([x, np.full_like(x, lift), z], -1).reshape(-1, 3) @ turn.T
    return v.astype(np.float32), f.astype(np.uint32)


def _grazing(rng, n, turn, half, least):
    """Rays that meet the plane y = 0 (turned) at angles down to `least`."""
    at = rng.uniform(-half, half, (3, n))
    at[1] = 0
    phi, c = rng.uniform(0, 2 * np.pi, n), 10 ** rng.uniform(np.log10(least), -1, n) * rng.choice([-1, 1], n)
    d = np.stack([np.cos(phi) * np.sqrt(1 - c * c), c, np.sin(phi) * np.sqrt(1 - c * c)])
    r = np.empty((8, n), np.float32)
    r[0:3] = turn @ (at - d * (0.01 + 8 * rng.random(n) ** 2))
    r[3:6], r[6], r[7] = W.normalize_f32((turn @ d).astype(np.float32)), 0.0, np.where(rng.random(n) < 0.2, np.inf, 1e30)
    return r


@pytest.mark.parametrize("merged", ["one mesh", "a mesh each", "instances"])
@pytest.mark.parametrize("seed", [0, 1])
def test_sheets_met_at_grazing_angles(merged, seed):
    """Sheets in nearly the same tilted plane: a triangle's distance is off by 2^-24 over the cosine, so that
    which sheet is met first, and whether before its box, is left to rounding and the order."""
    rng = np.random.default_rng(seed)
    turn = (TR.rotation_x(rng.uniform(0, 3)) * TR.rotation_z(rng.uniform(0, 3))).mat[:3, :3]
    sheets = [_sheet(12 + k, 2.0, turn, 1e-7 * rng.normal()) for k in range(8)]
    if merged == "one mesh":
        base = np.cumsum([0] + [len(v) for v, _ in sheets])
        objects = [pb.Simple(pb.TriangleMesh(np.concatenate([v for v, _ in sheets]),
                                             np.concatenate([f + b for (_, f), b in zip(sheets, base)]).astype(np.uint32)))]
    elif merged == "a mesh each":
        objects = [pb.Simple(pb.TriangleMesh(v, f)) for v, f in sheets]
    else:
        sheet = pb.TriangleMesh(*_sheet(6, 1.0, turn, 0.0))
        objects = [pb.Transformed(pb.Simple(sheet), TR.translation([float(x) for x in turn @ [a, 0, b]]))
                   for a, b in rng.uniform(-2, 2, (16, 2))]
    s = _commit(objects, bvh_bins=16)
    for _ in range(6):
        hit, _ = _same(s, _grazing(rng, 2_000_000, turn, 2.0, 1e-5))
        assert hit.mean() > 0.3


def _call(ctx, s, rays, out):
    """One asynchronous query on the context's stream: nearest hits into (prim, t, obj) or occlusion into (occ,)."""
    n = rays.shape[1]
    if len(out) == 1:
        ctx.check(ctx.lib.pbrt_trace_any(s.h, rays.data_ptr(), n, out[0].data_ptr()), "any")
    else:
        ctx.check(ctx.lib.pbrt_trace_closest(s.h, rays.data_ptr(), n, *[x.data_ptr() for x in out]), "closest")


def _outputs(n, kind):
    if kind == "any":
        return (torch.full((n,), 7, dtype=torch.uint8, device="cuda"),)
    return (torch.full((n,), 7, dtype=torch.int32, device="cuda"), torch.full((n,), 7.0, device="cuda"),
            torch.full((n,), 7, dtype=torch.int32, device="cuda"))


@pytest.mark.parametrize("n", [(1 << 18) + 1, 600_000, (1 << 24) + 300_001])
def test_captured_calls_use_nothing_shared(n):
    """Nearest hits and occlusion of more rays than one small kernel takes, recorded into graphs, replayed
    on one stream while eager calls of other rays run on another: each its own answers, every time."""
    v, f = W.displaced_icosphere(5, seed=4)
    ctx = pb.Context(0)
    s = pb.Scene(ctx).add_object(pb.Simple(pb.TriangleMesh(v, f))).commit(bvh_bins=16, bvh_max_leaf=4)
    base = [W.incoherent_rays(600_000, v.min(0), v.max(0), seed=k) for k in (5, 6)]
    mine = torch.from_numpy(base[0]).cuda()[:, torch.arange(n, device="cuda") % 600_000].contiguous()
    other = torch.from_numpy(base[1]).cuda()
    torch.cuda.synchronize()
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    want = {}
    for kind in ("closest", "any"):
        for name, rays in (("mine", mine), ("other", other)):
            want[kind, name] = [x.clone() for x in (s.intersect(rays, with_object=True) if kind == "closest" else
                                                    [s.intersect_p(rays)])]
    for kind in ("closest", "any"):
        out = _outputs(n, kind)
        torch.cuda.synchronize()
        ctx.set_stream(first.cuda_stream)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=first):
            _call(ctx, s, mine, out)
        ctx.set_stream(second.cuda_stream)
        for eager in ("any", "closest"):
            for _ in range(3):
                for x in out:
                    x.fill_(7)
                beside = _outputs(600_000, eager)
                torch.cuda.synchronize()
                with torch.cuda.stream(first):
                    g.replay()
                _call(ctx, s, other, beside)
                torch.cuda.synchronize()
                assert all(torch.equal(a, b) for a, b in zip(out, want[kind, "mine"]))
                assert all(torch.equal(a, b) for a, b in zip(beside, want[eager, "other"]))
        ctx.set_stream(None)
        del g


def test_survivor_queue_across_streams_that_come_and_go():
    """Asynchronous calls on streams that are destroyed while their work runs: a new stream, which may have
    an old one's handle, waits for that work's use of the survivor queue all the same."""
    import ctypes

    import torch.cuda

    rt = torch.cuda.cudart()
    v, f = W.displaced_icosphere(5, seed=4)
    ctx = pb.Context(0)
    s = pb.Scene(ctx).add_object(pb.Simple(pb.TriangleMesh(v, f))).commit(bvh_bins=16, bvh_max_leaf=4)
    n = 1_500_000
    rays = [torch.from_numpy(W.incoherent_rays(n, v.min(0), v.max(0), seed=k)).cuda() for k in (5, 6)]
    torch.cuda.synchronize()
    want = [s.intersect(r, with_object=True) for r in rays]
    for _ in range(6):
        outs = [_outputs(n, "closest") for _ in rays]
        torch.cuda.synchronize()
        for r, out in zip(rays, outs):
            st = ctypes.c_void_p()
            assert int(rt.cudaStreamCreate(ctypes.addressof(st))) == 0
            ctx.set_stream(st.value)
            _call(ctx, s, r, out)
            ctx.set_stream(None)
            assert int(rt.cudaStreamDestroy(st.value)) == 0
        torch.cuda.synchronize()
        for out, w in zip(outs, want):
            assert all(torch.equal(a, b) for a, b in zip(out, w))


def test_scenes_and_caches_destroyed_while_another_thread_captures():
    """A thread that destroys a scene and a cache leaves another thread's capture alone."""
    import threading

    from pbrt_b200.cache import RadianceCache

    v, f = W.displaced_icosphere(4, seed=4)
    scene = pb.Scene(pb.Context(0)).add_object(pb.Simple(pb.TriangleMesh(v, f))).commit()
    other = pb.Context(0)
    doomed = pb.Scene(other).add_object(pb.Simple(pb.TriangleMesh(v, f))).commit()
    cache = RadianceCache((0.0,) * 3, (1.0,) * 3, ctx=other)
    rays = torch.from_numpy(W.incoherent_rays(5000, v.min(0), v.max(0), seed=3)).cuda()
    torch.cuda.synchronize()
    want = scene.intersect(rays, with_object=True)
    out, st, g = _outputs(5000, "closest"), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    scene.ctx.set_stream(st.cuda_stream)
    with torch.cuda.graph(g, stream=st, capture_error_mode="thread_local"):
        _call(scene.ctx, scene, rays, out)
        t = threading.Thread(target=lambda: (doomed.release(), cache.close()))
        t.start()
        t.join()
    scene.ctx.set_stream(None)
    g.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(out, want))


@pytest.mark.parametrize("n", [1000, 300_000])
def test_occlusion_at_an_infinite_distance(n):
    """A short direction puts a hit's parameter beyond the largest float: it lies within [tmin, inf]."""
    v = np.array([[-1, -1, 1], [1, -1, 1], [0, 1, 1]], np.float32) * np.float32(1e15)
    s = _commit([pb.Simple(pb.TriangleMesh(v, np.array([[0, 1, 2]], np.uint32)))])
    rng = np.random.default_rng(3)
    base = np.zeros((8, 1000), np.float32)
    base[0:2] = rng.uniform(-1e14, 1e14, (2, 1000))
    base[5] = 10.0 ** rng.uniform(-30, -15, 1000)
    base[7] = np.where(rng.random(1000) < 0.5, np.inf, 1e30)
    r = np.ascontiguousarray(base[:, np.arange(n) % 1000])
    want, _ = s.intersect_p_counted(r)
    assert np.array_equal(s.intersect_p(r), want)
    assert np.array_equal(s.intersect_p(torch.from_numpy(r).cuda()).cpu().numpy(), want)
    assert 0 < want.sum() < n and want[np.isinf(r[7]) & (r[5] < 1e-24)].any()


def test_intervals_that_are_not_numbers_among_objects():
    rng = np.random.default_rng(9)
    objects, at = _analytic(rng)
    objects = objects + [pb.Simple(pb.TriangleMesh(*W.displaced_icosphere(3, seed=9)))]
    plane = [pb.Transformed(pb.Simple(pb.Plane()), TR.translation([0.0, -2.0, 0.0]))]
    for scene in (objects, objects + plane, [pb.Simple(pb.Sphere(1.0))]):
        rays = _rays(rng, 24_000, 3.0, at)
        for k, (row, x) in enumerate([(6, np.nan), (7, np.nan), (7, np.inf), (7, -np.inf), (6, np.inf), (6, -np.inf),
                                      (7, -1.0), (7, 0.0)]):
            rays[row, k::8] = x
        _same(_commit(scene), rays)


@pytest.mark.parametrize("device_build", [False, True])
@pytest.mark.parametrize("leaf", [1, 4])
def test_memory_of_a_mesh(device_build, leaf):
    """A mesh's device memory: 58 bytes of arrays and 8 of leaf notes a triangle, 32 a node, and 192 a wide
    node, of which no interior node of every second level has one."""
    v, f = W.displaced_icosphere(6, seed=4)
    s = _commit([pb.Simple(pb.TriangleMesh(v, f))], device_build=device_build, bvh_bins=16, bvh_max_leaf=leaf)
    i = s.info()
    interior = i["mesh_node_count"] - i["mesh_leaf_count"]
    wide = i["device_bytes"] - 66 * len(f) - 32 * i["mesh_node_count"]
    assert wide < 192 * interior * 0.7, f"{wide / interior:.0f} bytes an interior node"


def test_films_by_the_walk_and_by_the_per_object_queries():
    """A render's queries walk the wide tree; a persistent batch asks the top level and each object's own
    tree, one thread per path: the same film, of objects of every kind, a large mesh among them."""
    rng = np.random.default_rng(4)
    objects, at = _unordered(rng)
    objects += _analytic(rng)[0] + [pb.Simple(pb.TriangleMesh(*W.displaced_icosphere(5, seed=9)))]
    ctx = pb.Context(0)
    s = pb.Scene(ctx)
    for o in objects:
        s.add_object(o)
    s.add_light(pb.BackgroundInfiniteLight([1.0, 1.0, 1.0], [0.5, 0.7, 1.0]))
    s.add_light(pb.PointLight([0.0, 8.0, 0.0], [40.0, 40.0, 40.0]))
    s.commit()
    _, cam = W.many_spheres(10, width=128, height=96)
    film = s.render(cam, 8, 8, seed=3, rr_start=4)
    ctx.set_batch_kernel("persistent")
    try:
        b = Batch([s], [render_params(cam, 8, 8, seed=3, rr_start=4)], ctx)
        other = b.render(0)[0]
    finally:
        ctx.set_batch_kernel("wavefront")
    np.testing.assert_array_equal(film, other)
    assert film.std() > 0.01
