"""The wide walk (wide_bvh.cuh) against the binary tree's: ids, t and occlusion bit for bit.

The instrumented nearest-hit query walks the binary nodes one thread per ray; every other
query walks the wide ones. The meshes and rays here are those where a conservative walk with
another visiting order could differ: leaves that share a distance (overlapping sheets), leaves
of more triangles than a packed reference holds, coordinates and directions of any scale, rays
along the axes, empty and NaN intervals."""
import numpy as np
import pytest
import torch

import oracle
import pbrt_b200 as pb
from pbrt_b200 import workloads as W
from pbrt_b200.scene import Batch, render_params

pytestmark = pytest.mark.gpu


def _one():
    return np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]], np.float32), np.array([[0, 1, 2]], np.uint32)


def _stacked():  # 40 copies of one triangle: inseparable, one leaf of 40
    v, f = _one()
    return v, np.repeat(f, 40, 0)


def _sheets():  # the same plane tessellated twice on different grids: equal distances in different leaves
    vs, fs, base = [], [], 0
    for n in (7, 10):
        g = np.linspace(-1, 1, n + 1)
        x, y = np.meshgrid(g, g, indexing="ij")
        vs.append(np.stack([x, y, np.zeros_like(x)], -1).reshape(-1, 3))
        i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
        a = (i * (n + 1) + j).reshape(-1)
        quad = np.stack([a, a + n + 1, a + n + 2, a, a + n + 2, a + 1], -1).reshape(-1, 3)
        fs.append(quad + base)
        base += (n + 1) ** 2
    return np.concatenate(vs).astype(np.float32), np.concatenate(fs).astype(np.uint32)


def _ball(scale, shift):
    v, f = W.displaced_icosphere(4, seed=9)
    return (v * np.float32(scale) + np.float32(shift)).astype(np.float32), f


_MESHES = {
    "one triangle": _one, "stacked": _stacked, "sheets": _sheets, "ball": lambda: _ball(1, 0),
    "tiny": lambda: _ball(1e-6, 0), "huge": lambda: _ball(1e9, 0), "far off": lambda: _ball(1e-2, 100),
    "beyond the grid": lambda: _ball(1e13, 0),
}


def _rays(v, f, seed):
    rng = np.random.default_rng(seed)
    lo, hi = v.min(0).astype(np.float64), v.max(0).astype(np.float64)
    size = max(float((hi - lo).max()), 1e-30)
    n = 4000
    r = W.incoherent_rays(n, lo, hi, seed=seed, near=0.0)
    # aimed at vertices, edge midpoints and interiors, from near and far
    p = v[f[rng.integers(0, f.shape[0], n)]].astype(np.float64)
    w = rng.choice([0.0, 0.5, 1.0, 0.3], size=(n, 3)) + 1e-12
    tgt = (p * (w / w.sum(1, keepdims=True))[..., None]).sum(1)
    org = tgt + rng.normal(size=(n, 3)) * size * 10.0 ** rng.uniform(-2, 3, (n, 1))
    aim = r.copy()
    aim[0:3] = org.T.astype(np.float32)
    d = tgt - aim[0:3].T.astype(np.float64)
    aim[3:6] = W.normalize_f32((d / np.abs(d).max(1, keepdims=True)).T.astype(np.float32))
    flat = aim[:, : n // 2].copy()  # along one or two axes
    axis = rng.integers(0, 3, flat.shape[1])
    flat[3 + axis, np.arange(flat.shape[1])] = np.where(rng.random(flat.shape[1]) < 0.5, 0.0, -0.0)
    half = flat[:, ::2].copy()
    k = rng.integers(0, 3, half.shape[1])
    half[3:6] = 0
    half[3 + k, np.arange(half.shape[1])] = rng.choice([1.0, -1.0], half.shape[1])
    slow = aim[:, : n // 4].copy()  # unnormalised directions
    slow[3:6] *= (10.0 ** rng.uniform(-14, 14, slow.shape[1])).astype(np.float32)
    cut = aim[:, : n // 4].copy()  # intervals that end near the surface, or are empty, or start below 0
    dist = np.linalg.norm(d, axis=1)[: n // 4]
    cut[6] = rng.choice([0.0, -1.0, 1e-4], cut.shape[1])
    cut[7] = dist * rng.choice([0.0, -1.0, 0.5, 1.0, 1.0000001, 0.9999999], cut.shape[1])
    out = np.concatenate([r, aim, flat, half, slow, cut], axis=1).astype(np.float32)
    out[7, ::7] = np.float32(3.4028235e38)
    return np.ascontiguousarray(out)


@pytest.mark.parametrize("bins,max_leaf", [(8, 1), (16, 4)])
@pytest.mark.parametrize("mesh", list(_MESHES))
def test_wide_equals_binary(mesh, bins, max_leaf):
    v, f = _MESHES[mesh]()
    rays = _rays(v, f, seed=len(mesh))
    s = pb.Scene().add_object(pb.Simple(pb.TriangleMesh(v, f))).commit(bvh_bins=bins, bvh_max_leaf=max_leaf)
    for n in (rays.shape[1], rays.shape[1] - 3, 1):  # planes aligned for bulk copies, or not
        r = np.ascontiguousarray(rays[:, :n])
        bp, bt, _ = s.intersect_instrumented(r)
        for got in (s.intersect(r), [x.cpu().numpy() for x in s.intersect(torch.from_numpy(r).cuda())]):
            assert np.array_equal(got[0].view(np.uint32), bp), f"{(got[0].view(np.uint32) != bp).sum()} ids differ"
            assert np.array_equal(got[1], bt)
        occ = oracle.MeshBVH(v, f, np.float32, bins=bins, max_leaf=max_leaf).occluded(r)
        assert np.array_equal(s.intersect_p(r), occ)
        assert np.array_equal(s.intersect_p(torch.from_numpy(r).cuda()).cpu().numpy(), occ)
    if mesh == "ball":
        assert (bp != pb.PBRT_MISS).any() or n == 1


def test_intervals_that_are_not_numbers():
    v, f = _ball(1, 0)
    s = pb.Scene().add_object(pb.Simple(pb.TriangleMesh(v, f))).commit()
    rays = np.repeat(W.incoherent_rays(512, v.min(0), v.max(0), seed=3), 6, axis=1)
    for k, (row, x) in enumerate([(6, np.nan), (7, np.nan), (7, np.inf), (7, -np.inf), (6, np.inf), (0, np.nan)]):
        rays[row, k::6] = x
    bp, bt, _ = s.intersect_instrumented(rays)
    wp, wt = s.intersect(rays)
    assert np.array_equal(wp, bp) and np.array_equal(wt, bt)
    assert np.array_equal(s.intersect_p(rays) != 0, (bp != pb.PBRT_MISS))


def test_occlusion_under_capture_and_on_several_streams():
    """A captured occlusion query replays to the same answers; asynchronous queries on changing
    streams do not disturb one another's survivor queue."""
    v, f = W.displaced_icosphere(5, seed=4)
    ctx = pb.Context(0)
    s = pb.Scene(ctx).add_object(pb.Simple(pb.TriangleMesh(v, f))).commit(bvh_bins=16, bvh_max_leaf=4)
    r = [torch.from_numpy(W.incoherent_rays(200_000, v.min(0), v.max(0), seed=k)).cuda() for k in (5, 6)]
    want = [(s.intersect(x), s.intersect_p(x)) for x in r]
    st = [torch.cuda.Stream() for _ in r]
    n = r[0].shape[1]
    for _ in range(5):
        got = []
        for x, q in zip(r, st):
            ctx.set_stream(q.cuda_stream)
            prim = torch.zeros(n, dtype=torch.int32, device="cuda")
            t = torch.zeros(n, device="cuda")
            occ = torch.zeros(n, dtype=torch.uint8, device="cuda")
            q.wait_stream(torch.cuda.current_stream())
            ctx.check(ctx.lib.pbrt_trace_any(s.h, x.data_ptr(), n, occ.data_ptr()), "any")
            ctx.check(ctx.lib.pbrt_trace_closest(s.h, x.data_ptr(), n, prim.data_ptr(), t.data_ptr(), None), "closest")
            got.append((prim, t, occ))
        torch.cuda.synchronize()
        for (prim, t, occ), ((p0, t0), o0) in zip(got, want):
            assert torch.equal(prim, p0) and torch.equal(t, t0) and torch.equal(occ, o0)
    occ = torch.zeros(n, dtype=torch.uint8, device="cuda")
    ctx.set_stream(st[0].cuda_stream)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st[0]):
        ctx.check(ctx.lib.pbrt_trace_any(s.h, r[0].data_ptr(), n, occ.data_ptr()), "any")
    ctx.set_stream(None)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(occ, want[0][1])


@pytest.mark.parametrize("n", [1, 7, 8, 9, 33, 4099, (1 << 15) - 1, 1 << 15, (1 << 15) + 1, 1 << 18, (1 << 18) + 1])
def test_few_and_many_rays(n):
    """Host and device calls around the sizes where the staging, the rays per warp and the kernels
    change: the binary query's answers, object ids, and occlusion from the same hits."""
    for v, f in (_ball(1, 0), _sheets()):
        base = _rays(v, f, seed=17)
        r = np.ascontiguousarray(base[:, np.arange(n) % base.shape[1]])
        s = pb.Scene().add_object(pb.Simple(pb.TriangleMesh(v, f))).commit(bvh_bins=16, bvh_max_leaf=4)
        bp, bt, _ = s.intersect_instrumented(r)
        for rays in (r, torch.from_numpy(r).cuda()):
            p, t, o = [x if isinstance(x, np.ndarray) else x.cpu().numpy() for x in s.intersect(rays, with_object=True)]
            assert np.array_equal(p.view(np.uint32), bp) and np.array_equal(t, bt)
            assert np.array_equal(o.view(np.uint32), np.where(bp == pb.PBRT_MISS, pb.PBRT_MISS, 0).astype(np.uint32))
        occ = oracle.MeshBVH(v, f, np.float32, bins=16, max_leaf=4).occluded(base)[np.arange(n) % base.shape[1]]
        assert np.array_equal(s.intersect_p(r), occ)
        assert np.array_equal(s.intersect_p(torch.from_numpy(r).cuda()).cpu().numpy(), occ)


def test_survivor_queue_on_several_streams():
    """Asynchronous calls of more rays than one kernel takes, on changing streams."""
    v, f = W.displaced_icosphere(5, seed=4)
    ctx = pb.Context(0)
    s = pb.Scene(ctx).add_object(pb.Simple(pb.TriangleMesh(v, f))).commit(bvh_bins=16, bvh_max_leaf=4)
    n = 600_000
    r = [torch.from_numpy(W.incoherent_rays(n, v.min(0), v.max(0), seed=k)).cuda() for k in (5, 6)]
    want = [(s.intersect(x), s.intersect_p(x)) for x in r]
    st = [torch.cuda.Stream() for _ in r]
    for _ in range(4):
        got = []
        for x, q in zip(r, st):
            ctx.set_stream(q.cuda_stream)
            prim, t = torch.zeros(n, dtype=torch.int32, device="cuda"), torch.zeros(n, device="cuda")
            occ = torch.zeros(n, dtype=torch.uint8, device="cuda")
            q.wait_stream(torch.cuda.current_stream())
            ctx.check(ctx.lib.pbrt_trace_any(s.h, x.data_ptr(), n, occ.data_ptr()), "any")
            ctx.check(ctx.lib.pbrt_trace_closest(s.h, x.data_ptr(), n, prim.data_ptr(), t.data_ptr(), None), "closest")
            got.append((prim, t, occ))
        torch.cuda.synchronize()
        for (prim, t, occ), ((p0, t0), o0) in zip(got, want):
            assert torch.equal(prim, p0) and torch.equal(t, t0) and torch.equal(occ, o0)
    ctx.set_stream(None)


def _mixed_scene():
    """Meshes merged into the wide tree, one placed twice, coplanar sheets in different objects,
    transformed instances, analytic shapes, a compound, a solid and an unbounded plane."""
    v, f = _ball(1, 0)
    ball = pb.TriangleMesh(v, f)
    sv, sf = _sheets()
    sheet = pb.TriangleMesh(sv * np.float32(3) + np.float32([0, 0, 2]), sf)
    again = pb.TriangleMesh(sv * np.float32(2) + np.float32([0.5, 0, 2]), sf[:, ::-1])
    tr = pb.Transform
    s = pb.Scene()
    for o in (pb.Simple(ball), pb.Simple(ball), pb.Simple(sheet), pb.Simple(again),
              pb.Transformed(pb.Simple(ball), tr.translation([3.0, 1.0, 0.5]) * tr.rotation_x(0.4)),
              pb.Transformed(pb.Simple(pb.Sphere(0.7)), tr.translation([-2.0, 0.0, 0.0])),
              pb.Transformed(pb.Simple(pb.Sphere(0.7)), tr.translation([-2.0, 0.0, 0.0])),
              pb.Simple(pb.AABox((1.0, 5.0, 1.0))), pb.Transformed(pb.Simple(pb.Cylinder(0.4, 2.0)), tr.translation([0, 2.0, 1.0])),
              pb.Transformed(pb.Simple(pb.Rectangle(4.0, 4.0)), tr.translation([0.0, -1.5, 0.0])),
              pb.Compound([pb.Transformed(pb.Simple(pb.Sphere(0.5)), tr.translation([0.0, 0.0, 3.0])), pb.Simple(ball)]),
              pb.Simple(pb.Csg("subtraction", [(pb.Sphere(1.2), tr.translation([4.0, 0.0, 4.0])),
                                               (pb.AABox((1.0, 1.0, 4.0)), tr.translation([4.0, 0.0, 4.0]))])),
              pb.Transformed(pb.Simple(pb.Plane()), tr.translation([0.0, -2.0, 0.0]))):
        s.add_object(o)
    return s


def _only_meshes():
    s = pb.Scene()
    for k, (scale, shift) in enumerate([(1, 0), (0.5, 0.7), (1e-3, 0.2), (2, 0)]):
        s.add_object(pb.Simple(pb.TriangleMesh(*_ball(scale, shift))))
    s.add_object(pb.Simple(pb.TriangleMesh(*_sheets())))
    s.add_object(pb.Simple(pb.TriangleMesh(*_one())))
    return s


@pytest.mark.parametrize("build", [_mixed_scene, _only_meshes])
def test_scene_walk_equals_the_counted_queries(build):
    """Any scene's nearest hits and occlusion by the walk over its one wide tree against the
    counted queries, which take the binary trees one object at a time: the same objects,
    primitives and distances, equal distances between objects included."""
    s = build().commit()
    v = np.array([[-5, -3, -3], [5, 3, 5]], np.float32)
    rays = _rays(np.concatenate([v, _sheets()[0], _ball(1, 0)[0]]), np.arange(600, dtype=np.uint32).reshape(-1, 3), 17)
    for n in (rays.shape[1], 31, 1):
        r = np.ascontiguousarray(rays[:, :n])
        bp, bt, bo, _ = s.intersect_counted(r)
        wp, wt, wo = s.intersect(r, with_object=True)
        assert np.array_equal(wo, bo) and np.array_equal(wt, bt)
        hit = bo != pb.PBRT_MISS
        assert np.array_equal(wp[hit], bp[hit])
        bocc, _ = s.intersect_p_counted(r)
        assert np.array_equal(s.intersect_p(r), bocc)
    assert hit.any() or n == 1


def test_small_scenes_by_both_walks():
    """A closed box, whose waves of at most 786,432 paths run one thread per ray and larger ones
    persistently: the same film from one wave of 1.05 M paths as from waves of 2^18."""
    desc, cam = W.cornell_box(256, 256)
    films = []
    for wave in (1 << 18, 0):
        ctx = pb.Context(0)
        ctx.set_tuning(wave_paths=wave)
        ctx.set_batch_branches(1)
        scene = pb.Scene.from_description(desc, ctx).commit()
        b = Batch([scene], [render_params(cam, 16, 6, seed=5)], ctx)
        films += [b.render(0)[0], scene.render(cam, 16, 6, seed=5)]
    for f in films[1:]:
        np.testing.assert_array_equal(f, films[0])
