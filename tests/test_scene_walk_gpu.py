"""Scene::intersect over mixed scenes by the walk of the wide tree (scene_walk.cuh) against the
counted queries, which take the binary trees one object at a time: the same objects, primitives and
distances where a walk in another order, or with another far end, could answer differently."""
import numpy as np
import pytest
import torch

import pbrt_b200 as pb
from pbrt_b200 import workloads as W

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
