"""Rays whose answer depends on the reference's object order get exactly the
reference's answer.

Every ray starts inside the bounds of all objects of its scene, so whatever it
hits lies in a mesh that contains its origin, among several such meshes.  The
objects are axis-parallel rectangles, whose edges are edges of their boxes, and
the rays aim at points of these edges: there the rounded box tests of the
reference's trees reject triangles that the triangle test alone accepts, so a
search with other trees or wider box tests finds hits that the reference does
not.  The oracle is the same query in the reference's linear object order, and
everything it returns has to be equal."""
import numpy as np
import pytest

from lambda_b200 import _lib as L

pytestmark = pytest.mark.gpu


def rectangles(rng, n):
    """n rectangles across random axes inside the unit cube, as vertices and
    faces."""
    V, F = [], []
    for k in range(n):
        axis = int(rng.integers(0, 3))
        b, c = [(1, 2), (2, 0), (0, 1)][axis]
        lo = rng.uniform(0.02, 0.7, 2)
        hi = lo + rng.uniform(0.05, 0.28, 2)
        at = rng.uniform(0.02, 0.98)
        for y, z in ((lo[0], lo[1]), (hi[0], lo[1]), (hi[0], hi[1]), (lo[0], hi[1])):
            v = np.zeros(3)
            v[axis], v[b], v[c] = at, y, z
            V.append(v)
        F += [[4 * k, 4 * k + 1, 4 * k + 2], [4 * k, 4 * k + 2, 4 * k + 3]]
    return np.array(V, np.float32), np.array(F)


def scene_of(n_objects, n_meshes, per_mesh, seed):
    from lambda_b200.scene import (Camera, LightDef, Material, Object, SceneData, SpectralConfig, Transform,
                                   TriMeshData)
    rng = np.random.default_rng(seed)
    cfg = SpectralConfig(hero_k=4)
    sc = SceneData(cfg)
    sc.cam = Camera([0.5, -3, 0.5], [0.5, 0.5, 0.5], [0, 0, 1], 16, 40, 1.0)
    sc.materials.append(Material("lambertian", "m", albedo=np.full(cfg.n_bins, 0.5, np.float32)))
    sc.lights.append(LightDef("point", "l", radiance=np.ones(cfg.n_bins, np.float32), pos=[0, 0, 2]))
    corners = []
    for k in range(n_meshes):
        V, F = rectangles(rng, per_mesh)
        corners.append(V.reshape(-1, 4, 3))
        # the two corners of the unit cube are positions of every mesh, and so
        # in its bounds
        V = np.concatenate([np.zeros((1, 3)), V, np.ones((1, 3))])
        sc.meshes.append(TriMeshData("r%d" % k, V, np.array([[0, 0, 1], [0, 0, 1]]),
                                     np.concatenate([F + 1, np.ones_like(F)], axis=1)))
    for i in range(n_objects):
        sc.objects.append(Object("trimesh", "o%d" % i, Transform(), 0, i, i % n_meshes))
    return sc, np.concatenate(corners)


def edge_rays(corners, n, seed):
    """From points among the rectangles to points of their edges."""
    rng = np.random.default_rng(seed)
    r, e = rng.integers(0, len(corners), n), rng.integers(0, 4, n)
    s = rng.uniform(0, 1, (n, 1)).astype(np.float32)
    a, b = corners[r, e], corners[r, (e + 1) % 4]
    o = rng.uniform(0.3, 0.7, (n, 3)).astype(np.float32)
    d = (a + (b - a) * s).astype(np.float64) - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.concatenate([o, d.astype(np.float32)], axis=1)


# 6 and 40 objects: one and two groups of 32 in the object loop; 1024 and 1025:
# its largest scene in steps, and the smallest that always has a warp per ray,
# with meshes that several objects share, so that equal distances tie
@pytest.mark.parametrize("n_objects,n_meshes,per_mesh", [(6, 6, 6), (40, 40, 2), (1024, 8, 6), (1025, 8, 6)])
def test_equals_the_reference_order(n_objects, n_meshes, per_mesh):
    from lambda_b200.renderer import Context
    from lambda_b200.scene import FlatScene
    sc, corners = scene_of(n_objects, n_meshes, per_mesh, n_objects)
    ctx = Context(0)
    ctx.upload(FlatScene(sc))
    n = 200_003 if n_objects < 100 else 20_011
    rays = edge_rays(corners, n, 3)
    a = ctx.trace(rays)
    ordered = ctx.stats()["order_rays"]
    b = ctx.trace(rays, flags=L.FLAG_REFERENCE_ORDER)
    ctx.close()
    assert ordered > n // 10
    hit = b["obj"] != np.uint32(0xFFFFFFFF)
    assert 0.1 < hit.mean()
    bad = np.flatnonzero((a["t"].view(np.uint32) != b["t"].view(np.uint32)) | (a["obj"] != b["obj"]) |
                         (a["face"] != b["face"]))
    assert bad.size == 0, (bad.size, a[bad[:3]], b[bad[:3]])
    assert a.tobytes() == b.tobytes()


@pytest.mark.parametrize("n_objects,n_meshes,per_mesh", [(6, 6, 6), (40, 40, 2)])
def test_few_and_many_rays(n_objects, n_meshes, per_mesh):
    """Launches of few order-dependent rays (a warp each) and of 8192 and more
    (in steps): on both sides of the line, with single lanes and full warps."""
    from lambda_b200.renderer import Context
    from lambda_b200.scene import FlatScene
    sc, corners = scene_of(n_objects, n_meshes, per_mesh, n_objects)
    ctx = Context(0)
    ctx.upload(FlatScene(sc))
    rays = edge_rays(corners, 60_000, 4)
    b = ctx.trace(rays, flags=L.FLAG_REFERENCE_ORDER)
    ends = [1, 2, 33, 1000]
    for want in (8191, 8192, 8193, 14207, 14208):
        lo, hi = 0, len(rays)  # the number of order-dependent rays grows with the number of rays
        while lo < hi:
            m = (lo + hi) // 2
            ctx.trace(rays[:m])
            lo, hi = (m + 1, hi) if ctx.stats()["order_rays"] < want else (lo, m)
        ctx.trace(rays[:lo])
        assert ctx.stats()["order_rays"] == want
        ends.append(lo)
    for n in ends + [len(rays)]:
        a = ctx.trace(rays[:n])
        assert a.tobytes() == b[:n].tobytes(), n
    ctx.close()
