"""Children of one tree node whose distances differ by few units in the last
place.  Rays along +x from x = -1 meet stacks of triangles at x = a units in
the last place of 1, the two halves of one square in random order: each
triangle's box covers the square, so a child that is entered first need not be
hit first.  The arithmetic has no rounding (all edges are powers of two, all
offsets exact), so the answer is known: the smallest distance among the
triangles on the ray's side of the square's diagonal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ULP = 2.0 ** -23  # of the distances in [1, 2)
STACKS = 64


def stacks_mesh(a, half):
    """a, half: (STACKS, height)"""
    from lambda_b200.scene import TriMeshData
    corners = np.array([[[-8, -8], [8, -8], [-8, 8]], [[8, 8], [-8, 8], [8, -8]]], np.float64)
    V = np.zeros(a.shape + (3, 3))
    V[..., 0] = a[..., None] * ULP
    V[..., 1:] = corners[half]
    V[..., 1] += 32.0 * np.arange(STACKS)[:, None, None]
    n = a.size
    F = np.concatenate([1 + np.arange(3 * n).reshape(n, 3), np.ones((n, 3), int)], axis=1)
    return TriMeshData("stacks", np.concatenate([np.zeros((1, 3)), V.reshape(-1, 3)]),
                       np.array([[0, 0, 1], [1, 0, 0]]), F)


# heights of one node's children and of two levels; distances within and beyond
# what a bound kept with a mask of children can resolve
@pytest.mark.parametrize("height", [3, 8, 16, 21, 40])
@pytest.mark.parametrize("spread", [12, 60, 120, 400])
def test_nearest_of_near_equal(height, spread):
    from lambda_b200.renderer import Context
    from lambda_b200.scene import (Camera, FlatScene, LightDef, Material, Object, SceneData, SpectralConfig,
                                   Transform)
    rng = np.random.default_rng([height, spread])
    cfg = SpectralConfig(hero_k=4)
    sc = SceneData(cfg)
    sc.cam = Camera([0, 0, 3], [0, 0, 0], [0, 1, 0], 16, 40, 1.0)
    sc.materials.append(Material("lambertian", "m", albedo=np.full(cfg.n_bins, 0.5, np.float32)))
    sc.lights.append(LightDef("point", "l", radiance=np.ones(cfg.n_bins, np.float32), pos=[0, 0, 2]))
    # six objects, so that the instance BVH is used; only the first is met
    for k in range(6):
        sc.objects.append(Object("trimesh" if k == 0 else "sphere", "o", Transform.translate([0, 0, -100.0 * k]), 0, k))
    ctx = Context(0)
    wrong = []
    for _ in range(6):
        a, half = rng.integers(0, spread, (STACKS, height)), rng.integers(0, 2, (STACKS, height))
        half[:, :2] = [0, 1]
        sc.meshes = [stacks_mesh(a, half)]
        ctx.upload(FlatScene(sc))
        yz = rng.integers(-500, 500, (STACKS, 16, 2)) / 128
        yz[yz.sum(-1) == 0] = 1.0
        p = np.zeros((STACKS, 16, 6), np.float32)
        p[..., 0], p[..., 3] = -1, 1
        p[..., 1:3] = yz
        p[..., 1] += 32.0 * np.arange(STACKS)[:, None]
        got = ctx.trace(p.reshape(-1, 6)).reshape(STACKS, 16)
        side = (yz.sum(-1) > 0).astype(int)
        want = np.where(half[:, None, :] == side[:, :, None], a[:, None, :], 1 << 20).min(-1)
        bad = np.argwhere((got["t"] != (1 + want * ULP).astype(np.float32)) | (got["obj"] != 0))
        wrong += [(int(j), int(k), int(want[j, k]), (float(got["t"][j, k]) - 1) / ULP) for j, k in bad]
    ctx.close()
    assert not wrong, (len(wrong), wrong[:5])
