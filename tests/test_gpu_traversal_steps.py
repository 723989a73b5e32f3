"""The persistent traversal kernels at the sizes where their warp-wide steps
change path: ray counts around a warp and a block, scenes whose nodes have
many hit children (group entries on the stack), objects entered from inside,
and lanes that finish at very different times.  The oracle is the same query
in the reference's linear object order (LGPU_FLAG_REFERENCE_ORDER), which
shares neither the step loop nor the trees."""
import os

import numpy as np
import pytest

from lambda_b200 import _lib as L
from lambda_b200 import synth

pytestmark = pytest.mark.gpu

MISS = np.uint32(0xFFFFFFFF)


def crowded(out_dir, n):
    """n heavily overlapping instances around the origin: rays cross many
    bounds at every level."""
    import json
    path = synth.instanced(out_dir, n_instances=n, subdiv=3, width=64)
    with open(path) as f:
        sc = json.load(f)
    rng = np.random.default_rng(5)
    for o in sc["objects"][1:]:
        s = float(rng.uniform(0.3, 1.4)) * (1.0 if n < 100 else 0.25)
        o["transform"] = {"scale": [s, s * float(rng.uniform(0.3, 1.0)), s],
                          "rotate": {"axis": [float(x) for x in rng.normal(size=3)],
                                     "degrees": float(rng.uniform(0, 360))},
                          "translate": [float(x) for x in rng.uniform(-0.8, 0.8, 3)]}
    with open(path, "w") as f:
        json.dump(sc, f)
    return path


def rays_of(n, seed):
    rng = np.random.default_rng(seed)
    o = rng.normal(size=(n, 3)) * rng.choice([0.3, 1.0, 6.0], (n, 1))
    d = rng.normal(size=(n, 3))
    far = np.linalg.norm(o, axis=1) > 3
    d[far] = rng.uniform(-0.8, 0.8, (int(far.sum()), 3)) - o[far]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d[::17, int(rng.integers(0, 3))] = 0.0  # axis-parallel components
    return np.concatenate([o, d], axis=1).astype(np.float32)


# 5 and 40 objects: one and two groups of the in-kernel object loop; 1100: the
# separate launch for larger scenes
@pytest.fixture(scope="module", params=[5, 40, 1100])
def ctx(request, tmp_path_factory):
    from lambda_b200.renderer import Context
    from lambda_b200.scene import load_nls
    c = Context(0)
    c.upload(load_nls(crowded(os.path.join(str(tmp_path_factory.mktemp("crowd")), str(request.param)), request.param)))
    yield c
    c.close()


@pytest.mark.parametrize("n", [1, 11, 31, 32, 33, 127, 129, 5000, 200003])
def test_closest_and_any(ctx, n):
    rays = rays_of(n, n)
    a, b = ctx.trace(rays), ctx.trace(rays, flags=L.FLAG_REFERENCE_ORDER)
    assert np.array_equal(a["t"].view(np.uint32), b["t"].view(np.uint32))
    # another face of a shared edge may be reported at an exactly equal
    # distance (about one ray in a million)
    assert np.count_nonzero(a["obj"] != b["obj"]) + np.count_nonzero(a["face"] != b["face"]) <= n // 50000
    if n == 200003:
        assert ctx.stats()["device_checks"] == 0
        ctx.trace(rays)
        assert ctx.stats()["order_rays"] > 0  # the object loop was taken
    hit = a["obj"] != MISS
    assert n < 100 or 0.05 < hit.mean() < 0.95
    # shadow rays just short of, at and beyond the closest hit, and one that
    # skips the object found
    t = np.where(hit, a["t"], np.float32(10.0)).astype(np.float32)
    for scale, skip in ((0.5, MISS), (1.0, MISS), (1.5, MISS), (1.5, a["obj"])):
        x = ctx.trace_any(rays, t * np.float32(scale), skip)
        y = ctx.trace_any(rays, t * np.float32(scale), skip, flags=L.FLAG_REFERENCE_ORDER)
        assert np.array_equal(x, y), (scale, np.count_nonzero(x != y))
