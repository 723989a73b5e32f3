"""The adjoint's shading launches by material put each gradient where it
belongs.  A material that no object uses takes a scene from one launch for all
paths to the launches over lists without changing any path, so every entry of
the gradients has to be the same but for the order of its sum, and the unused
material's entries have to be zero."""
import json
import os

import numpy as np
import pytest

from lambda_b200 import synth

pytestmark = pytest.mark.gpu

EXTRA = {"blinn": {"name": "extra", "type": "blinn", "Kd": {"val": 0.5}},
         "thinfilm": {"name": "extra", "type": "thinfilm", "film_ior": {"val": 1.4}}}


@pytest.mark.parametrize("width", [1, 16, 17, 45])
@pytest.mark.parametrize("extra", ["blinn", "thinfilm"])
def test_entry_by_entry(tmp_path, width, extra):
    from lambda_b200.renderer import Context
    from lambda_b200.scene import load_nls
    nls = synth.box_room(str(tmp_path), width=width)
    with open(nls) as f:
        j = json.load(f)
    got = []
    for name in ("none", extra):
        path = os.path.join(str(tmp_path), name + ".nls")
        with open(path, "w") as f:
            json.dump(dict(j, materials=j["materials"] + ([EXTRA[name]] if name in EXTRA else [])), f)
        ctx = Context(0)
        flat = ctx.upload(load_nls(path))
        w, h = ctx.size
        d = np.random.default_rng(1).normal(size=(h, w, 3)).astype(np.float32)
        got.append(ctx.adjoint(5, 6, 0.85, d, seed=4, image=True) + (flat,))
        ctx.close()
    (gs0, gm0, im0, flat0), (gs1, gm1, im1, flat1) = got
    assert np.array_equal(im0.view(np.uint32), im1.view(np.uint32))
    # the unused material and its spectra lie before the emitters' and lights'
    assert int(flat1.scene.n_materials) == int(flat0.scene.n_materials) + 1
    x = [m.name for m in flat1.sc.materials].index("extra")
    own = [s for s in flat1.materials[x].spectrum if s >= 0]
    assert own and np.all(gs1[own] == 0) and np.all(gm1[x] == 0)
    gs1, gm1 = np.delete(gs1, own, axis=0), np.delete(gm1, x, axis=0)
    assert gm0.shape == gm1.shape
    assert gs0.shape == gs1.shape
    assert width == 1 or np.any(gs0 != 0)
    # each entry is a sum of at most N = pixels x samples x vertices x hero
    # wavelengths float terms in any order, whose rounding is a random walk of
    # at most sqrt(N) steps of 2^-24 of the largest partial sum; that is at
    # most the norm of the array here (terms of both signs: a few times)
    n = 5 * w * h * 7 * 16
    for a, b in ((gs0, gs1), (gm0, gm1)):
        a, b = a.astype(np.float64), b.astype(np.float64)
        assert np.all(np.isfinite(a)) and np.all(np.isfinite(b))
        assert np.abs(a - b).max() <= 4 * np.sqrt(n) * 2.0 ** -24 * np.linalg.norm(a)
        assert np.array_equal(a != 0, b != 0)
