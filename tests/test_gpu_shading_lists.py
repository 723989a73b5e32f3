"""Scenes with a Blinn or thin-film material shade their Lambertian and
unshaded hits from a list, others in place.  A material that no object uses
takes a scene from one way to the other without changing any path, so the two
images have to be the same, bit for bit."""
import json
import os

import numpy as np
import pytest

from lambda_b200 import synth

pytestmark = pytest.mark.gpu

EXTRA = {"blinn": {"name": "extra", "type": "blinn", "Kd": {"val": 0.5}},
         "thinfilm": {"name": "extra", "type": "thinfilm", "film_ior": {"val": 1.4}}}


@pytest.fixture(scope="module")
def scenes(tmp_path_factory):
    """(width, unshaded left wall) -> the scene's three files."""
    out = {}
    for width in (1, 16, 17, 45):
        for unshaded in (False, True):
            d = str(tmp_path_factory.mktemp("lists"))
            nls = synth.box_room(d, width=width)
            with open(nls) as f:
                j = json.load(f)
            if unshaded:
                j["materials"][1] = {"name": "left", "type": "microfacet"}
            files = {}
            for name in ("none", "blinn", "thinfilm"):
                k = dict(j, materials=j["materials"] + ([EXTRA[name]] if name in EXTRA else []))
                files[name] = os.path.join(d, name + ".nls")
                with open(files[name], "w") as f:
                    json.dump(k, f)
            out[width, unshaded] = files
    return out


# 1, 256, 289 and 2025 pixels: one lane, a full block, one over it, several
@pytest.mark.parametrize("width", [1, 16, 17, 45])
@pytest.mark.parametrize("unshaded", [False, True])
@pytest.mark.parametrize("extra", ["blinn", "thinfilm"])
def test_same_image(scenes, width, unshaded, extra):
    from lambda_b200.renderer import Context
    from lambda_b200.scene import load_nls
    images, grads = [], []
    for name in ("none", extra):
        ctx = Context(0)
        ctx.upload(load_nls(scenes[width, unshaded][name]))
        images.append([ctx.render(spp, 6, 0.85, seed=4) for spp in (1, 5)])
        w, h = ctx.size
        d = np.random.default_rng(1).normal(size=(h, w, 3)).astype(np.float32)
        grads.append(ctx.adjoint(5, 6, 0.85, d, seed=4, image=True))
        ctx.close()
    for a, b in zip(*images):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    # gradients: the same terms summed in any order (some 10^4 floats); the
    # unused material's entries are zero
    for a, b in zip(*grads):
        na, nb = (np.linalg.norm(x.astype(np.float64)) for x in (a, b))
        assert np.isfinite(na) and abs(na - nb) <= 2e-5 * nb


def test_list_longer_than_its_grid(tmp_path):
    """2^21 paths: the list's launch has 16 blocks of 256 per SM, a third of
    its hits."""
    from lambda_b200.renderer import Context
    from lambda_b200.scene import load_nls
    nls = synth.box_room(str(tmp_path), width=1024)
    with open(nls) as f:
        j = json.load(f)
    images = []
    for name in ("none", "blinn"):
        path = os.path.join(str(tmp_path), name + ".nls")
        with open(path, "w") as f:
            json.dump(dict(j, materials=j["materials"] + ([EXTRA[name]] if name in EXTRA else [])), f)
        ctx = Context(0)
        ctx.upload(load_nls(path))
        images.append(ctx.render(2, 4, 0.85, seed=4))
        ctx.close()
    assert np.array_equal(images[0].view(np.uint32), images[1].view(np.uint32))
