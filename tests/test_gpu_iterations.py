"""How a chunk's iterations are enqueued: all at once (items fit the queue and
paths end within 16 iterations), in checked groups with a captured graph, and
with new paths generated in later iterations; and the shading launches that a
scene's materials leave out.  Every way has to give the same image as the
one-thread-per-pixel kernel's paths do, bit for bit among themselves."""
import os

import numpy as np
import pytest

from lambda_b200 import _lib as L
from lambda_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scenes(tmp_path_factory):
    d = str(tmp_path_factory.mktemp("iters"))
    return {"mixed": synth.mixed(os.path.join(d, "mixed"), width=72), "box": synth.box_room(os.path.join(d, "box"), width=64)}


# 13, 14 and 15 bounces: 15, 16 and 17 iterations (the last one over the limit)
@pytest.mark.parametrize("bounces", [0, 1, 2, 13, 14, 15, 33])
@pytest.mark.parametrize("name", ["mixed", "box"])
def test_same_image(scenes, name, bounces):
    from lambda_b200.renderer import Context
    from lambda_b200.scene import load_nls
    ctx = Context(0)
    ctx.upload(load_nls(scenes[name]))
    base = ctx.render(9, bounces, 0.85, seed=2)
    n0 = ctx.stats()["paths"]
    for kw in (dict(graphs=0), dict(graphs=1, queue_cap=1024), dict(graphs=0, queue_cap=3000),
               dict(graphs=1, queue_cap=1 << 24)):
        ctx.set_wave_config(**kw)
        img = ctx.render(9, bounces, 0.85, seed=2)
        assert np.array_equal(base.view(np.uint32), img.view(np.uint32)), kw
        assert ctx.stats()["paths"] == n0
    ctx.close()


def test_materials_changed_after_upload(scenes):
    """A material whose type changes by lgpu_update_materials gets its
    launch."""
    from lambda_b200.renderer import Context
    from lambda_b200.scene import FlatScene, load_nls
    flat = FlatScene(load_nls(scenes["box"]))
    ctx = Context(0)
    ctx.upload(flat)
    ctx.render(4, 4, 0.8, seed=1)
    film, albedo = flat.materials[1], flat.materials[1].spectrum[0]
    flat.spectra[albedo] = 1.45
    film.type, film.alpha, film.d = L.MAT_THINFILM, 8.0, 450.0
    film.spectrum[1] = flat.materials[2].spectrum[0]
    flat.spectra[film.spectrum[1]] = 1.6
    ctx.update_materials(flat)
    updated = ctx.render(4, 4, 0.8, seed=1)
    other = Context(0)
    other.upload(flat)
    fresh = other.render(4, 4, 0.8, seed=1)
    assert np.array_equal(updated.view(np.uint32), fresh.view(np.uint32))
    ctx.close()
    other.close()
