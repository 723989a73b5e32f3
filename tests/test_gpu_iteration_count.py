"""A small render is enqueued without waiting for the device, but not beyond
its paths' end: its iterations are counted (by its launches) where the roulette
probability or an empty view ends the paths long before the scattering limit
does, and the image is that of the longer way (a limit beyond what is enqueued
so, which no path reaches)."""
import os

import numpy as np
import pytest

from lambda_b200 import synth

pytestmark = pytest.mark.gpu


def counter(launches):
    """Launches -> iterations, from a render that takes 2 (no scattering) and
    one that takes 16 (14 scatterings, nearly no roulette)."""
    few, many = launches(0, 0.999), launches(14, 0.999)
    assert (many - few) % 14 == 0
    return lambda n: 2 + (n - few) * 14 / (many - few)


@pytest.mark.parametrize("p", [0.0, 0.1, 0.3, 0.5])
@pytest.mark.parametrize("batch", [False, True])
def test_low_probability(tmp_path, p, batch):
    from lambda_b200.renderer import Context
    from lambda_b200.scene import load_nls
    sc = load_nls(synth.mixed(os.path.join(str(tmp_path), "mixed"), width=16))
    ctx = Context(0)
    ctx.upload_many([sc])

    def render(bounces, q):
        if batch:
            jobs = [dict(scene=0, spp=1, max_scatterings=bounces, sample_p=s, seed=3) for s in (q / 2, q)]
            return np.asarray(ctx.render_batch(jobs)[1])
        return ctx.render(1, bounces, q, seed=3)

    def launches(bounces, q):
        render(bounces, q)
        return ctx.stats()["launches"]

    iterations = counter(launches)
    img = render(14, p)
    # 208 or 416 paths: on average less than 0.3 of one is left after 1, 4, 7
    # and 11 iterations with these probabilities; iterations come in pairs, one
    # of them in hand
    assert iterations(ctx.stats()["launches"]) <= {0.0: 4, 0.1: 6, 0.3: 10, 0.5: 14}[p]
    other = render(40, p)
    assert np.array_equal(img.view(np.uint32), other.view(np.uint32))
    ctx.close()


@pytest.mark.parametrize("bounces", [3, 4, 8, 14])
def test_view_of_nothing(tmp_path, bounces):
    from lambda_b200.renderer import Context
    from lambda_b200.scene import Camera, load_nls
    sc = load_nls(synth.mixed(os.path.join(str(tmp_path), "mixed"), width=16))
    ctx = Context(0)
    ctx.upload(sc)

    def launches(b, q):
        ctx.render(1, b, q, seed=3)
        return ctx.stats()["launches"]

    iterations = counter(launches)
    sc.cam = Camera([0, 0, 500], [0, 1, 900], [0, 0, 1], 16, 40, 1.25)
    ctx.upload(sc)
    img = ctx.render(1, bounces, 0.999, seed=3)
    assert not img.any()
    assert iterations(ctx.stats()["launches"]) <= 4
    ctx.close()
