"""Each way of enqueuing a render's iterations (pairs without waiting, up to 16
iterations; checked groups beyond) against the restatement on the same random
streams, with the bounds of that comparison's other tests: a path dropped, cut
short or shaded twice by all of the ways would show here and not in the
comparison among them."""
import os

import pytest

from lambda_b200 import synth
from oracle import restatement as R
from tests.test_gpu_oracle import _compare

pytestmark = pytest.mark.gpu


# 13, 14 and 15 scatterings: 15, 16 and 17 iterations
@pytest.mark.parametrize("bounces", [0, 1, 2, 3, 13, 14, 15, 33])
@pytest.mark.parametrize("name", ["mixed", "box"])
def test_same_paths_as_the_restatement(tmp_path, name, bounces):
    from lambda_b200.renderer import Context
    from lambda_b200.scene import flatten, load_nls
    make = {"mixed": synth.mixed, "box": synth.box_room}[name]
    fs = flatten(load_nls(make(os.path.join(str(tmp_path), name), width=48)))
    ctx = Context(0)
    ctx.upload(fs)
    g = ctx.render(5, bounces, 0.85, seed=2)
    h, w = g.shape[:2]
    assert ctx.stats()["paths"] == 5 * w * h
    _compare(g, R.Oracle(fs).render(5, bounces, 0.85, rng=R.RNG_PCG, seed=2))
    ctx.close()
