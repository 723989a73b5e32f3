"""The adjoint's two replays: with the primal pass's hits recorded (up to 8
GiB of them) and re-traced beyond.  A frame whose hits do not fit is compared
with the mean of two halves of its samples, whose hits do: the paths are the
same, so gradients and images agree to the rounding of their float sums."""
import os

import numpy as np
import pytest

from lambda_b200 import synth

pytestmark = pytest.mark.gpu

# 64 vertices x 36 B x 512^2 pixels: 16 samples are 9.7 GB, 8 are 4.8 GB
BOUNCES, SPP, W = 62, 16, 512


def scenes(tmp):
    rng = np.random.default_rng(4)
    yield synth.diff_scene(os.path.join(tmp, "diff"), rng.uniform(0.2, 0.8, (64, 32)),
                           rng.uniform(200, 800, (8, 8)), width=W)
    yield synth.mixed(os.path.join(tmp, "mixed"), width=W, ar=1.0)


def test_recorded_and_traced_replay(tmp_path):
    from lambda_b200.renderer import Context
    from lambda_b200.scene import load_nls
    for nls in scenes(str(tmp_path)):
        ctx = Context(0)
        ctx.upload(load_nls(nls))
        w, h = ctx.size
        d = np.random.default_rng(1).normal(size=(h, w, 3)).astype(np.float32)
        whole = ctx.adjoint(SPP, BOUNCES, 0.7, d, seed=3, image=True)
        rays_whole = ctx.stats()["rays"]
        halves = [ctx.adjoint(SPP // 2, BOUNCES, 0.7, d, seed=3, spp_offset=o, image=True) for o in (0, SPP // 2)]
        # the traced replay casts the extension rays twice
        assert rays_whole > 1.2 * 2 * ctx.stats()["rays"]
        for a, b0, b1 in zip(whole, *halves):
            a, b = a.astype(np.float64), 0.5 * (b0.astype(np.float64) + b1.astype(np.float64))
            assert np.all(np.isfinite(a)) and np.any(a != 0)
            # sums of some 10^5 float terms in any order
            assert np.linalg.norm(a - b) <= 2e-5 * np.linalg.norm(b)
        ctx.close()
