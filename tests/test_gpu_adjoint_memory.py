"""The adjoint records its hits only where they leave as much of the device's
memory free as they take: with little memory free the replay traces its rays
instead, the gradients are the same, and what another allocation could have
before the call it still can have."""
import os

import numpy as np
import pytest

from lambda_b200 import synth

pytestmark = pytest.mark.gpu

W, SPP, BOUNCES = 512, 16, 14
HITS = (BOUNCES + 2) * 36 * W * W * SPP  # 2.4 GB


def test_little_memory(tmp_path):
    import torch
    from lambda_b200.renderer import Context
    from lambda_b200.scene import load_nls
    sc = load_nls(synth.mixed(os.path.join(str(tmp_path), "mixed"), width=W, ar=1.0))
    d = np.random.default_rng(1).normal(size=(W, W, 3)).astype(np.float32)
    free = lambda: torch.cuda.mem_get_info()[0]

    def adjoint():
        """The gradients, the rays traced and the memory it took."""
        ctx = Context(0)
        ctx.upload(sc)
        f = free()
        g = ctx.adjoint(SPP, BOUNCES, 0.8, d, seed=3)
        return ctx, g, ctx.stats()["rays"], f - free()

    ctx, g0, rays0, took = adjoint()
    assert ctx.size == (W, W) and took > HITS
    ctx.close()
    # room for the arena and one and a half times the hits
    keep = took - HITS + HITS * 3 // 2
    filler = torch.empty(free() - keep - (256 << 20), dtype=torch.uint8, device="cuda")
    try:
        ctx, g1, rays1, less = adjoint()
        other = torch.empty(HITS, dtype=torch.uint8, device="cuda")
        del other
    finally:
        del filler
        torch.cuda.empty_cache()
    ctx.close()
    assert rays1 > 1.2 * rays0 and less < took - HITS // 2
    for a, b in zip(g0, g1):
        # float sums of some 10^6 terms in any order
        assert np.linalg.norm(a - b) <= 2e-5 * np.linalg.norm(b)
