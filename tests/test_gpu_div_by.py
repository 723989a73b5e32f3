"""The film's and the spectra's divisions by scene constants (div_by): the
spectrum probe and whole images at spectral settings whose constants divide
differently (5 nm bins exactly, the default's 320/79 nm not, an odd one), and
at a setting too small for the corrected quotient, which takes the division.
The oracle is the restatement's spectrum lookup in numpy float32, whose
division IEEE rounds; the coordinate decides which two bins are blended, so a
last-bit difference shows."""
import numpy as np
import pytest

from lambda_b200 import _lib as L
from lambda_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bins,lo,hi", [(80, 400.0, 720.0), (81, 380.0, 780.0), (37, 391.3, 777.7),
                                        (80, 4e-13, 7.2e-13)])
def test_lookup_coordinate(tmp_path, bins, lo, hi):
    from lambda_b200.renderer import Context
    from lambda_b200.scene import FlatScene, SpectralConfig, load_nls
    nls = synth.box_room(str(tmp_path / "box"), width=16)
    sc = load_nls(nls, SpectralConfig(bins, 400.0, 720.0, 4) if hi < 1 else SpectralConfig(bins, lo, hi, 4))
    flat = FlatScene(sc)
    flat.scene.spec.lambda_inf, flat.scene.spec.lambda_sup = np.float32(lo), np.float32(hi)
    rng = np.random.default_rng(3)
    flat.spectra[0] = rng.uniform(0, 1, bins)
    ctx = Context(0)
    ctx.upload(flat)
    f = np.float32
    inf, sup = f(lo), f(hi)
    delta = f(f(sup - inf) / f(bins - 1))
    n = 50000
    lam = (rng.uniform(0, 1, (n, 4)) * (hi - lo) + lo).astype(np.float32)
    lam[:, 0] = (inf + rng.integers(0, bins, n).astype(np.float32) * delta).astype(np.float32)  # on the bins
    lam = np.clip(lam, np.nextafter(inf, f(1e30)), np.nextafter(sup, f(0)))
    q = np.zeros(n, L.PROBE_DTYPE)
    q["op"], q["index"], q["lambda"][:, :4] = L.PROBE_SPECTRUM, 0, lam
    got = ctx.probe(q)["value"][:, :4]
    x = ((lam - inf) / delta).astype(np.float32)
    i = np.minimum(x.astype(np.uint32), bins - 2)
    t = (x - i.astype(np.float32)).astype(np.float32)
    v = flat.spectra[0].astype(np.float32)
    want = (((f(1) - t) * v[i]).astype(np.float32) + (t * v[i + 1]).astype(np.float32)).astype(np.float32)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    ctx.close()
