"""The tone map's two access paths (16-byte words, single channels) and its
byte conversion: sizes around a word and a block, arrays at every alignment,
and values next to the rounding boundaries of the sRGB byte.  The oracle is
the reference's formula (src/renderer.cpp:149-176, cg.hpp:149-162, 181-194) in
double precision."""
import ctypes

import numpy as np
import pytest

from lambda_b200 import _lib as L

pytestmark = pytest.mark.gpu

Y_MID = 0.12


def oracle(img):
    x = img.astype(np.float64)
    lum = 0.2126 * x[..., 0] + 0.7152 * x[..., 1] + 0.0722 * x[..., 2]
    e = Y_MID / np.exp(np.log(np.maximum(lum, 2.0 ** -23)).mean())
    t = 10.0 * e * x
    tm = t * (0.3 * t + 0.14) / (t * (0.3 * t + 2.8) + 10.0)
    s = np.where(tm > 0.0031308, 1.055 * np.power(np.maximum(tm, 0.0031308), 1 / 2.4) - 0.055, 12.92 * tm)
    return tm, 255.0 * s + 0.5


def run(img, off_in=0, off_tm=0, off_24=0):
    import torch
    h, w = img.shape[:2]
    n = 3 * w * h
    src = torch.zeros(n + 8, device="cuda")
    src[off_in:off_in + n] = torch.from_numpy(img.reshape(-1)).cuda()
    tm, b = torch.full((n + 8,), -7.0, device="cuda"), torch.full((n + 8,), 99, dtype=torch.uint8, device="cuda")
    rc = L.lib().lgpu_tonemap_noalloc(src.data_ptr() + 4 * off_in, w, h, ctypes.c_float(Y_MID),
                                      tm.data_ptr() + 4 * off_tm, b.data_ptr() + off_24, 0)
    assert rc == 0
    tm, b = tm.cpu().numpy(), b.cpu().numpy()
    # nothing beyond the arrays is written
    assert np.all(np.delete(tm, np.s_[off_tm:off_tm + n]) == -7.0)
    assert np.all(np.delete(b, np.s_[off_24:off_24 + n]) == 99)
    return tm[off_tm:off_tm + n].reshape(img.shape), b[off_24:off_24 + n].reshape(img.shape)


@pytest.mark.parametrize("w,h", [(1, 1), (2, 1), (3, 1), (4, 1), (5, 3), (17, 15), (641, 359), (1920, 1080)])
def test_paths(w, h):
    rng = np.random.default_rng(w * h)
    img = np.exp(rng.normal(-1.0, 2.0, (h, w, 3))).astype(np.float32)
    img[rng.uniform(size=img.shape) < 0.05] *= -0.2  # out of gamut
    tm, b = run(img)
    want, v = oracle(img)
    # float arithmetic: some ten roundings and the exposure's expf and logf
    assert np.allclose(tm, want, rtol=4e-6, atol=1e-7)
    lo = np.clip(np.floor(v - 1e-3), 0, 255)
    hi = np.clip(np.floor(v + 1e-3), 0, 255)
    assert np.all((b >= lo) & (b <= hi))
    for offs in ((1, 0, 0), (0, 2, 0), (0, 0, 1), (3, 1, 2), (4, 4, 4)):
        tm2, b2 = run(img, *offs)
        assert np.array_equal(tm.view(np.uint32), tm2.view(np.uint32)) and np.array_equal(b, b2), offs
