"""R-weighting inside a reconstruction: FP32 rows of a width that has no register-resident
transform of its own length keep the generic kernel's arithmetic, bit for bit -- a volume's
mean is a small difference of large sums, which any other transform of the rows moves."""
import ctypes
import math

import numpy as np
import pytest

import tiltgpu as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [100, 151, 443, 509, 1000, 1023, 1440, 1598])
@pytest.mark.parametrize("kw", [dict(fill_mode="zero"), dict(log=True), dict(sirt=2, sirt_relax=0.3, fill_mode="edge")])
def test_fp32_sessions_keep_the_generic_kernels_bits(n, kw, monkeypatch):
    ang = np.linspace(-50, 50, 7).astype(np.float32)
    x = (3.0 + np.random.default_rng(n).standard_normal((7, 5, n))).astype(np.float32)
    opts = dict(thickness=20, radial=(0.35, 0.035), **kw)
    got, st = T.reconstruct(x, ang, **opts)
    monkeypatch.setenv("TG_FILTER_GENERIC", "1")
    want, wst = T.reconstruct(x, ang, **opts)
    np.testing.assert_array_equal(got, want)
    assert st == wst


@pytest.mark.parametrize("n", [11, 97, 131, 254])
def test_the_convolution_sums_in_the_order_of_the_samples(n):
    # one fused multiply-add per sample, in order, with f32 taps: exact.  One view at 0 degrees
    # and one depth: the volume's rows are the filtered rows
    x = np.random.default_rng(n).standard_normal((1, 3, n)).astype(np.float32)
    vol, _ = T.reconstruct(x, np.array([0.0], np.float32), thickness=1, no_cosine_stretch=True, fill_mode="edge",
                           radial=(10.0, 0.05))
    i = np.arange(n)
    w = np.where(i <= n // 2, i, n - i).astype(np.float32) / np.float32(n // 2 + 1)
    h = []
    for m in range(n):
        acc = 0.0
        for k in range(n):
            acc += float(w[k]) * math.cos(2.0 * math.pi * k * m / n)
        h.append(np.float32(acc / n))
    fmaf = ctypes.CDLL("libm.so.6").fmaf
    fmaf.restype, fmaf.argtypes = ctypes.c_float, [ctypes.c_float] * 3
    want = np.zeros((3, n), np.float32)
    for r in range(3):
        for k in range(n):
            s = 0.0
            for m in range(n):
                s = fmaf(float(h[(k - m) % n]), float(x[0, r, m]), s)
            want[r, k] = s
    np.testing.assert_array_equal(vol[:, 0, :], want)
