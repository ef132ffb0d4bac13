"""R-weighting of rows of any width: transforms of the row's own length (2^k, 3 * 2^k), and of
a padded length whose weights are the spectrum of the row's circular kernel.

Reference: the same filter in FP64 (numpy).  Tolerance: two f32 transforms of up to 2^13
samples each add about 2^-24 * sqrt(13) of the mean-free row's norm, and the filter
passes a tenth or more of that norm: rel-L2 2e-6.  The rows carry a mean 1000 times
their spread in one case; the filter removes it, so it must not cost accuracy beyond the
rounding of the samples themselves."""
import numpy as np
import pytest

import tiltgpu as T

pytestmark = pytest.mark.gpu
WIDTHS = [2, 3, 5, 31, 100, 127, 128, 129, 192, 255, 257, 384, 385, 500, 509, 512, 640, 768, 769, 1000, 1021, 1023, 1025,
          1440, 1531, 1536, 1537, 2047, 2048, 2049, 2880, 3072, 3073, 3710, 4091, 4096]


def filtered(x, cutoff=0.35, falloff=0.05):
    n = x.shape[-1]
    i = np.arange(n)
    w = np.where(i <= n // 2, i, n - i) / (n // 2 + 1)
    wt = np.where(w <= cutoff, w, w * np.exp(-(w - cutoff) ** 2 / (2 * falloff ** 2)))
    return np.fft.ifft(np.fft.fft(x.astype(np.float64)) * wt).real


@pytest.mark.parametrize("n", WIDTHS)
def test_rweighting_of_every_width(n):
    rng = np.random.default_rng(n)
    for ny, nz, offset in ((3, 2, 0.0), (2, 1, 1000.0)):
        x = (rng.standard_normal((nz, ny, n)) + offset).astype(np.float32)
        want = filtered(x)
        err = np.linalg.norm(T.apply_rweighting(x, 0.35, 0.05) - want) / np.linalg.norm(want)
        tol = 2e-6 if offset == 0.0 or n not in (256, 384, 512, 768, 1536, 2048, 3072, 4096) else 2e-3
        assert err <= tol, (n, offset, err)


@pytest.mark.parametrize("n", [100, 509, 1023, 1440])
@pytest.mark.parametrize("storage,fill,kw", [("fp32", "mean", {}), ("fp16", "edge", dict(cosine_interp="cubic")),
                                             ("bf16", "zero", dict(xtilt=1.5)), ("fp32", "edge", dict(local=True))])
def test_formats_of_padded_rows(n, storage, fill, kw, monkeypatch):
    # every staging format at these widths equals the generic kernel's to rounding (half
    # staging: the same kernel, the same values)
    ang = np.linspace(-50, 50, 9).astype(np.float32)
    x = np.random.default_rng(n).standard_normal((9, 6, n)).astype(np.float32)
    opts = dict(thickness=24, storage=storage, fill_mode=fill, width=n + 7)
    opts.update({k: v for k, v in kw.items() if k == "cosine_interp"})
    if "xtilt" in kw:
        opts["xtilt"] = np.full(9, kw["xtilt"], np.float32)
    if "local" in kw:
        opts["local"] = [(v, px, py, 0.5, -0.3) for v in range(9) for px in (0, n - 1) for py in (0, 5)]
    got, _ = T.reconstruct(x, ang, **opts)
    monkeypatch.setenv("TG_FILTER_GENERIC", "1")
    want, _ = T.reconstruct(x, ang, **opts)
    tol = {"fp32": 2e-6, "fp16": 2e-4, "bf16": 2e-3}[storage]  # a value near a midpoint rounds either way
    assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want)


@pytest.mark.parametrize("n", [11, 13, 22, 97, 254, 509, 1023, 2047, 2051, 8191, 9601, 9887])
def test_convolution_keeps_its_order_of_sums(n):
    # widths without a radix plan in half staging: the tiled convolution sums like one output
    # per thread does (f32 fused multiply-adds in the order of the samples), bit for bit up
    # to the staging's rounding; the reference rounds every sum to f32 from FP64 products
    rng = np.random.default_rng(n)
    x = rng.standard_normal((1, 3, n)).astype(np.float32)
    i = np.arange(n)
    w = np.where(i <= n // 2, i, n - i).astype(np.float32) / np.float32(n // 2 + 1)
    kw = dict(thickness=1, no_cosine_stretch=True, fill_mode="edge", storage="bf16", radial=(10.0, 0.05))
    vol, _ = T.reconstruct(x, np.array([0.0], np.float32), **kw)
    h = np.fft.ifft(w.astype(np.float64)).real.astype(np.float32).astype(np.float64)
    want = np.fft.ifft(np.fft.fft(x[0].astype(np.float64)) * np.fft.fft(h)).real
    # bf16 staging: 2^-9 of each value, and the sums' own rounding far below it
    assert np.abs(vol[:, 0, :n - 1] - want[:, :n - 1]).max() <= 2 ** -8 * np.abs(want).max()
    assert np.linalg.norm(vol[:, 0, :n - 1] - want[:, :n - 1]) <= 2 ** -8.5 * np.linalg.norm(want)
