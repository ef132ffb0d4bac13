"""FP32 back-projection of R-weighted series on the tensor cores: edges of its tiles
(hexagons of 14 columns x 13 depths, groups of 256 slices, pairs of views), of its
operand window (z-factors widen it to two products) and values that are not finite.

Tolerance: the sums keep the FP32 result of the separately rounded interpolation to
a few times 2^-24 per sample; what remains against the f32 oracle is the other FFT of
the R-weighting, for which the whole-path tests allow rel-L2 1e-5."""
import numpy as np
import pytest

import oracle as O
import tiltgpu as T
from tgutil import angles, rel_l2, smooth_stack

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.fixture(autouse=True)
def tensor_core_kernel(monkeypatch):
    # small series would take the CUDA-core kernel
    monkeypatch.setenv("TG_BP_VARIANT", "14")


def compare(nx, ny, ang, seed, zfactor=None, **kw):
    nz = len(ang)
    proj = smooth_stack(nz, ny, nx, seed=seed)
    okw = dict(kw)
    if zfactor is not None:
        okw["zfactor"] = zfactor
    with T.Session(nx, ny, nz, ang, **okw) as s:
        assert s.kernel_info()["variant_name"] == "tcgen05-hex126"
        s.upload(proj)
        s.reconstruct()
        vol, st = s.download()
    ref, rst = O.run(O.Params(nx, ny, nz, ang, **okw), proj, 32)
    assert rel_l2(vol, ref) <= TOL
    for k in ("amin", "amax"):
        assert st[k] == pytest.approx(rst[k], rel=1e-4, abs=1e-5)
    assert abs(st["amean"] - rst["amean"]) <= 1e-5 * max(abs(rst["amin"]), abs(rst["amax"]))


@pytest.mark.parametrize("ny", [1, 15, 16, 17, 129, 255, 256, 257, 300])
def test_slice_groups(ny):
    compare(40, ny, angles(-60, 60, 20), 1000 + ny, thickness=12)


@pytest.mark.parametrize("onx,onz", [(2, 1), (6, 4), (7, 5), (13, 9), (14, 13), (15, 14), (200, 3), (33, 170)])
@pytest.mark.parametrize("fill", ["mean", "edge"])
def test_output_edges(onx, onz, fill):
    compare(64, 6, angles(-62, 62, 15.5), onx * 100 + onz, width=onx, thickness=onz, fill_mode=fill)


@pytest.mark.parametrize("nz", [1, 2, 3, 31, 32, 33, 64, 65])
def test_view_counts(nz):
    ang = np.linspace(-70, 70, nz).astype(np.float32) if nz > 1 else np.array([17.1], np.float32)
    compare(48, 5, ang, 50 + nz, thickness=30)


@pytest.mark.parametrize("zf", [0.5, 1.3, 2.0])
def test_zfactors(zf):
    ang = angles(-80, 80, 16)
    z = np.linspace(1.0, zf, len(ang)).astype(np.float32)
    compare(96, 9, ang, int(zf * 10), zfactor=z, thickness=41, max_cosine_tilt=70.0)


def test_tiny_row():
    compare(2, 3, angles(-45, 45, 15), 5, thickness=20, width=30)


def test_large_enough_series_take_it_by_themselves(monkeypatch):
    monkeypatch.delenv("TG_BP_VARIANT")
    ang = angles(-60, 60, 2)
    for (nx, ny, thick, kw), want in {(512, 512, 200, ()): True, (512, 16, 200, ()): False, (32, 512, 16, ()): False,
                                      (512, 512, 200, (("no_weight", True),)): False,
                                      (512, 512, 200, (("storage", "fp16"),)): False}.items():
        with T.Session(nx, ny, len(ang), ang, thickness=thick, **dict(kw)) as s:
            name = s.kernel_info()["variant_name"]
        assert (name == "tcgen05-hex126") == want, (nx, ny, thick, kw, name)


def test_batched_and_iterated_results_equal_the_series_alone():
    shapes = [(64, 20, 17, 30, 0), (48, 270, 9, 24, 2), (80, 33, 12, 40, 3), (64, 20, 16, 31, 2)]

    def make(i):
        nx, ny, nz, thick, sirt = shapes[i]
        ang = np.linspace(-58, 58, nz).astype(np.float32)
        s = T.Session(nx, ny, nz, ang, thickness=thick, sirt=sirt, sirt_relax=0.5,
                      xtilt=np.full(nz, 1.5, np.float32) if i == 3 else None)
        s.upload(smooth_stack(nz, ny, nx, seed=300 + i))
        return s
    alone = []
    for i in range(len(shapes)):
        with make(i) as s:
            s.reconstruct()
            alone.append(s.download())
    sessions, b = [make(i) for i in range(len(shapes))], T.Batch()
    for s in sessions:
        b.add(s)
    for _ in range(2):
        b.reconstruct()
        for (va, sa), s in zip(alone, sessions):
            vb, sb = s.download()
            np.testing.assert_array_equal(vb, va)
            assert sa == sb
    b.close()
    for s in sessions:
        s.close()


def test_scale_of_the_data_does_not_matter():
    # rows are staged times a power of two taken from their range
    ang = angles(-60, 60, 10)
    proj = smooth_stack(len(ang), 7, 64, seed=8)
    kw = dict(thickness=24, radial=(0.35, 0.035))
    base, _ = T.reconstruct(proj, ang, **kw)
    for e in (-100, -20, 40, 100):
        vol, _ = T.reconstruct(np.ldexp(proj, e).astype(np.float32), ang, **kw)
        np.testing.assert_array_equal(vol, np.ldexp(base, e).astype(np.float32))
    zero, _ = T.reconstruct(np.zeros_like(proj), ang, **kw)
    assert not zero.any()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_values_that_are_not_finite_stay_in_their_rows(bad):
    # the R-weighting spreads a bad sample over its row and the one that shares its transform
    # (rows 2j and 2j + 1); the others come out as ever (zero fill: no mean carries it on)
    ang = angles(-60, 60, 12)
    proj = smooth_stack(len(ang), 20, 72, seed=9)
    kw = dict(thickness=18, fill_mode="zero")
    good, _ = T.reconstruct(proj, ang, **kw)
    proj[3, 11, 40] = bad
    vol, _ = T.reconstruct(proj, ang, **kw)
    assert np.isnan(vol[11]).any() and np.isfinite(good).all()
    rest = np.delete(vol, [10, 11], 0)
    assert np.isfinite(rest).all()
    assert rel_l2(rest, np.delete(good, [10, 11], 0)) <= TOL
    ref, _ = O.run(O.Params(72, 20, len(ang), ang, **kw), proj, 32)
    np.testing.assert_array_equal(np.isfinite(vol[11]), np.isfinite(ref[11]))
