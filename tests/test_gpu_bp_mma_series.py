"""The tensor-core back-projector over many series: their tensor maps, their time limits and
the values they are staged with.

Tolerance against the shared-memory kernel (rel-L2 1e-5): both are within a few 2^-24 per
sample of the exact interpolation of the same filtered rows."""
import numpy as np
import pytest

import tiltgpu as T
from tgutil import angles, rel_l2, smooth_stack

pytestmark = pytest.mark.gpu
TOL = 1e-5
TENSOR, SHARED = "14", "0"


@pytest.fixture(autouse=True)
def tensor_core_kernel(monkeypatch):
    monkeypatch.setenv("TG_BP_VARIANT", TENSOR)


def session(nx, ny, ang, proj, **kw):
    s = T.Session(nx, ny, len(ang), ang, **kw)
    s.upload(proj)
    return s


SHAPES = [(64, 20, 9, 24), (40, 130, 12, 31), (96, 17, 7, 12), (33, 48, 20, 40), (128, 8, 5, 70), (64, 21, 9, 23)]


@pytest.mark.parametrize("how", ["one", "batch", "server"])
def test_series_that_follow_each_other_on_the_same_memory(how, monkeypatch):
    # freed buffers come back at the addresses of the series before, with another shape
    ang = [np.linspace(-55, 55, nz).astype(np.float32) for _, _, nz, _ in SHAPES]
    proj = [smooth_stack(nz, ny, nx, seed=70 + i) for i, (nx, ny, nz, _) in enumerate(SHAPES)]
    monkeypatch.setenv("TG_BP_VARIANT", SHARED)
    want = [T.reconstruct(p, a, thickness=s[3])[0] for p, a, s in zip(proj, ang, SHAPES)]
    monkeypatch.setenv("TG_BP_VARIANT", TENSOR)
    n = len(SHAPES)
    sv = T.Server(budget_bytes=1 << 30) if how == "server" else None
    for turn in range(4):
        order = [(i + turn) % n for i in range(n)][::1 if turn % 2 else -1]
        if how == "one":
            got = {i: T.reconstruct(proj[i], ang[i], thickness=SHAPES[i][3])[0] for i in order}
        elif how == "server":
            outs = {i: np.empty_like(want[i]) for i in order}
            jobs = [sv.submit(proj[i], ang[i], out=outs[i], thickness=SHAPES[i][3]) for i in outs]
            for j in jobs:
                assert sv.wait(j)["status"] == 0
                sv.release(j)
            got = outs
        else:
            ss, b = {i: session(SHAPES[i][0], SHAPES[i][1], ang[i], proj[i], thickness=SHAPES[i][3]) for i in order}, T.Batch()
            for s in ss.values():
                b.add(s)
            b.reconstruct()
            got = {i: s.download()[0] for i, s in ss.items()}
            b.close()
            for s in ss.values():
                s.close()
        for i, v in got.items():
            assert rel_l2(v, want[i]) <= TOL, (turn, i)
    if sv:
        sv.close()


# ---- a wait that runs out: a status, no endless barrier, and the session works again ----

def fails(call):
    with pytest.raises(T.TiltGpuError) as e:
        call()
    assert e.value.code == -4 and "timed out" in str(e.value)


@pytest.mark.parametrize("sirt", [0, 2])
@pytest.mark.parametrize("nz,skip", [(31, 1), (31, 15), (31, 0), (6, 2), (3, 1), (1, 0)])
@pytest.mark.parametrize("ny", [40, 272])  # consumer warps with and without columns of their own
def test_bounded_wait_times_out_and_session_recovers(nz, skip, sirt, ny):
    ang = np.linspace(-60, 60, nz).astype(np.float32)
    kw = dict(thickness=61, sirt=sirt, sirt_relax=0.5) if sirt else dict(thickness=61)
    with session(200, ny, ang, smooth_stack(nz, ny, 200, seed=nz), **kw) as s:
        assert s.kernel_info()["variant_name"] == "tcgen05-hex126"
        s.reconstruct()
        good, st = s.download()
        s.inject_wait_fault(skip_stage=skip, wait_limit_us=5000)
        fails(s.reconstruct)
        s.inject_wait_fault(-1, 0)
        s.reconstruct()
        again, st2 = s.download()
    np.testing.assert_array_equal(again, good)
    assert st == st2


def test_bounded_wait_in_a_batch():
    ang = [np.linspace(-55, 55, nz).astype(np.float32) for _, _, nz, _ in SHAPES]
    ss = [session(nx, ny, ang[i], smooth_stack(nz, ny, nx, seed=20 + i), thickness=th, sirt=2 * (i % 2), sirt_relax=0.5)
          for i, (nx, ny, nz, th) in enumerate(SHAPES)]
    b = T.Batch()
    for s in ss:
        b.add(s)
    b.reconstruct()
    good = [s.download()[0] for s in ss]
    ss[2].inject_wait_fault(skip_stage=3, wait_limit_us=5000)
    fails(b.reconstruct)
    for s in ss:  # series whose tiles were in the same blocks report it too
        try:
            s.synchronize()
        except T.TiltGpuError as e:
            assert e.code == -4
    ss[2].inject_wait_fault(-1, 0)
    b.reconstruct()
    for s, g in zip(ss, good):
        np.testing.assert_array_equal(s.download()[0], g)
    b.close()
    for s in ss:
        s.close()


# ---- values that are not finite: the blocks of 8 slices that hold them, and no other ----

@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_a_bad_sample_leaves_the_other_blocks_as_they_were(bad):
    ang = angles(-60, 60, 12)
    proj = smooth_stack(len(ang), 37, 90, seed=4)
    kw = dict(thickness=44, fill_mode="zero")
    with session(90, 37, ang, proj, **kw) as s:
        s.reconstruct()
        good, _ = s.download()
        proj[2, 11, 40] = proj[5, 36, 3] = bad
        s.upload(proj)
        s.reconstruct()
        vol, _ = s.download()
        blocks = np.r_[8:16, 32:37]
        np.testing.assert_array_equal(np.delete(vol, blocks, 0), np.delete(good, blocks, 0))
        assert np.isnan(vol[11]).any() and np.isnan(vol[36]).any()
        rest = np.r_[8:10, 12:16, 32:36]
        assert rel_l2(vol[rest], good[rest]) <= TOL
        proj = smooth_stack(len(ang), 37, 90, seed=4)
        s.upload(proj)
        s.reconstruct()
        np.testing.assert_array_equal(s.download()[0], good)


@pytest.mark.parametrize("sirt", [0, 1])
def test_a_series_full_of_bad_rows_does_not_hold_up_the_next_one(sirt):
    # in one batched launch the good series' tiles follow the bad one's in every block; its
    # waits are shorter than the bad one's tiles of a block together
    nb, ng = 61, 20
    angb, angg = np.linspace(-60, 60, nb).astype(np.float32), np.linspace(-60, 60, ng).astype(np.float32)
    kw = dict(fill_mode="zero", sirt=sirt, sirt_relax=0.5)
    bad = smooth_stack(nb, 256, 300, seed=1)
    bad[0, ::2, 7] = np.nan
    good = smooth_stack(ng, 40, 200, seed=2)
    with session(200, 40, angg, good, thickness=300, **kw) as g:
        g.reconstruct()
        want, _ = g.download()
        with session(300, 256, angb, bad, thickness=300, **kw) as s:
            b = T.Batch()
            b.add(s)
            b.add(g)
            g.inject_wait_fault(-1, 20000)
            s.inject_wait_fault(-1, 20000)
            b.reconstruct()
            np.testing.assert_array_equal(g.download()[0], want)
            assert np.isnan(s.download()[0]).any(axis=(1, 2)).all()
            b.close()


# ---- mean fill: a view's mean is not bound to the range of the rows that are staged ----

def both(monkeypatch, run):
    out = []
    for v in (SHARED, TENSOR):
        monkeypatch.setenv("TG_BP_VARIANT", v)
        out.append(run())
    return out


@pytest.mark.parametrize("top,mean", [(10.0, 5000.0), (1e-3, 4.0), (0.0, 70000.0), (0.0, 1e-20), (1e6, 1e-6), (1.0, -3e30)])
def test_dark_slab_of_a_bright_series(top, mean, monkeypatch):
    ang = angles(-60, 60, 10)
    proj = (top * smooth_stack(len(ang), 20, 64, seed=3)).astype(np.float32)
    means = (mean * np.linspace(0.5, 1.5, len(ang))).astype(np.float32)

    def run():  # wide enough that voxels project outside the rows
        with session(64, 20, ang, proj, width=90, thickness=50) as s:
            s.set_view_means(means)
            s.reconstruct()
            return s.download()
    (want, wst), (got, st) = both(monkeypatch, run)
    assert np.isfinite(want).all() and np.isfinite(got).all()
    assert rel_l2(got, want) <= TOL
    assert st["amin"] == pytest.approx(wst["amin"], rel=1e-5) and st["amax"] == pytest.approx(wst["amax"], rel=1e-5)


def test_residuals_far_below_the_means(monkeypatch):
    # an empty volume stays empty where the projections are a millionth of their pinned means
    ang = angles(-60, 60, 8)
    proj = smooth_stack(len(ang), 20, 64, seed=6)

    def run():
        with session(64, 20, ang, proj, width=90, thickness=50, sirt=3, sirt_relax=0.1) as s:
            s.set_view_means(np.full(len(ang), 3e6, np.float32))
            s.sirt_restore(np.zeros(s.out_shape, np.float32), 0)
            s.sirt_iterate(3)
            s.sirt_end()
            return s.download()[0]
    want, got = both(monkeypatch, run)
    assert np.isfinite(got).all()
    assert rel_l2(got, want) <= TOL


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_bad_samples_with_mean_fill(bad, monkeypatch):
    # the view's mean is not finite either: every voxel outside that view's rows takes it, and
    # those inside keep the values of their own rows
    ang = angles(-60, 60, 12)
    proj = smooth_stack(len(ang), 37, 90, seed=4)
    proj[9, 11, 40] = bad

    def run():
        with session(90, 37, ang, proj, width=120, thickness=60) as s:
            s.reconstruct()
            return s.download()[0]
    want, got = both(monkeypatch, run)
    np.testing.assert_array_equal(np.isfinite(got), np.isfinite(want))
    good = np.isfinite(want)
    assert good.any() and not good[0].all()
    assert rel_l2(got[good], want[good]) <= TOL


# ---- rows of very different size: each keeps the accuracy of its own ----

def slices_agree(got, want, but=()):
    for y in range(len(want)):
        assert y in but or rel_l2(got[y], want[y]) <= TOL, y


@pytest.mark.parametrize("n,kw", [(72, {}), (64, {}), (256, dict(log=True)), (97, dict(cosine_interp="cubic")),
                                  (64, dict(xtilt=1.5)), (64, dict(sirt=2, sirt_relax=0.2))])
@pytest.mark.parametrize("size", [1e3, 1e12, 1e30])
def test_a_finite_outlier_costs_its_own_rows_only(n, kw, size, monkeypatch):
    ang = angles(-60, 60, 12)
    kw = dict(kw)
    if "xtilt" in kw:
        kw["xtilt"] = np.full(len(ang), kw["xtilt"], np.float32)
    proj = smooth_stack(len(ang), 21, n, seed=9)
    proj[3, 11, n // 2] = size

    def run():  # thick and wide: some voxels are outside the outlier's row
        with session(n, 21, ang, proj, thickness=n // 2, width=n + n // 2, fill_mode="zero", **kw) as s:
            s.reconstruct()
            return s.download()[0]
    want, got = both(monkeypatch, run)
    if "xtilt" in kw or "log" in kw:
        assert rel_l2(got, want) <= TOL
    if "xtilt" not in kw:
        # row 10 shares row 11's transform and takes over its rounding, which the second
        # iteration's other last bits make another one
        slices_agree(got, want, but=(10,) if "sirt" in kw else ())
        clean = np.abs(want[10:12]).max(0) < 10.0  # voxels that the outlier's row does not reach
        assert rel_l2(got[10:12, clean], want[10:12, clean]) <= TOL


@pytest.mark.parametrize("ny", [16, 67])
@pytest.mark.parametrize("sirt", [0, 1])
def test_rows_of_many_magnitudes(ny, sirt, monkeypatch):
    ang = angles(-60, 60, 15)
    rng = np.random.default_rng(ny)
    proj = smooth_stack(len(ang), ny, 80, seed=12)
    proj *= np.exp2(rng.integers(-60, 60, (1, (ny + 1) // 2, 1)).repeat(2, 1)[:, :ny]).astype(np.float32)

    def run():
        with session(80, ny, ang, proj, thickness=40, fill_mode="zero", sirt=sirt, sirt_relax=0.2) as s:
            s.reconstruct()
            return s.download()[0]
    want, got = both(monkeypatch, run)
    slices_agree(got, want)


def test_views_of_many_magnitudes(monkeypatch):
    # blank and faint views beside bright ones: the faint ones' voxels outside the bright
    # ones' rows are theirs alone
    ang = np.float32([0, 50])
    proj = smooth_stack(2, 20, 64, seed=5)
    for faint in (0.0, 1e-3, 1e-9):
        proj[1] = faint * smooth_stack(1, 20, 64, seed=7)[0]

        def run():
            with session(64, 20, ang, proj, width=110, thickness=12, fill_mode="zero") as s:
                s.reconstruct()
                return s.download()[0]
        want, got = both(monkeypatch, run)
        assert rel_l2(got, want) <= TOL
        alone = np.abs(want) <= 20 * faint
        assert alone.any() and rel_l2(got[alone], want[alone]) <= TOL


@pytest.mark.parametrize("e", [-126, -118, -60, 100, 112])
def test_data_near_the_ends_of_the_f32_range(e, monkeypatch):
    ang = angles(-60, 60, 12)
    proj = np.ldexp(smooth_stack(len(ang), 20, 64, seed=8), e).astype(np.float32)

    def run():
        with session(64, 20, ang, proj, thickness=24) as s:
            s.reconstruct()
            return s.download()[0]
    want, got = both(monkeypatch, run)
    # results below the smallest normal number are rounded to its 2^-23
    tiny = 2.0 ** -148 * np.sqrt(want.size)
    assert np.linalg.norm(np.ldexp(got.astype(np.float64) - want, 100)) <= np.ldexp(TOL * np.linalg.norm(want.astype(np.float64)) + tiny, 100)
