"""Pinned tile shapes: tg_session_set_variant and TG_BP_VARIANT on series that take the
tensor-core back-projector by themselves."""
import numpy as np
import pytest

import tiltgpu as T
from tgutil import angles, rel_l2, smooth_stack

pytestmark = pytest.mark.gpu
TENSOR = "tcgen05-hex126"
NX, NY, TH = 256, 256, 96
ANG = angles(-60, 60, 3)


def make(**kw):
    s = T.Session(NX, NY, len(ANG), ANG, thickness=TH, **kw)
    s.upload(smooth_stack(len(ANG), NY, NX, seed=11))
    return s


def tensor(s):
    return s.kernel_info()["variant_name"].startswith(TENSOR)


def run(s):
    s.reconstruct()
    return s.download()


@pytest.mark.parametrize("kw", [{}, dict(sirt=2, sirt_relax=0.3), dict(xtilt=np.full(len(ANG), 1.0, np.float32))])
def test_set_variant_pins_the_named_tile_shape(kw, monkeypatch):
    with make(**kw) as s:
        assert tensor(s)
        first, st = run(s)
        bytes0 = s.device_bytes()
        monkeypatch.setenv("TG_BP_VARIANT", "3")
        with make(**kw) as p:
            want, wst = run(p)
            name = p.kernel_info()["variant_name"]
        monkeypatch.delenv("TG_BP_VARIANT")
        s.set_variant(3)
        assert s.kernel_info()["variant_name"] == name and not tensor(s) and s.kernel_info()["variant"] == 3
        got, gst = run(s)
        np.testing.assert_array_equal(got, want)
        assert gst == wst and rel_l2(first, want) <= 1e-5
        for auto in (-1, 14):  # by itself again, or by name
            s.set_variant(auto)
            assert tensor(s) and s.device_bytes() == bytes0
            again, ast = run(s)
            np.testing.assert_array_equal(again, first)
            assert ast == st
            s.set_variant(3)
            np.testing.assert_array_equal(run(s)[0], want)


def test_set_variant_between_batched_runs():
    kw = dict(sirt=2, sirt_relax=0.3)
    with make(**kw) as a, make(**kw) as c:
        first, _ = run(a)
        c.set_variant(3)
        want, _ = run(c)
        b = T.Batch()
        b.add(a)
        b.add(c)
        for va, vc in ((14, 3), (3, 14), (14, 14), (3, 3)):
            a.set_variant(va)
            c.set_variant(vc)
            b.reconstruct()
            for s, v in ((a, va), (c, vc)):
                np.testing.assert_array_equal(s.download()[0], first if v == 14 else want)
        b.close()


@pytest.mark.parametrize("env,want", [("14", True), ("15", True), ("99", True), ("-1", True), ("0", False), ("13", False)])
def test_environment_names_a_kernel_or_is_ignored(env, want, monkeypatch):
    monkeypatch.setenv("TG_BP_VARIANT", env)
    with make() as s:
        assert tensor(s) == want


def test_what_is_no_variant_is_refused():
    with make() as s, make(storage="fp16") as h:
        for v in (-2, 15):
            with pytest.raises(T.TiltGpuError):
                s.set_variant(v)
        with pytest.raises(T.TiltGpuError):
            h.set_variant(14)
