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
