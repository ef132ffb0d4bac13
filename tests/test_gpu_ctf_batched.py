"""Batched strips of the GPU phase flip against the oracle's restatement of
apps/ctfphaseflip/src/main.rs, at the sizes where the batching has edges: rows
that do not fill a CTA, lengths with prime radices above 7, several chunks of
views, a view whose strips exceed a chunk, a tilt axis along which the strip
index runs against x.

Tolerance: rel-L2 <= 1e-5 of the corrected stack -- FFTs of at most 1000 samples
in each direction, whose rounding in f32 grows with sqrt(log2 n) * 2^-24 per
transform (about 1e-6 for four of them), with prime radices up to 61 summed term
by term (sqrt(61) * 2^-24 each).
"""
import numpy as np
import pytest

import oracle as O
import tiltgpu as T
from test_gpu_ctf import stack
from tgutil import rel_l2

pytestmark = pytest.mark.gpu

CASES = [
    (dict(pixel_size=2.0, strip_width=33), (2, 17, 99)),                        # 3 * 11 columns; 17 rows: one over a CTA's 16
    (dict(pixel_size=2.0, strip_width=26), (3, 122, 130)),                      # 2 * 13 by 2 * 61
    (dict(pixel_size=2.0, strip_width=1), (2, 9, 20)),                          # one-sample rows
    (dict(pixel_size=2.0, strip_width=64), (45, 200, 256)),                     # chunks of 40 and 5 views
    (dict(pixel_size=2.0, strip_width=4, tilt_axis_angle=45.0), (2, 300, 300)),  # several chunks within a view
    (dict(pixel_size=1.5, strip_width=16, tilt_axis_angle=100.0), (2, 75, 64)),
    (dict(pixel_size=1.0, strip_width=256, defocus=-100.0), (1, 1000, 600)),    # fewer rows per CTA
]


@pytest.mark.parametrize("kw,shape", CASES)
def test_batched_strips_vs_oracle(kw, shape):
    st_in = stack(*shape, seed=shape[1])
    ang = np.linspace(-50, 50, shape[0]).astype(np.float32)
    out, stats = T.ctf_phaseflip(st_in, ang, **kw)
    okw = dict(kw)
    okw["pixel_a"] = okw.pop("pixel_size")
    want, wst = O.ctfphaseflip(O.CtfParams(**okw), st_in, ang)
    assert rel_l2(out, want) <= 1e-5, rel_l2(out, want)
    for k in ("amin", "amax", "amean"):
        assert stats[k] == pytest.approx(wst[k], rel=1e-5, abs=1e-6)
