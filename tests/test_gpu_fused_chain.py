"""The fused cleanup kernel's chain (small plans) at the edges of its VLC bit
array and MEL runs: blocks of every width class up to 64 and beyond, one to a
few rows, near-blank content (long MEL runs), noise (many VLC bytes, few runs)
and bytes above 0x8F before all-ones bytes, against the two-kernel form and
the source pixels."""
import numpy as np
import pytest

from signinum_b200 import PixelFormat, encode
from signinum_b200.plan import Plan

pytestmark = pytest.mark.gpu

SHAPES = [(64, 64, 4, 4), (63, 61, 4, 4), (33, 9, 4, 4), (1, 1, 4, 4), (2, 1, 4, 4), (3, 65, 0, 8), (5, 200, 1, 7),
          (32, 32, 3, 3), (17, 3, 3, 3), (62, 64, 4, 4), (128, 32, 5, 3), (200, 16, 6, 2)]


@pytest.mark.parametrize("amplitude", [0, 1, 2, 9, 255])
def test_fused_chain_matches_two_kernels(amplitude):
    rng = np.random.default_rng(500 + amplitude)
    for w, h, cb, cb_h in SHAPES:
        # Sparse: most samples at one value; dense: every sample random.
        px = np.full(w * h, 128, np.int64)
        pick = rng.random(w * h) < (0.05 if amplitude in (1, 9) else 1.0)
        px[pick] += rng.integers(-amplitude, amplitude + 1, int(pick.sum()))
        px = px.clip(0, 255).astype(np.uint8)
        tiles = [encode.encode_lossless(px, w, h, 1, 8, levels=levels, cb_exp=cb, cb_exp_h=cb_h, use_mct=False)
                 for levels in (0, 1)]
        plan = Plan(tiles, PixelFormat.Gray8)
        for form in (1, 0):
            plan.set_cleanup_form(form)
            plan.execute_async()
            assert plan.wait()[0] == 0
            for i in range(len(tiles)):
                assert plan.download(i) == px.tobytes(), (w, h, cb, cb_h, form, i)
