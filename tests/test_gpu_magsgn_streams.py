"""MagSgn streams at the edges of the unstuffing steps: runs of 0xFF bytes at
every place of a lane's eight bytes and across steps, streams of a few bytes
and of several steps, one block per warp (64 wide), two per warp (32 wide and
narrower), at every alignment the codestream gives them.  Lossless, against
the source pixels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def dense_ones(rng, w, h, share, depth):
    """Samples whose magnitude and sign bits are mostly ones: minus a power of
    two around the DC level (sign 1, magnitude - 1 all ones), the rest noise."""
    mid = 1 << (depth - 1)
    px = np.full(w * h, mid - (mid >> 1), np.int64)
    px[rng.random(w * h) < 0.3] = mid - (mid >> 3)
    noise = rng.random(w * h) >= share
    px[noise] = rng.integers(0, 1 << depth, int(noise.sum()))
    return px.astype(np.uint8 if depth == 8 else "<u2")


@pytest.mark.parametrize("share", [0.0, 0.5, 0.97, 1.0])
@pytest.mark.parametrize("w,h,cb,depth", [
    (64, 64, 4, 8), (65, 37, 4, 16), (193, 130, 4, 12),  # 64 wide: a warp per block
    (32, 32, 3, 8), (161, 67, 3, 16),                    # 32 wide: half a warp
    (7, 5, 2, 8), (50, 41, 1, 12), (19, 33, 0, 8),       # streams of a few bytes
])
def test_dense_ff_streams_lossless(w, h, cb, depth, share):
    from signinum_b200 import encode
    from signinum_b200.j2k_cuda import BackendRequest, Codec, PixelFormat

    rng = np.random.default_rng(w * 1000 + h + int(100 * share))
    tiles, pixels = [], []
    for levels in (0, 0, 1):
        px = dense_ones(rng, w, h, share, depth)
        tiles.append(encode.encode_lossless(px, w, h, 1, depth, levels=levels, cb_exp=cb, use_mct=False))
        pixels.append(px)
    fmt = PixelFormat.Gray8 if depth == 8 else PixelFormat.Gray16
    for s, px in zip(Codec.decode_tiles_to_device(tiles, fmt, BackendRequest.Cuda), pixels):
        assert s.to_bytes() == px.tobytes()
    # The two-kernel form (small plans run the fused one).
    from signinum_b200.plan import Plan

    plan = Plan(tiles, fmt)
    plan.set_cleanup_form(0)
    plan.execute_async()
    assert plan.wait()[0] == 0
    for i, px in enumerate(pixels):
        assert plan.download(i) == px.tobytes()
