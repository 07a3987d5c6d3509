"""Levels at the edges of the DWT kernels' strips (128 columns reversible, 120
irreversible) and row pairs: widths on either side of a whole strip, widths of
one to five, heights of one to three and on either side of a unit, aligned and
unaligned rows; lossless against the source pixels, lossy and regions against
the oracle."""
import numpy as np
import pytest

from signinum_b200 import BackendRequest, Codec, PixelFormat, Rect, encode
from tests.test_gpu_decode import cpu

pytestmark = pytest.mark.gpu

WIDTHS = (1, 2, 3, 4, 5, 119, 120, 121, 127, 128, 129, 130, 132, 240, 241, 254, 255, 256, 257, 260, 384, 509)
HEIGHTS = (1, 2, 3, 4, 63, 64, 65, 130)


def pixels(rng, w, h, comps):
    return rng.integers(0, 256, w * h * comps).astype(np.uint8)


@pytest.mark.parametrize("comps", [1, 3])
@pytest.mark.parametrize("h", HEIGHTS)
def test_reversible_edges(h, comps):
    rng = np.random.default_rng(100 * h + comps)
    px = [pixels(rng, w, h, comps) for w in WIDTHS]
    for levels in (1, 2):
        tiles = [encode.encode_lossless(p, w, h, comps, 8, levels=levels, use_mct=comps == 3)
                 for w, p in zip(WIDTHS, px)]
        fmt = PixelFormat.Gray8 if comps == 1 else PixelFormat.Rgb8
        for w, p, s in zip(WIDTHS, px, Codec.decode_tiles_to_device(tiles, fmt, BackendRequest.Cuda)):
            assert s.to_bytes() == p.tobytes(), (w, h, levels)
        if comps == 3:
            for w, p, s in zip(WIDTHS, px, Codec.decode_tiles_to_device(tiles, PixelFormat.Rgba8, BackendRequest.Cuda)):
                got = np.frombuffer(s.to_bytes(), np.uint8).reshape(-1, 4)
                assert np.array_equal(got[:, :3].reshape(-1), p) and (got[:, 3] == 255).all(), (w, h, levels)


@pytest.mark.parametrize("comps", [1, 3])
@pytest.mark.parametrize("h", HEIGHTS)
def test_irreversible_edges(h, comps):
    rng = np.random.default_rng(100 * h + comps + 7)
    fmt = PixelFormat.Gray8 if comps == 1 else PixelFormat.Rgb8
    tiles = [encode.encode_irreversible(pixels(rng, w, h, comps), w, h, comps, 8, levels=2, use_mct=comps == 3)
             for w in WIDTHS]
    for w, cs, s in zip(WIDTHS, tiles, Codec.decode_tiles_to_device(tiles, fmt, BackendRequest.Cuda)):
        assert s.to_bytes() == cpu(cs, fmt)[0], (w, h)


@pytest.mark.parametrize("lossy", [False, True])
def test_regions_across_strips(lossy):
    rng = np.random.default_rng(9 + lossy)
    w, h = 523, 201
    px = pixels(rng, w, h, 3)
    cs = encode.encode_irreversible(px, w, h, 3, 8, levels=3) if lossy else encode.encode_lossless(px, w, h, 3, 8, levels=3)
    full = np.frombuffer(cpu(cs, PixelFormat.Rgb8)[0], np.uint8).reshape(h, w, 3)
    for x, y, rw, rh in ((0, 0, 128, 64), (119, 63, 10, 3), (120, 1, 121, 65), (127, 0, 2, 201), (383, 130, 140, 71),
                         (522, 200, 1, 1), (1, 7, 509, 40)):
        s = Codec.decode_tile_region_to_device(cs, PixelFormat.Rgb8, Rect(x, y, rw, rh), BackendRequest.Cuda)
        assert np.array_equal(np.frombuffer(s.to_bytes(), np.uint8).reshape(rh, rw, 3), full[y:y + rh, x:x + rw])
