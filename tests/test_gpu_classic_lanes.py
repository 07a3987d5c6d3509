"""Classic (EBCOT) plans of enough code blocks that the lanes of a warp decode
different blocks: 1, 8, 17 and 18 blocks per warp with the column words in
shared memory and 32 in scratch (on 148 SMs), blocks of partial stripes and
columns, styles' transitions, lossless against the source pixels.  Other lane
counts, and damaged streams, run in the CPU emulation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,cb,cb_h,style", [
    (64, 64, 0, 0, 0),      # 4 x 4, 768 blocks: one lane
    (257, 131, 0, 0, 0),    # 6,729 blocks, ragged edges: eight lanes
    (509, 303, 0, 0, 0x08),   # 29,280 blocks: 32 lanes, words in scratch, vertically causal
    (509, 303, 0, 1, 0x05),   # 4 x 8, 17 lanes, bypass and termination on every pass
    (640, 253, 1, 0, 0x22),   # 8 x 4, 18 lanes, context reset and segmentation symbols
    (333, 1023, 4, 4, 0x2F),  # 64 x 64, one lane, every style at once
])
def test_many_blocks_lossless(w, h, cb, cb_h, style):
    from signinum_b200 import encode
    from signinum_b200.j2k_cuda import BackendRequest, Codec, PixelFormat

    px = encode.he_rgb8(97 * w + h, w, h, 9.0)
    cs = encode.encode_classic(px, w, h, 3, 8, style=style, levels=3, cb_exp=cb, cb_exp_h=cb_h)
    s = Codec.decode_tile_to_device(cs, PixelFormat.Rgb8, BackendRequest.Cuda)
    assert np.array_equal(np.frombuffer(s.to_bytes(), np.uint8), px)


def test_large_and_many_small_blocks_in_one_plan():
    """A 64 x 64 block sets the slot size of a plan whose 29,000 small blocks
    then exceed what shared memory holds at once."""
    from signinum_b200 import encode
    from signinum_b200.j2k_cuda import BackendRequest, Codec, PixelFormat

    tiles, pixels = [], []
    for w, h, cb, levels in ((64, 64, 4, 0), (509, 303, 0, 2), (130, 70, 4, 1)):
        px = encode.he_rgb8(w + h, w, h, 5.0)
        tiles.append(encode.encode_classic(px, w, h, 3, 8, levels=levels, cb_exp=cb))
        pixels.append(px)
    for s, px in zip(Codec.decode_tiles_to_device(tiles, PixelFormat.Rgb8, BackendRequest.Cuda), pixels):
        assert np.array_equal(np.frombuffer(s.to_bytes(), np.uint8), px)
