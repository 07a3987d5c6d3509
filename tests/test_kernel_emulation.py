"""The decode kernels' CUDA source run on CPU threads (tests/kernel_emu):
every HT, classic (EBCOT), IDWT and pack kernel on the golden fixtures and
on seeded random reversible, irreversible and classic codestreams, built with AddressSanitizer, and
compared with the oracle (coefficients per code block, then pixels, exact).
The classic kernel runs as it is launched: CTAs of one warp with 1, 5 or as
many blocks in flight as its shared pool holds, and with 24 and 32 blocks
whose column words are in scratch.  Out-of-bounds accesses and parity breaks
show up here without a GPU.  Three helpers that are inline PTX on the device
(the warp scan, the predicated load, the saturating pack) run their C++ forms
here; the PTX forms are compared by the GPU tests alone."""
import json
import pathlib
import shutil
import subprocess
import sys

import numpy as np
import pytest

from tests.helpers import (WIDE_BLOCKS, precinct_codestream, random_classic, random_codestream, random_irreversible,
                           wide_block_codestream)

EMU = pathlib.Path(__file__).parent / "kernel_emu"
ROOT = EMU.parents[1]
CSRC = ROOT / "signinum_b200" / "csrc"

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    out = tmp_path_factory.mktemp("kernel_emu")
    subprocess.run([sys.executable, str(EMU / "make_sources.py"), str(out)], check=True)
    flags = ["g++", "-std=c++20", "-O1", "-fsanitize=address", "-ffp-contract=off", f"-I{EMU}", f"-I{CSRC}",
             f"-I{ROOT / 'oracle'}"]
    units = [out / "ht_decode_emu.cpp", out / "idwt_pack_emu.cpp", out / "classic_emu.cpp", EMU / "emu_main.cpp",
             CSRC / "host" / "codestream.cpp",
             ROOT / "oracle" / "oracle.cpp", ROOT / "oracle" / "oracle_ht.cpp", ROOT / "oracle" / "oracle_ebcot.cpp",
             ROOT / "oracle" / "oracle_capi.cpp"]
    procs = [subprocess.Popen(flags + ["-c", str(u), "-o", str(out / (u.stem + ".o"))]) for u in units]
    assert all(p.wait() == 0 for p in procs)
    subprocess.run(flags + ["-o", str(out / "emu")] + [str(out / (u.stem + ".o")) for u in units] + ["-lpthread"],
                   check=True)
    return out


def run(emu, fmts, codestreams, options=(), timeout=600):
    paths = []
    for k, cs in enumerate(codestreams):
        p = emu / f"case_{fmts}_{k}.j2k"
        p.write_bytes(cs)
        paths.append(str(p))
    r = subprocess.run([str(emu / "emu"), fmts, *options] + paths, capture_output=True, text=True, timeout=timeout)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    assert r.stdout.strip().endswith("fails 0")


def test_golden_fixtures_through_emulated_kernels(emu):
    fx = json.loads((pathlib.Path(__file__).parent / "golden" / "openhtj2k.json").read_text())["fixtures"]
    run(emu, "03", [bytes.fromhex(f["j2k_hex"]) for f in fx.values()])


@pytest.mark.parametrize("kind", ["reversible", "irreversible", "classic"])
def test_random_codestreams_through_emulated_kernels(emu, kind):
    rng = np.random.default_rng({"reversible": 31, "irreversible": 97, "classic": 7}[kind])
    make = {"reversible": random_codestream, "irreversible": random_irreversible, "classic": random_classic}[kind]
    by_comps = {1: [], 3: []}
    while len(by_comps[1]) < 4 or len(by_comps[3]) < 4:
        cs, _, _, _, comps, _ = make(rng, max_side=100)
        by_comps[comps].append(cs)
    run(emu, "03", by_comps[1])  # Gray8, Gray16
    run(emu, "124", by_comps[3])  # Rgb8, Rgba8, Rgb16


def test_wide_code_blocks_through_emulated_kernels(emu):
    """HT blocks wider or higher than 64 (the VLC and MagSgn kernels' wide
    paths) under AddressSanitizer."""
    rng = np.random.default_rng(4200)
    by_comps = {1: [], 3: []}
    for cb in WIDE_BLOCKS:
        cs, _, _, _, comps, _ = wide_block_codestream(rng, cb, max_w=160, max_h=72)
        by_comps[comps].append(cs)
    if by_comps[1]:
        run(emu, "03", by_comps[1])
    if by_comps[3]:
        run(emu, "124", by_comps[3])


@pytest.mark.parametrize("kind", ["ht", "classic", "lossy"])
def test_precinct_partitions_through_emulated_kernels(emu, kind):
    """Precinct partitions through the product's host parser (which builds
    the job tables) and the emulated kernels."""
    rng = np.random.default_rng({"ht": 4400, "classic": 4401, "lossy": 4402}[kind])
    by_comps = {1: [], 3: []}
    while len(by_comps[1]) < 3 or len(by_comps[3]) < 3:
        cs, _, _, _, comps = precinct_codestream(rng, kind, max_side=90)
        by_comps[comps].append(cs)
    run(emu, "03", by_comps[1])
    run(emu, "124", by_comps[3])


def test_interior_strips_through_emulated_kernels(emu):
    """Levels wide enough for strips with no edge column (the 5/3 lifting's
    interior form: a strip from column 128 on that ends at least two columns
    before the level's edge), lossless RGB and gray, under AddressSanitizer."""
    from signinum_b200 import encode
    from tests.helpers import random_tile

    rng = np.random.default_rng(4500)
    by_comps = {1: [], 3: []}
    for w, h, comps, levels in [(300, 14, 3, 0), (390, 9, 3, 1), (517, 6, 1, 2), (640, 11, 3, 2), (259, 20, 1, 1)]:
        bd = 8 if comps == 3 else 12
        px = random_tile(rng, w, h, comps, bd, int(rng.integers(0, 2)))
        by_comps[comps].append(encode.encode_lossless(px.reshape(-1).view(np.uint8), w, h, comps, bd, levels=levels,
                                                      cb_exp=4, cb_exp_h=3))
    run(emu, "03", by_comps[1])
    run(emu, "124", by_comps[3])


@pytest.mark.parametrize("style", [0x00, 0x01, 0x02, 0x04, 0x05, 0x08, 0x2F])
def test_damaged_classic_segments_through_emulated_kernels(emu, style):
    """FF 80 .. FF 8F at the start of codeword segments and inside them: the
    MQ decoder's C register underflows there, and an iteration of the kernel
    that codes no sample must leave the decoder as it is all the same.
    Coefficients and pixels equal the oracle's; the time limit fails a decoder
    that such a pair sends into a loop."""
    from signinum_b200 import encode
    from tests.helpers import random_tile

    rng = np.random.default_rng(4600 + style)
    streams = []
    for w, h, cb, cb_h, levels in [(24, 24, 4, 4, 0), (33, 18, 3, 1, 0), (40, 29, 2, 2, 1), (9, 70, 0, 4, 0),
                                   (130, 7, 6, 2, 0), (64, 64, 4, 4, 0)]:
        px = random_tile(rng, w, h, 1, 8, int(rng.integers(0, 2)))
        streams.append(encode.encode_classic(px.reshape(-1), w, h, 1, 8, style=style, levels=levels, cb_exp=cb,
                                             cb_exp_h=cb_h))
    for seed in (1, 100):
        run(emu, "0", streams, ["-d", str(seed)], timeout=60)


@pytest.mark.parametrize("seed", [10, 20, 30])
def test_damaged_cleanup_segments_through_emulated_kernels(emu, seed):
    """Damaged HT blocks, most of odd width, one and two per warp: where the
    oracle decodes the damaged codestream the coefficients and pixels equal
    its, also where the damage makes samples right of the block's last column
    significant (which take no bits of the MagSgn stream); where it rejects the
    codestream the kernels do so too."""
    from signinum_b200 import encode
    from tests.helpers import random_tile

    rng = np.random.default_rng(4700)
    streams = []
    for w, h, bd, cb in [(65, 16, 16, 4), (63, 12, 16, 4), (33, 9, 16, 3), (31, 14, 12, 3), (9, 7, 8, 1), (129, 8, 16, 5),
                         (7, 30, 16, 3), (13, 13, 16, 2), (65, 30, 16, 4), (67, 8, 12, 2)]:
        px = random_tile(rng, w, h, 1, bd, 1)
        streams.append(encode.encode_lossless(px.reshape(-1).view(np.uint8), w, h, 1, bd, levels=0, cb_exp=cb, cb_exp_h=3,
                                              use_mct=False))
    run(emu, "0", streams, ["-d", str(seed)])
