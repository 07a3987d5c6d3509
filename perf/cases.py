"""The decode work that programs using this package do, as measurable cases.

A case is a dict of plain values; prepare() encodes its tiles from a seed
(synthetic H&E-like and fluorescence-like pixels, the distributions of the
package's own benchmark) and makes what a program keeps between calls (a
device plan, a server); run() is one pass through the public entry points and
returns the decoded pixels as byte tensors; work() counts the bytes a pass
cannot do without: each codestream read once, each pixel written once.

Fields of a case:
  entry     "call": codestreams in host memory through the drop-in
            (Codec.decode_tile*_to_device for one tile, decode_tiles_to_device
            for more), surfaces out; "plan": a device-resident plan replayed;
            "serve": requests submitted to a Server and collected
  coding    "ht" lossless 5/3, "lossy" 9/7 + ICT with HT blocks, "classic"
            lossless 5/3 with EBCOT blocks
  format    output pixel format
  tiles     tiles per pass; distinct: codestreams encoded for them (a batch
            repeats them, each at a place of its own in device memory)
  side      the largest tile side; mix: "uniform" tiles of side x side,
            "uneven" tiles of side, side/2, side/4, side/8, "ragged" tiles of
            any width and height from side/8 to side
  request   "full", "region", "scaled" (a quarter of the resolution) or
            "mixed" (60 % full, 25 % scaled, 15 % region)
  block     code-block side, 0 for 32 and 64 in turn
  tune      a long-lived plan's launch shapes are autotuned once
"""
import math

import numpy as np
import torch

from signinum_b200 import encode, j2k_cuda
from signinum_b200.j2k_cuda import BackendRequest, Codec, Downscale, PixelFormat, Rect, SgnRequest
from signinum_b200.plan import Plan
from signinum_b200.server import Server, collect

FORMATS = {"gray8": PixelFormat.Gray8, "rgb8": PixelFormat.Rgb8, "rgba8": PixelFormat.Rgba8,
           "gray16": PixelFormat.Gray16, "rgb16": PixelFormat.Rgb16}
# Coded bytes per pixel of the generated tiles (sigma 6; "mixed noise" where
# the tiles of a batch differ), measured once over each distribution.
CODED = {("ht", "rgb8"): 2.03, ("lossy", "rgb8"): 0.99, ("classic", "rgb8"): 1.90, ("ht", "gray8"): 0.65,
         ("lossy", "gray8"): 0.35, ("classic", "gray8"): 0.60, ("ht", "gray16"): 0.90, ("ht", "rgb16"): 3.6}
MIXED_NOISE = 1.1
REGION = 256  # side of a viewer's region request
MAX_OUTPUTS = 64


def case(name, entry, coding="ht", format="rgb8", tiles=1, distinct=1, side=512, mix="uniform", request="full",
         block=64, tune=False):
    return {"name": name, "entry": entry, "coding": coding, "format": format, "tiles": tiles, "distinct": distinct,
            "side": side, "mix": mix, "request": request, "block": block, "tune": tune}


def listed():
    return [
        # A viewer's single small tile through the drop-in: latency and launches.
        case("call_tile_256", "call", side=256),
        # A viewer's region of a large tile: the same call, most blocks pruned.
        case("call_region_of_1024", "call", side=1024, request="region", block=32),
        # A caller that hands over a batch of separate host buffers.
        case("call_uneven_32", "call", tiles=32, distinct=32, side=1024, mix="uneven", block=0),
        # The request stream of a tile server in a burst: full, reduced, region.
        case("serve_mixed_48", "serve", tiles=48, distinct=32, side=1024, mix="uneven", request="mixed", block=0),
        # One resident tile decoded again and again: the shortest device work.
        case("plan_tile_512", "plan"),
        # The uniform batch of the benchmark, handed on as one tensor.
        case("plan_uniform_256x512", "plan", tiles=256, distinct=16, tune=True),
        # The uneven batch of the benchmark (its headline): mixed sizes, noise,
        # block sizes, near-blank tiles.
        case("plan_uneven_1024", "plan", tiles=1024, distinct=48, side=1024, mix="uneven", block=0, tune=True),
        # High-bit-depth fluorescence tiles.
        case("plan_gray16_48x2048", "plan", format="gray16", tiles=48, distinct=3, side=2048, tune=True),
        # Lossy slides: 9/7, ICT.
        case("plan_lossy_128x512", "plan", coding="lossy", tiles=128, distinct=16),
        # Slides coded before HT: classic Tier-1.
        case("plan_classic_64x512", "plan", coding="classic", tiles=64, distinct=12),
        # Edge tiles of slides and cropped fields: odd widths and heights, RGBA.
        case("plan_ragged_rgba_60", "plan", format="rgba8", tiles=60, distinct=20, side=900, mix="ragged", block=0),
        # Overviews: a quarter of the resolution of large tiles.
        case("plan_scaled_64x1024", "plan", tiles=64, distinct=8, side=1024, request="scaled"),
    ]


def draw(rng):
    """One more case of the same ranges, its sizes spread over their logarithm."""
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    entry = rng.choice(["call", "plan", "plan", "plan", "serve"])
    coding = "ht" if entry == "serve" else rng.choice(["ht", "ht", "ht", "lossy", "classic"])
    if entry == "serve":
        fmt = "rgb8"
    elif coding == "ht":
        fmt = rng.choice(["rgb8", "rgb8", "rgba8", "gray8", "gray16", "rgb16"])
    else:
        fmt = rng.choice(["rgb8", "rgba8", "gray8"])
    mix = "uneven" if entry == "serve" else rng.choice(["uniform", "uneven", "ragged"])
    request = "mixed" if entry == "serve" else rng.choice(["full", "full", "full", "region", "scaled"])
    side = logint(300, 1024) if entry == "serve" or request == "region" else logint(100, 1600)
    if mix == "uneven":
        side = max(128, side - side % 8)
    # Total pixels: up to the listed cases' of the same kind.
    most = 16e6 if coding == "classic" or entry != "plan" else 150e6 if coding == "ht" else 33e6
    mean = side * side * {"uniform": 1.0, "uneven": 0.34, "ragged": 0.25}[mix]
    tiles = logint(1, max(1, min(600, most / mean)))
    if entry == "call":
        tiles = min(tiles, MAX_OUTPUTS)
    if entry == "serve":
        tiles = max(4, min(tiles, 60))
    distinct = max(1, min(tiles, int(5e6 / mean), 24))
    return {"entry": entry, "coding": coding, "format": fmt, "tiles": tiles, "distinct": distinct, "side": side,
            "mix": mix, "request": request, "block": rng.choice([0, 32, 64]), "tune": False}


# ---------------------------------------------------------------------------
# Tiles

def tile_specs(c):
    """(width, height, sigma or None for near-blank, levels, code-block exponent)
    of the distinct tiles.  A function of the case alone, so that inputs of
    another seed are other pixels and other codestreams of the same work."""
    n, side = c["distinct"], c["side"]
    r = np.random.default_rng(1234 + n + side)
    # Spread evenly over noise and size, then paired up at random.
    sigma = 30.0 * (r.permutation(n) + 0.5) / n
    blank = r.permutation(n) < n // 5
    u, v = (r.permutation(n) + 0.5) / n, (r.permutation(n) + 0.5) / n
    specs = []
    for k in range(n):
        if c["mix"] == "uniform":
            w = h = side
            s = 6.0
        elif c["mix"] == "uneven":
            w = h = side >> (k % 4)
            s = None if blank[k] else float(sigma[k])
        else:
            w, h = (max(1, int(round(side * 0.125 ** (1.0 - t)))) for t in (u[k], v[k]))
            s = float(sigma[k])
        if c["entry"] == "call" and c["tiles"] == 1:
            w = h = side
            s = 6.0
        if c["request"] in ("scaled", "mixed"):
            # A quarter of the resolution is offered for sides it divides.
            w, h = max(4, w - w % 4), max(4, h - h % 4)
        levels = 3 if max(w, h) < 200 else 4 if max(w, h) < 400 else 5 if max(w, h) < 800 or c["mix"] == "uniform" else 6
        if c["format"] == "gray16" and max(w, h) >= 1500:
            levels = 6
        block = c["block"] or (32 if (k // 4) % 2 else 64)
        specs.append((w, h, s, levels, 3 if block == 32 else 4))
    return specs


def pixels(seed, w, h, sigma, fmt):
    if fmt == "gray16":
        return encode.fluor_gray16(seed, w, h), 1, 16
    rgb = encode.blank_rgb8(seed, w, h) if sigma is None else encode.he_rgb8(seed, w, h, sigma)
    if fmt == "gray8":
        return np.ascontiguousarray(rgb.reshape(-1, 3)[:, 1]), 1, 8
    if fmt == "rgb16":  # twelve-bit colour
        low = np.random.default_rng(seed & 0xFFFFFFFF).integers(0, 16, rgb.size, dtype=np.uint16)
        return rgb.astype("<u2") * np.uint16(16) + low, 3, 12
    return rgb, 3, 8


def encode_tile(c, seed, spec):
    w, h, sigma, levels, cb = spec
    px, comps, depth = pixels(seed, w, h, sigma, c["format"])
    opts = {"levels": levels, "cb_exp": cb, "use_mct": comps == 3}
    if c["coding"] == "lossy":
        return encode.encode_irreversible(px, w, h, comps, depth, 1 / 256, **opts)
    if c["coding"] == "classic":
        return encode.encode_classic(px, w, h, comps, depth, **opts)
    return encode.encode_lossless(px, w, h, comps, depth, **opts)


def tile_requests(c, specs):
    """Per tile of a pass: (kind, region or None), a function of the case alone."""
    out = []
    for i in range(c["tiles"]):
        w, h = specs[i % len(specs)][:2]
        kind = c["request"]
        if kind == "mixed":
            kind = ("full", "scaled", "full", "region", "full", "scaled", "full", "full", "full", "scaled", "full",
                    "region", "full", "scaled", "full", "full", "scaled", "full", "region", "full")[i % 20]
        rect = None
        if kind == "region":
            rw, rh = min(REGION, w), min(REGION, h)
            rect = Rect((w - rw) * 3 // 7, (h - rh) * 5 // 9, rw, rh)
        out.append((kind, rect))
    return out


def out_dims(spec, request):
    kind, rect = request
    if kind == "region":
        return rect.w, rect.h
    d = 4 if kind == "scaled" else 1
    return -(-spec[0] // d), -(-spec[1] // d)


def work(c):
    specs = tile_specs(c)
    requests = tile_requests(c, specs)
    bpp = FORMATS[c["format"]].bytes_per_pixel()
    rate = CODED[(c["coding"], "rgb8" if c["format"] == "rgba8" else c["format"])]
    if c["mix"] != "uniform":
        rate *= MIXED_NOISE
    total = 0.0
    for i, rq in enumerate(requests):
        w, h = out_dims(specs[i % len(specs)], rq)
        # A reduced or cropped image needs about its own share of the coded bytes.
        total += w * h * (rate + bpp)
    return {"bytes": total, "flops": 0.0}


# ---------------------------------------------------------------------------
# State and pass

class Pixels:
    """A surface's device memory for torch; `owner` keeps it alive."""

    def __init__(self, raw, fmt, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {
            "shape": (raw.height, raw.width, FORMATS[fmt].bytes_per_pixel()), "typestr": "|u1",
            "data": (raw.device_ptr, False), "strides": None, "version": 3}


def tensor(raw, fmt, owner):
    return torch.as_tensor(Pixels(raw, fmt, owner), device="cuda")


def native_requests(requests):
    out = []
    for kind, rect in requests:
        r = SgnRequest()
        r.kind = {"full": 0, "region": 1, "scaled": 2}[kind]
        if rect is not None:
            r.x, r.y, r.w, r.h = rect.x, rect.y, rect.w, rect.h
        r.downscale = 4 if kind == "scaled" else 1
        out.append(r)
    return out


def prepare(c, seed):
    specs = tile_specs(c)
    with encode._pool() as ex:
        coded = list(ex.map(lambda k: encode_tile(c, encode._mix(seed, 77, k), specs[k]), range(len(specs))))
    st = {"case": c, "requests": tile_requests(c, specs)}
    tiles = [coded[i % len(coded)] for i in range(c["tiles"])]
    if c["entry"] == "call":
        st["tiles"] = [bytes(bytearray(t)) for t in tiles]  # a host buffer of its own per tile
        st["native"] = None if c["request"] == "full" else native_requests(st["requests"])
    elif c["entry"] == "serve":
        st["server"] = Server(device_budget_bytes=2 << 30, resident_capacity_bytes=256 << 20)
        ids = [st["server"].register(t) for t in coded]
        st["ids"] = [ids[i % len(ids)] for i in range(c["tiles"])]
    else:
        fmt = FORMATS[c["format"]]
        plan = Plan(tiles, fmt, None if c["request"] == "full" else native_requests(st["requests"]))
        if c["tune"]:
            plan.autotune()
        st["plan"] = plan
        st["views"] = [tensor(s, c["format"], plan) for s in plan.surfaces()]
        if len(tiles) > MAX_OUTPUTS:
            # The batch handed on as one tensor, gathered on the plan's stream.
            st["stream"] = torch.cuda.ExternalStream(plan.ctx.stream())
            st["flat"] = [v.reshape(-1) for v in st["views"]]
            st["batch"] = torch.empty(sum(v.numel() for v in st["views"]), dtype=torch.uint8, device="cuda")
    return st


def run(st):
    c = st["case"]
    fmt = FORMATS[c["format"]]
    if c["entry"] == "plan":
        st["plan"].execute_async()
        if "batch" not in st:
            return st["views"]
        with torch.cuda.stream(st["stream"]):
            torch.cat(st["flat"], out=st["batch"])
        return st["batch"]
    if c["entry"] == "serve":
        server = st["server"]
        tickets = [server.submit(tid, fmt, rect, Downscale.Quarter if kind == "scaled" else None)
                   for tid, (kind, rect) in zip(st["ids"], st["requests"])]
        results = collect(server, tickets)
        return [tensor(results[t].surface._raw, c["format"], results[t].surface) for t in tickets]
    if c["tiles"] == 1:
        kind, rect = st["requests"][0]
        data = st["tiles"][0]
        if kind == "region":
            s = Codec.decode_tile_region_to_device(data, fmt, rect, BackendRequest.Cuda)
        elif kind == "scaled":
            s = Codec.decode_tile_scaled_to_device(data, fmt, Downscale.Quarter, BackendRequest.Cuda)
        else:
            s = Codec.decode_tile_to_device(data, fmt, BackendRequest.Cuda)
        return [tensor(s._raw, c["format"], s)]
    surfaces = Codec.decode_tiles_to_device(st["tiles"], fmt, BackendRequest.Cuda, st["native"])
    return [tensor(s._raw, c["format"], s) for s in surfaces]


def exact(c, seed):
    """Decoded pixels are whole numbers, equal from run to run; there is no
    64-bit form of them."""
    return None
