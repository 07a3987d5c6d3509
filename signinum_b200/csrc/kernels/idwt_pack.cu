// Inverse reversible 5/3 DWT and the fused last level + inverse RCT + DC
// shift + pixel pack, on sm_100a.
//
// Arithmetic follows the reference exactly: per level, interleave the four
// sub-bands, then the horizontal lifting pass (update even samples with
// floor((l + r) / 4 + 1/2), then predict odd samples with floor((l + r) / 2)),
// then the vertical pass (crates/signinum-j2k-native/src/j2c/idwt.rs:535-555,
// :741-765, :972-1014), with periodic symmetric extension at the edges
// (:908-925).  All values are integers, so int32 with arithmetic shifts gives
// the reference's f32 floors bit for bit.
//
// Mapping: one warp per unit = a strip of 128 columns x `seg` rows of a level.
// Lane k owns image columns 4k .. 4k+3 of the strip, i.e. band columns 2k and
// 2k+1 of the low and high bands, read as 8-byte pairs, so every band load
// and every row store is coalesced.  Horizontal lifting of a row needs the
// odd neighbour on the left and the updated even neighbour on the right: both
// come from warp shuffles (the strip's edge lanes load the extra band samples
// they need).  The vertical pass streams down the rows keeping the previous
// odd row and the previous updated even row in registers.  Symmetric
// extension is done by reflecting row/column indices (it commutes with the
// lifting steps): the lanes' column offsets are reflected once per unit, so
// the edges run the same code.  No barriers.
//
// The last level keeps the streams of all components of a pixel in the same
// lane and finishes the pixels there: inverse RCT (mct.rs:117-150),
// +2^(bd-1) (decode.rs:1720-1729, :1748-1752) and the conversion to the
// requested pixel format (crates/signinum-j2k-native/src/lib.rs:1772-1840,
// :2202-2294; crates/signinum-j2k/src/decode.rs:345-356, :517-545); each lane
// packs its four pixels into 32-bit words and stores them itself, or through
// the warp's row buffer where the row does not fall on lane boundaries.
#include <algorithm>
#include <cstdint>
#include <cstring>

#include "../device_plan.h"
#include "kernels.h"

namespace sgn {
namespace {

constexpr int kLanes = 32;
static_assert(kIdwtStripW == 4 * kLanes, "one strip is four columns per lane");

// Whole-sample symmetric extension of index i into [0, n).  Reflection keeps
// an index's parity; indices far outside (columns of lanes past a narrow
// level) end at the nearest in-range index of the same parity, so the band
// they select (low for even, high for odd) and the place in it stay in bounds.
__device__ __forceinline__ int reflect(int i, int n) {
  if ((unsigned)i < (unsigned)n) return i;
  if (n == 1) return 0;
#pragma unroll 1
  for (int k = 0; k < 4 && (unsigned)i >= (unsigned)n; ++k) i = i < 0 ? -i : 2 * (n - 1) - i;
  if (i < 0) return i & 1;
  if (i >= n) return (n - 1) - (((n - 1) ^ i) & 1);
  return i;
}

struct Bands {
  const int32_t* ll;
  const int32_t* hl;
  const int32_t* lh;
  const int32_t* hh;
};

// Whether every band row of a level of width w starts 8-byte aligned.
__device__ __forceinline__ bool aligned_bands(const Bands& B, int w) {
  const uintptr_t a = (uintptr_t)B.ll | (uintptr_t)B.hl | (uintptr_t)B.lh | (uintptr_t)B.hh;
  return (w & 3) == 0 && (a & 7) == 0;
}

// A lane's columns of a level: band offsets of its image columns c .. c+3
// (low band l0, l1; high band h0, h1), and of the samples the strip's edge
// lanes need besides: lane 0 the high band left of its columns (xh), lane 31
// the low and high band right of them (xl, xh).  Whole strips of a level
// whose rows are 8-byte aligned (VEC) read the pairs with one load each; at
// the level's edges their extra samples are among the lane's own.
struct Cols {
  int w, h;
  int l0, l1, h0, h1, xl, xh;
  bool left, right;  // VEC: lane 0 (31) has a sample to load on its left (right)
};

// *p where `go` holds, else 0: a predicated load, so that the loads around it
// stay in one batch.
__device__ __forceinline__ int load_if(bool go, const int32_t* p) {
#ifdef __CUDA_ARCH__
  int v;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\tmov.b32 %0, 0;\n\t@p ld.global.nc.b32 %0, [%1];\n\t}"
      : "=r"(v)
      : "l"(p), "r"((uint32_t)go));
  return v;
#else
  return go ? *p : 0;
#endif
}

template <bool VEC>
__device__ __forceinline__ Cols make_cols(int x0, int w, int h, int lane) {
  Cols o;
  const int c = x0 + 4 * lane;
  o.w = w;
  o.h = h;
  if (VEC) {
    o.l0 = o.h0 = c >> 1;
    o.l1 = o.h1 = 0;
    o.left = lane == 0 && x0 > 0;
    o.right = lane == kLanes - 1 && x0 + kIdwtStripW < w;
    o.xl = 2;
    o.xh = o.left ? -1 : 2;  // from the pair
  } else {
    o.l0 = reflect(c, w) >> 1;
    o.h0 = reflect(c + 1, w) >> 1;
    o.l1 = reflect(c + 2, w) >> 1;
    o.h1 = reflect(c + 3, w) >> 1;
    o.xl = reflect(c + 4, w) >> 1;
    o.xh = reflect(lane == 0 ? c - 1 : c + 5, w) >> 1;
    o.left = o.right = false;
  }
  return o;
}

// Band samples of one interleaved row at this lane's columns.  Loads only:
// lifting happens in lift_row, so a caller can keep the next rows' loads in
// flight while it lifts the current ones.
struct RawRow {
  int lo0, lo1, hi0, hi1;  // low / high band at columns c, c+2 / c+1, c+3
  int xl, xh;              // edge lanes: Cols::xl, Cols::xh
};

// Row r of the low and the high band.
template <bool VEC>
__device__ __forceinline__ RawRow load_row(const int32_t* low, const int32_t* high, int r, const Cols& o, int lane) {
  const int32_t* Lr = low + (size_t)r * ((o.w + 1) >> 1);
  const int32_t* Hr = high + (size_t)r * (o.w >> 1);
  RawRow R;
  if (VEC) {
    Lr += o.l0;
    Hr += o.h0;
    const int2 l = __ldg(reinterpret_cast<const int2*>(Lr));
    const int2 h = __ldg(reinterpret_cast<const int2*>(Hr));
    R.lo0 = l.x;
    R.lo1 = l.y;
    R.hi0 = h.x;
    R.hi1 = h.y;
    R.xh = load_if(o.left || o.right, Hr + o.xh);
    R.xl = load_if(o.right, Lr + 2);
    return R;
  }
  R.lo0 = __ldg(Lr + o.l0);
  R.lo1 = __ldg(Lr + o.l1);
  R.hi0 = R.hi1 = R.xl = R.xh = 0;
  if (o.w > 1) {
    R.hi0 = __ldg(Hr + o.h0);
    R.hi1 = __ldg(Hr + o.h1);
    if (lane == 0 || lane == kLanes - 1) {
      R.xh = __ldg(Hr + o.xh);
      R.xl = __ldg(Lr + o.xl);
    }
  }
  return R;
}

// Horizontal lifting of a loaded row: samples of the lane's image columns
// c .. c+3.  Columns past the right edge return garbage.
template <bool VEC>
__device__ __forceinline__ int4 lift_row(const RawRow& R, const Cols& o, int lane) {
  if (!VEC && o.w == 1) return make_int4(R.lo0, 0, 0, 0);
  int hm1 = __shfl_up_sync(0xFFFFFFFFu, R.hi1, 1);  // X[c-1]
  if (lane == 0) hm1 = !VEC || o.left ? R.xh : R.hi0;  // (X[-1] is X[1])
  const int e0 = R.lo0 - ((hm1 + R.hi0 + 2) >> 2);     // X[c]
  const int e1 = R.lo1 - ((R.hi0 + R.hi1 + 2) >> 2);   // X[c+2]
  int e2 = __shfl_down_sync(0xFFFFFFFFu, e0, 1);       // X[c+4]
  if (lane == kLanes - 1) e2 = !VEC || o.right ? R.xl - ((R.hi1 + R.xh + 2) >> 2) : e1;  // (X[w] is X[w-2])
  return make_int4(e0, R.hi0 + ((e0 + e1) >> 1), e1, R.hi1 + ((e1 + e2) >> 1));
}

__device__ __forceinline__ int4 vupdate(int4 xe, int4 a, int4 c) {
  return make_int4(xe.x - ((a.x + c.x + 2) >> 2), xe.y - ((a.y + c.y + 2) >> 2), xe.z - ((a.z + c.z + 2) >> 2),
                   xe.w - ((a.w + c.w + 2) >> 2));
}
__device__ __forceinline__ int4 vpredict(int4 xo, int4 a, int4 c) {
  return make_int4(xo.x + ((a.x + c.x) >> 1), xo.y + ((a.y + c.y) >> 1), xo.z + ((a.z + c.z) >> 1),
                   xo.w + ((a.w + c.w) >> 1));
}

// Vertical 5/3 stream over output rows [ys, ye) (ys even) of NC level images
// at once; emit(y, v[NC]) receives each finished row (four columns per lane).
// A component's next row pair is loaded as soon as its registers are free, so
// the loads of a whole pair are in flight while the current one is lifted and
// emitted.  What bounds it is the latency of those loads: the lifting state in
// registers at 16 warps per SM (RGB; 24 with one component) with every load
// predicated took the last level + pack of the uneven batch from 1.38 to 1.02
// ms (floor at the copy rate 0.80 ms) and of 256 tiles of 512 x 512 from 0.30
// to 0.22 ms, against state in shared memory at 32 warps with one component's
// rows ahead.  Two pairs ahead measured no faster.  tab: the components'
// bands.
template <int NC, bool VEC, typename Emit>
__device__ __forceinline__ void stream_rows(const Bands* tab, const Cols& o, int lane, int ys, int ye, Emit emit) {
  const int h = o.h;
  int4 v[NC];
  if (h == 1) {
#pragma unroll
    for (int c = 0; c < NC; ++c) v[c] = lift_row<VEC>(load_row<VEC>(tab[c].ll, tab[c].hl, 0, o, lane), o, lane);
    emit(0, v);
    return;
  }
  // Rows -1 .. h + 1 of the symmetric extension (h at least 2).
  auto row = [&](int y) { return abs(y < h ? y : 2 * (h - 1) - y) >> 1; };
  // Even rows lie in the low/high pair ll, hl and odd rows in lh, hh;
  // reflection keeps a row's parity.
  auto even = [&](int c, int y) { return load_row<VEC>(tab[c].ll, tab[c].hl, row(y), o, lane); };
  auto odd = [&](int c, int y) { return load_row<VEC>(tab[c].lh, tab[c].hh, row(y), o, lane); };
  int4 xo_prev[NC], ev_prev[NC];
  RawRow re[NC], ro[NC];
  {
    RawRow rp[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) rp[c] = odd(c, ys - 1);
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      re[c] = even(c, ys);
      ro[c] = odd(c, ys + 1);
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      xo_prev[c] = lift_row<VEC>(rp[c], o, lane);
      ev_prev[c] = make_int4(0, 0, 0, 0);
    }
  }
  for (int y = ys;; y += 2) {
    const bool more = y + 1 < ye;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int4 xe = lift_row<VEC>(re[c], o, lane), xo = lift_row<VEC>(ro[c], o, lane);
      if (more) {
        re[c] = even(c, y + 2);
        ro[c] = odd(c, y + 3);
      }
      const int4 ev = vupdate(xe, xo_prev[c], xo);
      v[c] = vpredict(xo_prev[c], ev_prev[c], ev);
      xo_prev[c] = xo;
      ev_prev[c] = ev;
    }
    if (y > ys) emit(y - 1, v);
    if (y < ye) emit(y, ev_prev);
    if (!more) return;
  }
}

template <typename Job>
__device__ __forceinline__ const Job& find_job(const Job* jobs, uint32_t njobs, uint32_t unit) {
  uint32_t lo = 0, hi = njobs - 1;
  while (lo < hi) {
    uint32_t mid = (lo + hi + 1) >> 1;
    if (jobs[mid].unit_begin <= unit) lo = mid;
    else hi = mid - 1;
  }
  return jobs[lo];
}

}  // namespace

namespace {

// Next work unit of the calling warp: the grid form takes one unit per warp;
// the queue form (persistent grid) takes units from a device counter until
// they run out.  Returns false when the warp is done.
__device__ __forceinline__ bool next_unit(uint32_t* queue, uint32_t nunits, bool& first, uint32_t& unit) {
  if (!queue) {
    unit = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const bool go = first && unit < nunits;
    first = false;
    return go;
  }
  uint32_t u = 0;
  if ((threadIdx.x & 31) == 0) u = atomicAdd(queue, 1u);
  unit = __shfl_sync(0xFFFFFFFFu, u, 0);
  return unit < nunits;
}

__device__ __forceinline__ void idwt_unit(const IdwtJob* __restrict__ jobs, uint32_t njobs, uint32_t unit) {
  const int lane = threadIdx.x & 31;
  const IdwtJob& job = find_job(jobs, njobs, unit);
  const uint32_t local = unit - job.unit_begin;
  const int x0 = (int)job.x_begin + (int)(local % job.strips) * kIdwtStripW;
  const int ys = (int)job.y_begin + (int)(local / job.strips) * (int)job.seg;
  const int w = (int)job.w, h = (int)job.h;
  const int ye = min(ys + (int)job.seg, (int)job.y_end);
  const Bands B{job.ll, job.hl, job.lh, job.hh};
  const int col = x0 + 4 * lane;
  int32_t* out = job.out;
  // Rows of w int32 from a 16-byte aligned base: 16-byte stores when w % 4 == 0.
  const bool vec_out = (w & 3) == 0 && (((uintptr_t)out) & 15) == 0;
  auto emit = [&](int y, const int4* v) {
    int32_t* row = out + (size_t)y * w;
    if (vec_out && col + 3 < w) {
      *reinterpret_cast<int4*>(row + col) = v[0];
    } else {
      if (col < w) row[col] = v[0].x;
      if (col + 1 < w) row[col + 1] = v[0].y;
      if (col + 2 < w) row[col + 2] = v[0].z;
      if (col + 3 < w) row[col + 3] = v[0].w;
    }
  };
  if (x0 + kIdwtStripW <= w && aligned_bands(B, w))
    stream_rows<1, true>(&B, make_cols<true>(x0, w, h, lane), lane, ys, ye, emit);
  else
    stream_rows<1, false>(&B, make_cols<false>(x0, w, h, lane), lane, ys, ye, emit);
}

}  // namespace

// QUEUE: persistent grid taking units from the device counter `queue`;
// otherwise one unit per warp.
// The grid form held to four CTAs per SM (64 registers, a few bytes of
// spills): more units in flight, which the large levels of uneven batches
// want (C2 levels 0.728 -> 0.680 ms) and the uniform 512^2 batch does not
// (0.158 -> 0.163 ms); the autotuner picks.
__global__ void __launch_bounds__(kIdwtWarps * 32, 4) idwt_level_lean_kernel(const IdwtJob* __restrict__ jobs,
                                                                            uint32_t njobs, uint32_t nunits) {
  const uint32_t unit = blockIdx.x * kIdwtWarps + (threadIdx.x >> 5);
  if (unit < nunits) idwt_unit(jobs, njobs, unit);
}

template <bool QUEUE>
__global__ void __launch_bounds__(kIdwtWarps * 32) idwt_level_kernel(const IdwtJob* __restrict__ jobs,
                                                                     uint32_t njobs, uint32_t nunits,
                                                                     uint32_t* queue) {
  if (!QUEUE) {
    const uint32_t unit = blockIdx.x * kIdwtWarps + (threadIdx.x >> 5);
    if (unit < nunits) idwt_unit(jobs, njobs, unit);
    return;
  }
  bool first = true;
  for (uint32_t unit; next_unit(queue, nunits, first, unit);) idwt_unit(jobs, njobs, unit);
}

namespace {

__device__ __forceinline__ uint32_t sat_u8f(float r) { return (uint32_t)fminf(fmaxf(r, 0.0f), 255.0f); }

// DIRECT: the sample needs only a clamp (8-bit samples to u8, or samples of
// more than 8 bits to u16); chosen per unit so the hot loop holds no float or
// division path.
template <bool DIRECT>
__device__ __forceinline__ uint32_t to_u8(int32_t v, uint32_t bd, uint32_t region) {
  if (DIRECT || bd == 8) return (uint32_t)min(max(v, 0), 255);
  if (region) {
    // sample_as_u8: round, clamp to the depth's maximum, rescale to 8 bits.
    float maxv = bd >= 16 ? 65535.0f : (float)max((1 << bd) - 1, 1);
    float c = fminf(fmaxf((float)v, 0.0f), maxv);
    return sat_u8f(roundf(__fmul_rn(__fdiv_rn(c, maxv), 255.0f)));
  }
  // interleave_and_convert slow path: round(v / (2^bd - 1) * 255) as u8.
  float d = (float)((1u << bd) - 1);
  return sat_u8f(roundf(__fmul_rn(__fdiv_rn((float)v, d), 255.0f)));
}

template <bool DIRECT>
__device__ __forceinline__ uint32_t to_u16(int32_t v, uint32_t bd) {
  int32_t maxv = (int32_t)((1u << bd) - 1);
  int32_t c = min(max(v, 0), maxv);
  if (!DIRECT && bd <= 8) {
    uint32_t mx = max((1u << bd) - 1, 1u);
    return ((uint32_t)c * 65535u + mx / 2) / mx;
  }
  return (uint32_t)c;
}

template <int FMT>
__host__ __device__ constexpr int pack_bpp() {
  return FMT == PACK_GRAY8 ? 1 : FMT == PACK_RGB8 ? 3 : FMT == PACK_RGBA8 ? 4 : FMT == PACK_GRAY16 ? 2 : 6;
}

// Byte q (a compile-time constant after unrolling) of a lane's packed words.
__device__ __forceinline__ void put_byte(uint32_t* wds, int q, uint32_t byte) { wds[q >> 2] |= byte << (8 * (q & 3)); }

// Four samples clamped to [0, 255], the first in the low byte.
__device__ __forceinline__ uint32_t pack_u8x4(int32_t a, int32_t b, int32_t c, int32_t d) {
#ifdef __CUDA_ARCH__
  uint32_t hi, r;
  asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(hi) : "r"(d), "r"(c), "r"(0));
  asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(b), "r"(a), "r"(hi));
  return r;
#else
  auto u = [](int32_t v) { return (uint32_t)min(max(v, 0), 255); };
  return u(a) | (u(b) << 8) | (u(c) << 16) | (u(d) << 24);
#endif
}

// Packs pixel p (components c0..c2 after the inverse RCT and DC shift) at
// byte p * bpp of the lane's four-pixel group.
template <int FMT, bool DIRECT>
__device__ __forceinline__ void put_pixel(uint32_t* wds, int p, int32_t c0, int32_t c1, int32_t c2, uint32_t bd,
                                          uint32_t reg) {
  constexpr int B = pack_bpp<FMT>();
  const int q = p * B;
  if (FMT == PACK_GRAY8) {
    put_byte(wds, q, to_u8<DIRECT>(c0, bd, reg));
  } else if (FMT == PACK_RGB8 || FMT == PACK_RGBA8) {
    put_byte(wds, q, to_u8<DIRECT>(c0, bd, reg));
    put_byte(wds, q + 1, to_u8<DIRECT>(c1, bd, reg));
    put_byte(wds, q + 2, to_u8<DIRECT>(c2, bd, reg));
    if (FMT == PACK_RGBA8) put_byte(wds, q + 3, 255u);
  } else if (FMT == PACK_GRAY16) {
    const uint32_t a = to_u16<DIRECT>(c0, bd);
    put_byte(wds, q, a & 0xFF);
    put_byte(wds, q + 1, a >> 8);
  } else {
    const uint32_t a = to_u16<DIRECT>(c0, bd), g = to_u16<DIRECT>(c1, bd), c = to_u16<DIRECT>(c2, bd);
    put_byte(wds, q, a & 0xFF);
    put_byte(wds, q + 1, a >> 8);
    put_byte(wds, q + 2, g & 0xFF);
    put_byte(wds, q + 3, g >> 8);
    put_byte(wds, q + 4, c & 0xFF);
    put_byte(wds, q + 5, c >> 8);
  }
}

__device__ __forceinline__ int lane_comp(const int4& v, int p) { return p == 0 ? v.x : p == 1 ? v.y : p == 2 ? v.z : v.w; }

// Row buffer per warp: up to 15 bytes of alignment shift + 128 pixels x 6 bytes.
constexpr int kRowWords = (16 + kIdwtStripW * 6) / 4;

// Writes one output row of a warp's strip: each lane's packed words (four
// pixels of BPP bytes) are staged in the warp's row buffer so that the copied
// range has the destination's alignment mod 16, then columns [xs, xe) go out
// as the bytes up to the first 16-byte boundary, 16-byte vectors and a tail.
// g: the destination of column xs in the row; lane k's words hold columns
// x0 + 4k .. x0 + 4k + 3.  When the destination is 4-byte aligned and the
// columns [xs, xs + nbytes / BPP) start and end on lane boundaries (whole
// strips of a tile, the common case), every lane inside writes its BPP words
// itself: four pixels of BPP bytes are BPP 32-bit words at a 4-byte aligned
// place.  Otherwise the row goes through the warp's buffer as below.
template <int BPP>
__device__ __forceinline__ void store_row(uint8_t* g, int x0, int xs, int nbytes, int lane, uint32_t* rowbuf,
                                          const uint32_t* wds) {
  const int xe = xs + nbytes / BPP;
  if ((((uintptr_t)g & 3) | ((xs - x0) & 3) | ((xe - x0) & 3)) == 0) {  // warp-uniform
    const int c = x0 + 4 * lane;
    if (c >= xs && c < xe) {
      uint32_t* d = reinterpret_cast<uint32_t*>(g + (size_t)(c - xs) * BPP);
#pragma unroll
      for (int k = 0; k < BPP; ++k) d[k] = wds[k];
    }
    return;
  }
  uint8_t* rowbytes = reinterpret_cast<uint8_t*>(rowbuf);
  const int sh = (int)(((uintptr_t)g - (uintptr_t)((xs - x0) * BPP)) & 15);
  if ((sh & 3) == 0) {
    uint32_t* dst = rowbuf + (sh >> 2) + lane * BPP;
#pragma unroll
    for (int k = 0; k < BPP; ++k) dst[k] = wds[k];
  } else {
    uint8_t* dst = rowbytes + sh + lane * 4 * BPP;
#pragma unroll
    for (int q = 0; q < 4 * BPP; ++q) dst[q] = (uint8_t)(wds[q >> 2] >> (8 * (q & 3)));
  }
  __syncwarp();
  const uint8_t* src = rowbytes + sh + (xs - x0) * BPP;
  int head = (int)((16 - ((uintptr_t)g & 15)) & 15);
  if (head > nbytes) head = nbytes;
  if (lane < head) g[lane] = src[lane];
  const int nvec = (nbytes - head) >> 4;
  const uint4* sv = reinterpret_cast<const uint4*>(src + head);
  uint4* gv = reinterpret_cast<uint4*>(g + head);
  for (int k = lane; k < nvec; k += 32) gv[k] = sv[k];
  const int done = head + (nvec << 4);
  if (lane < nbytes - done) g[done + lane] = src[done + lane];
  __syncwarp();
}

template <int NC, int FMT, bool DIRECT>
__device__ __forceinline__ void pack_unit(const PackJob& job, int x0, int ys, int ye, int lane, uint32_t* rowbuf,
                                          Bands* tab) {
  constexpr int BPP = pack_bpp<FMT>();
  const int w = (int)job.w;
  const int cx0 = (int)job.cx, cy0 = (int)job.cy, cx1 = cx0 + (int)job.cw, cy1 = cy0 + (int)job.ch;
  const uint32_t bd = job.bit_depth, reg = job.region_conv;
  const int32_t shift = 1 << (bd - 1);
  const bool mct = NC == 3 && job.mct;
  const int col = x0 + 4 * lane;
  const int xs = max(x0, cx0), xe = min(x0 + kIdwtStripW, cx1);
  const int nbytes = (xe - xs) * BPP;
  uint8_t* const first = job.out + (uint64_t)(xs - cx0) * BPP;
  const uint64_t pitch = job.pitch;
  auto emit = [&](int y, const int4* v) {
    if (y < cy0 || y >= cy1) return;  // warp-uniform
    // The DC shift joins the luma before the inverse RCT, whose other two
    // components are sums with the green that comes out of it.
    int32_t px[4][NC];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      px[p][0] = lane_comp(v[0], p) + shift;
      if (NC == 3) {
        const int32_t c1 = lane_comp(v[1], p), c2 = lane_comp(v[2], p);
        if (mct) {
          const int32_t g = px[p][0] - ((c2 + c1) >> 2);
          px[p][0] = c2 + g;
          px[p][1] = g;
          px[p][2] = c1 + g;
        } else {
          px[p][1] = c1 + shift;
          px[p][2] = c2 + shift;
        }
      }
    }
    uint32_t wds[BPP];
    if constexpr (DIRECT && FMT == PACK_GRAY8) {
      wds[0] = pack_u8x4(px[0][0], px[1][0], px[2][0], px[3][0]);
    } else if constexpr (DIRECT && FMT == PACK_RGB8) {
      wds[0] = pack_u8x4(px[0][0], px[0][1], px[0][2], px[1][0]);
      wds[1] = pack_u8x4(px[1][1], px[1][2], px[2][0], px[2][1]);
      wds[2] = pack_u8x4(px[2][2], px[3][0], px[3][1], px[3][2]);
    } else if constexpr (DIRECT && FMT == PACK_RGBA8) {
#pragma unroll
      for (int p = 0; p < 4; ++p) wds[p] = pack_u8x4(px[p][0], px[p][1], px[p][2], 255);
    } else {
#pragma unroll
      for (int k = 0; k < BPP; ++k) wds[k] = 0;
#pragma unroll
      for (int p = 0; p < 4; ++p)
        put_pixel<FMT, DIRECT>(wds, p, px[p][0], px[p][NC == 3 ? 1 : 0], px[p][NC == 3 ? 2 : 0], bd, reg);
    }
    store_row<BPP>(first + (uint64_t)(y - cy0) * pitch, x0, xs, nbytes, lane, rowbuf, wds);
  };
  if (job.lifting) {
    // The components' band descriptors: read from the job once per unit into
    // the warp's shared table (RGB), or in registers (gray).
    const int h = (int)job.h;
    Bands one{job.ll[0], job.hl[0], job.lh[0], job.hh[0]};
    bool vec = x0 + kIdwtStripW <= w && aligned_bands(one, w);
    if (NC == 3) {
      for (int c = 1; c < 3; ++c) vec = vec && aligned_bands(Bands{job.ll[c], job.hl[c], job.lh[c], job.hh[c]}, w);
      if (lane < 3) tab[lane] = Bands{job.ll[lane], job.hl[lane], job.lh[lane], job.hh[lane]};
      __syncwarp();
    }
    const Bands* B = NC == 3 ? tab : &one;
    if (vec) stream_rows<NC, true>(B, make_cols<true>(x0, w, h, lane), lane, ys, ye, emit);
    else stream_rows<NC, false>(B, make_cols<false>(x0, w, h, lane), lane, ys, ye, emit);
    if (NC == 3) __syncwarp();  // the table is rewritten by the warp's next unit
  } else {
    // Nothing left to lift: the image is the LL band itself.
    for (int y = ys; y < ye; ++y) {
      int4 v[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int32_t* row = job.ll[c] + (size_t)y * w;
        v[c].x = col < w ? __ldg(row + col) : 0;
        v[c].y = col + 1 < w ? __ldg(row + col + 1) : 0;
        v[c].z = col + 2 < w ? __ldg(row + col + 2) : 0;
        v[c].w = col + 3 < w ? __ldg(row + col + 3) : 0;
      }
      emit(y, v);
    }
  }
}

}  // namespace

template <int FMT, int NC, bool DIRECT>
__device__ __forceinline__ void pack_one(const PackJob* __restrict__ jobs, uint32_t njobs, uint32_t unit,
                                         uint32_t* rowbuf, Bands* tab) {
  const int lane = threadIdx.x & 31;
  const PackJob& job = find_job(jobs, njobs, unit);
  const uint32_t local = unit - job.unit_begin;
  const int x0 = (int)(job.cx & ~(uint32_t)(kIdwtStripW - 1)) + (int)(local % job.strips) * kIdwtStripW;
  const int ys = (int)(job.cy & ~1u) + (int)(local / job.strips) * (int)job.seg;
  const int ye = min(ys + (int)job.seg, (int)(job.cy + job.ch));
  pack_unit<NC, FMT, DIRECT>(job, x0, ys, ye, lane, rowbuf, tab);
}

// One kernel per (pixel format, components, conversion) variant, with the
// jobs of a launch all of that variant (pack_variant): each variant gets the
// registers it needs and none of the others' code.  NC 3: RGB tiles, 1: gray;
// DIRECT: samples convert with a clamp alone.
template <int FMT, int NC, bool DIRECT, bool QUEUE>
__global__ void __launch_bounds__(kIdwtWarps * 32, NC == 3 ? 2 : 3) pack_kernel(const PackJob* __restrict__ jobs, uint32_t njobs,
                                                               uint32_t nunits, uint32_t* queue) {
  __shared__ __align__(16) uint32_t rowbufs[kIdwtWarps][kRowWords];
  __shared__ Bands tabs[kIdwtWarps][3];
  uint32_t* rowbuf = rowbufs[threadIdx.x >> 5];
  Bands* tab = tabs[threadIdx.x >> 5];
  if (!QUEUE) {
    const uint32_t unit = blockIdx.x * kIdwtWarps + (threadIdx.x >> 5);
    if (unit < nunits) pack_one<FMT, NC, DIRECT>(jobs, njobs, unit, rowbuf, tab);
    return;
  }
  bool first = true;
  for (uint32_t unit; next_unit(queue, nunits, first, unit);)
    pack_one<FMT, NC, DIRECT>(jobs, njobs, unit, rowbuf, tab);
}

// ---------------------------------------------------------------------------
// Irreversible 9/7 levels and the fused last level + inverse ICT + DC shift +
// pack (crates/signinum-j2k-native/src/j2c/idwt.rs:767-836, :1016-1140;
// mct.rs:80-115; decode.rs:1130-1151 for the dequantisation).
//
// Every sample goes through the reference's own sequence of f32 roundings:
// band coefficient x step, then per level the horizontal pass (even columns
// x K, odd x 1/K, then the four lifting steps delta, gamma, beta, alpha as
// fma(left + right, c, x)), then the same vertical pass.  Only __fmul_rn /
// __fadd_rn / fmaf are used, so no multiply is contracted into a
// neighbouring add and the results match the reference's f32 arithmetic bit
// for bit.  Symmetric extension is done by reflecting indices, which
// commutes with the lifting steps (reflected positions compute the same sums
// in the other order, and f32 addition is commutative).
//
// Mapping: a warp per strip of kStrip97 = 120 output columns x `seg` rows.
// Lane k holds the four columns x0 - 4 + 4k .. x0 - 1 + 4k, so lanes 0 and
// 31 hold the four columns on either side of the strip: a sample after the
// four lifting steps depends on the samples within four columns of it, so
// lanes 1..30 finish exact values while every lane runs the same code (each
// step takes one neighbour from the adjacent lane by a shuffle; the edge
// lanes' own results are not used).  Vertically a four-stage pipeline runs
// down the rows, loading rows 2m+2 and 2m+3 per step and finishing rows 2m
// (after beta) and 2m-1 (after alpha); a unit starting at row ys primes from
// row ys-3.  The lifting state sits in registers, a lane's column offsets are
// reflected once per unit, and a component's next rows load as soon as its
// registers are free.  What bounds it: the latency of the dependent f32 steps
// at 12 warps per SM.  128 tiles of 512 x 512 RGB: levels 0.36 -> 0.15 ms and
// last level + ICT + pack 0.59 -> 0.24 ms, against lifting state in shared
// memory and columns reflected per row; four CTAs per SM (128 registers, 90
// bytes of spills) 0.26 ms; the pack with every bit depth's conversion in one
// loop 0.54 ms.

constexpr float kNegAlpha97 = 1.5861343f, kNegBeta97 = 0.052980117f, kNegGamma97 = -0.8829111f,
                kNegDelta97 = -0.44350687f, kKappa97 = 1.2301741f;
constexpr int kWarps97 = 4;  // warps per CTA of the 9/7 pack kernel
static_assert(kStrip97 == 4 * (kLanes - 2), "lanes 1..30 hold a strip's output columns");

namespace {

struct Src97 {
  const int32_t* ll;
  const int32_t* hl;
  const int32_t* lh;
  const int32_t* hh;
  float q[4];  // dequantisation steps of ll, hl, lh, hh
};

// A lane's columns: band offsets of its image columns c .. c+3 (low band l0,
// l1; high band h0, h1).  VEC: the strip's 128 columns lie inside the level
// and its rows are 8-byte aligned, so each band's pair is one load.
struct Cols97 {
  int w, h;
  int l0, l1, h0, h1;
  bool ll_band;  // ll is the LL band; otherwise the previous level's f32 image
};

__device__ __forceinline__ bool vec97(const Src97& S, int w, int c0) {
  const uintptr_t a = (uintptr_t)S.ll | (uintptr_t)S.hl | (uintptr_t)S.lh | (uintptr_t)S.hh;
  return (w & 3) == 0 && (a & 7) == 0 && c0 >= 0 && c0 + 4 * kLanes <= w;
}

template <bool VEC>
__device__ __forceinline__ Cols97 make_cols97(int c, int w, int h, bool ll_band) {
  if (VEC) return Cols97{w, h, c >> 1, 0, c >> 1, 0, ll_band};
  return Cols97{w, h, reflect(c, w) >> 1, reflect(c + 2, w) >> 1, reflect(c + 1, w) >> 1, reflect(c + 3, w) >> 1, ll_band};
}

// The raw words of a lane's four columns of one interleaved row (low band at
// the even columns, high band at the odd ones), loaded ahead of their use.
struct Raw97 {
  int32_t e0, o0, e1, o1;
};

// Row r of the low and the high band.
template <bool VEC>
__device__ __forceinline__ Raw97 load97(const int32_t* low, const int32_t* high, int r, const Cols97& o) {
  const int32_t* lo = low + (size_t)r * ((o.w + 1) >> 1) + o.l0;
  const int32_t* hi = high + (size_t)r * (o.w >> 1) + o.h0;
  if (VEC) {
    const int2 l = __ldg(reinterpret_cast<const int2*>(lo));
    const int2 h = __ldg(reinterpret_cast<const int2*>(hi));
    return Raw97{l.x, h.x, l.y, h.y};
  }
  const bool high_band = o.w > 1;  // a single column has none
  return Raw97{__ldg(lo), load_if(high_band, hi), __ldg(lo + (o.l1 - o.l0)), load_if(high_band, hi + (o.h1 - o.h0))};
}

__device__ __forceinline__ float lstep(float l, float r, float c, float x) { return fmaf(__fadd_rn(l, r), c, x); }

// Dequantises (or reinterprets) a loaded row and runs the horizontal 9/7
// synthesis: the lane's four columns (exact on lanes 1..30).  IMAGE: the low
// band's words are the previous level's f32 samples.
__device__ __forceinline__ float4 lift97(const Raw97& R, float ql, float qh, bool image, bool single, float K, float IK) {
  float e0 = image ? __int_as_float(R.e0) : __fmul_rn(__int2float_rn(R.e0), ql);
  float e1 = image ? __int_as_float(R.e1) : __fmul_rn(__int2float_rn(R.e1), ql);
  float o0 = __fmul_rn(__int2float_rn(R.o0), qh), o1 = __fmul_rn(__int2float_rn(R.o1), qh);
  if (single) return make_float4(e0, 0.0f, 0.0f, 0.0f);
  e0 = __fmul_rn(e0, K);
  e1 = __fmul_rn(e1, K);
  o0 = __fmul_rn(o0, IK);
  o1 = __fmul_rn(o1, IK);
  // delta: even columns; gamma: odd; beta: even; alpha: odd.
  const float om1 = __shfl_up_sync(0xFFFFFFFFu, o1, 1);
  const float e0a = lstep(om1, o0, kNegDelta97, e0), e1a = lstep(o0, o1, kNegDelta97, e1);
  const float ep4a = __shfl_down_sync(0xFFFFFFFFu, e0a, 1);
  const float o0b = lstep(e0a, e1a, kNegGamma97, o0), o1b = lstep(e1a, ep4a, kNegGamma97, o1);
  const float om1b = __shfl_up_sync(0xFFFFFFFFu, o1b, 1);
  const float e0c = lstep(om1b, o0b, kNegBeta97, e0a), e1c = lstep(o0b, o1b, kNegBeta97, e1a);
  const float ep4c = __shfl_down_sync(0xFFFFFFFFu, e0c, 1);
  return make_float4(e0c, lstep(e0c, e1c, kNegAlpha97, o0b), e1c, lstep(e1c, ep4c, kNegAlpha97, o1b));
}

__device__ __forceinline__ float4 scale4(float4 v, float k) {
  return make_float4(__fmul_rn(v.x, k), __fmul_rn(v.y, k), __fmul_rn(v.z, k), __fmul_rn(v.w, k));
}
__device__ __forceinline__ float4 lstep4(float4 a, float4 b, float c, float4 x) {
  return make_float4(lstep(a.x, b.x, c, x.x), lstep(a.y, b.y, c, x.y), lstep(a.z, b.z, c, x.z),
                     lstep(a.w, b.w, c, x.w));
}

// Vertical 9/7 stream over rows [ys, ye) (ys even) of NC level images, one
// component after the other; emit(y, v[NC]) receives each finished row.
template <int NC, bool VEC, typename Emit>
__device__ __forceinline__ void stream97(const Src97* tab, const Cols97& o, int ys, int ye, float K, float IK,
                                         Emit emit) {
  const int h = o.h;
  const bool image = !o.ll_band, single = !VEC && o.w == 1;
  float4 v[NC];
  auto even97 = [&](int c, const Raw97& R) { return lift97(R, tab[c].q[0], tab[c].q[1], image, single, K, IK); };
  auto odd97 = [&](int c, const Raw97& R) { return lift97(R, tab[c].q[2], tab[c].q[3], false, single, K, IK); };
  if (h == 1) {
#pragma unroll
    for (int c = 0; c < NC; ++c) v[c] = even97(c, load97<VEC>(tab[c].ll, tab[c].hl, 0, o));
    emit(0, v);
    return;
  }
  // Rows -4 .. h + 3 of the symmetric extension (h at least 2; rows that no
  // finished row depends on may be asked for further out when h is 2).
  auto row = [&](int y) {
    int t = abs(y);
    t = t < h ? t : abs(2 * (h - 1) - t);
    t = t < h ? t : abs(2 * (h - 1) - t);
    return (t < h ? t : t & 1) >> 1;
  };
  auto even = [&](int c, int y) { return load97<VEC>(tab[c].ll, tab[c].hl, row(y), o); };
  auto odd = [&](int c, int y) { return load97<VEC>(tab[c].lh, tab[c].hh, row(y), o); };
  const int y1 = ye & ~1;  // the last step's even row
  int y = ys - 4;          // the step's even row: rows y + 2, y + 3 come in
  // Per component: the last odd row in, the last rows after delta and gamma,
  // and the last finished even row.
  float4 xp[NC], s1p[NC], s2p[NC], s3p[NC];
  Raw97 re[NC], ro[NC];
  {
    Raw97 rp[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) rp[c] = odd(c, ys - 3);
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      re[c] = even(c, y + 2);
      ro[c] = odd(c, y + 3);
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      xp[c] = scale4(odd97(c, rp[c]), IK);
      s1p[c] = s2p[c] = s3p[c] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
  }
  for (;; y += 2) {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const float4 xe = scale4(even97(c, re[c]), K);
      const float4 xo = scale4(odd97(c, ro[c]), IK);
      if (y < y1) {
        re[c] = even(c, y + 4);
        ro[c] = odd(c, y + 5);
      }
      const float4 s1 = lstep4(xp[c], xo, kNegDelta97, xe);   // row y + 2
      const float4 s2 = lstep4(s1p[c], s1, kNegGamma97, xp[c]);  // row y + 1
      const float4 s3 = lstep4(s2p[c], s2, kNegBeta97, s1p[c]);  // row y, final
      v[c] = lstep4(s3p[c], s3, kNegAlpha97, s2p[c]);            // row y - 1, final
      xp[c] = xo;
      s1p[c] = s1;
      s2p[c] = s2;
      s3p[c] = s3;
    }
    if (y > ys) emit(y - 1, v);
    if (y >= ys && y < ye) emit(y, s3p);
    if (y >= y1) return;
  }
}

__device__ __forceinline__ void idwt97_unit(const IdwtJob* __restrict__ jobs, uint32_t njobs, uint32_t unit, float IK) {
  const int lane = threadIdx.x & 31;
  const IdwtJob& job = find_job(jobs, njobs, unit);
  const uint32_t local = unit - job.unit_begin;
  const int x0 = (int)job.x_begin + (int)(local % job.strips) * kStrip97;
  const int ys = (int)job.y_begin + (int)(local / job.strips) * (int)job.seg;
  const int w = (int)job.w, h = (int)job.h;
  const int ye = min(ys + (int)job.seg, (int)job.y_end);
  const int col = x0 - 4 + 4 * lane;
  const Src97 S{job.ll, job.hl, job.lh, job.hh, {job.step[0], job.step[1], job.step[2], job.step[3]}};
  float* out = reinterpret_cast<float*>(job.out);
  const bool mine = lane >= 1 && lane <= kLanes - 2;
  const bool vec_out = (w & 3) == 0 && (((uintptr_t)out) & 15) == 0;
  const bool ll_band = job.ll_band != 0;
  auto emit = [&](int y, const float4* v) {
    if (!mine) return;
    float* rowp = out + (size_t)y * w;
    if (vec_out && col + 3 < w) {
      *reinterpret_cast<float4*>(rowp + col) = v[0];
    } else {
      if (col < w) rowp[col] = v[0].x;
      if (col + 1 < w) rowp[col + 1] = v[0].y;
      if (col + 2 < w) rowp[col + 2] = v[0].z;
      if (col + 3 < w) rowp[col + 3] = v[0].w;
    }
  };
  if (vec97(S, w, x0 - 4)) stream97<1, true>(&S, make_cols97<true>(col, w, h, ll_band), ys, ye, kKappa97, IK, emit);
  else stream97<1, false>(&S, make_cols97<false>(col, w, h, ll_band), ys, ye, kKappa97, IK, emit);
}

}  // namespace

template <bool QUEUE>
__global__ void __launch_bounds__(kIdwtWarps * 32) idwt97_level_kernel(const IdwtJob* __restrict__ jobs,
                                                                       uint32_t njobs, uint32_t nunits,
                                                                       uint32_t* queue) {
  const float IK = __fdiv_rn(1.0f, kKappa97);
  if (!QUEUE) {
    const uint32_t unit = blockIdx.x * kIdwtWarps + (threadIdx.x >> 5);
    if (unit < nunits) idwt97_unit(jobs, njobs, unit, IK);
    return;
  }
  bool first = true;
  for (uint32_t unit; next_unit(queue, nunits, first, unit);) idwt97_unit(jobs, njobs, unit, IK);
}

namespace {

__device__ __forceinline__ float lane_compf(const float4& v, int p) {
  return p == 0 ? v.x : p == 1 ? v.y : p == 2 ? v.z : v.w;
}

// `as u8` of a rounded f32: NaN and negatives 0, saturating at 255.
__device__ __forceinline__ uint32_t sat_u8_round(float r) {
  if (!(r > 0.0f)) return 0u;
  if (r >= 255.0f) return 255u;
  return (uint32_t)r;
}

// sat_u8_round(roundf(v)), roundf taking halves away from zero: v clamped to
// [0, 255] (NaN to 0) plus 2^23 is v rounded to the nearest integer, halves
// to even, in the low bits of the sum; where that took a half down, one more.
__device__ __forceinline__ uint32_t round_u8(float v) {
  const float c = fminf(fmaxf(v, 0.0f), 255.0f), y = __fadd_rn(c, 8388608.0f);
  const float d = __fadd_rn(c, -__fadd_rn(y, -8388608.0f));
  uint32_t bits;
#ifdef __CUDA_ARCH__
  bits = __float_as_uint(y);
#else
  std::memcpy(&bits, &y, 4);
#endif
  return (bits & 0xFFu) + (d == 0.5f ? 1u : 0u);
}

// Sample conversions of the f32 path (crates/signinum-j2k-native/src/lib.rs:1772-1840,
// :2202-2294; crates/signinum-j2k/src/decode.rs:345-356, :517-545).
// EIGHT: samples of eight bits, rounded and clamped (region request or not);
// chosen per unit so the hot loop holds no division path.
template <bool EIGHT>
__device__ __forceinline__ uint32_t f_to_u8(float v, uint32_t bd, uint32_t region) {
  if (EIGHT) return round_u8(v);
  const float r = roundf(v);
  if (region) {
    // sample_as_u8: round, clamp to the depth's maximum, rescale to 8 bits.
    const float maxv = bd >= 16 ? 65535.0f : (float)max((1 << bd) - 1, 1);
    const float c = fminf(fmaxf(r, 0.0f), maxv);
    return sat_u8_round(roundf(__fmul_rn(__fdiv_rn(c, maxv), 255.0f)));
  }
  // interleave_and_convert: rescaled.
  return sat_u8_round(roundf(__fmul_rn(__fdiv_rn(v, (float)((1u << bd) - 1)), 255.0f)));
}

// decode_native: round, clamp to [0, 2^bd - 1], widen depths <= 8 to 16 bits.
__device__ __forceinline__ uint32_t f_to_u16(float v, uint32_t bd) {
  const float maxv = (float)((1u << bd) - 1);
  const float r = roundf(v);
  const float c = r < 0.0f ? 0.0f : (r > maxv ? maxv : r);
  if (bd <= 8) {
    const uint32_t s = (uint32_t)(uint8_t)c, mx = max((1u << bd) - 1, 1u);
    return (s * 65535u + mx / 2) / mx;
  }
  return (uint32_t)c;
}

template <int FMT, bool EIGHT>
__device__ __forceinline__ void put_pixel97(uint32_t* wds, int p, float c0, float c1, float c2, uint32_t bd,
                                            uint32_t reg) {
  constexpr int B = pack_bpp<FMT>();
  const int q = p * B;
  if (FMT == PACK_GRAY8) {
    put_byte(wds, q, f_to_u8<EIGHT>(c0, bd, reg));
  } else if (FMT == PACK_RGB8 || FMT == PACK_RGBA8) {
    put_byte(wds, q, f_to_u8<EIGHT>(c0, bd, reg));
    put_byte(wds, q + 1, f_to_u8<EIGHT>(c1, bd, reg));
    put_byte(wds, q + 2, f_to_u8<EIGHT>(c2, bd, reg));
    if (FMT == PACK_RGBA8) put_byte(wds, q + 3, 255u);
  } else if (FMT == PACK_GRAY16) {
    const uint32_t a = f_to_u16(c0, bd);
    put_byte(wds, q, a & 0xFF);
    put_byte(wds, q + 1, a >> 8);
  } else {
    const uint32_t a = f_to_u16(c0, bd), g = f_to_u16(c1, bd), c = f_to_u16(c2, bd);
    put_byte(wds, q, a & 0xFF);
    put_byte(wds, q + 1, a >> 8);
    put_byte(wds, q + 2, g & 0xFF);
    put_byte(wds, q + 3, g >> 8);
    put_byte(wds, q + 4, c & 0xFF);
    put_byte(wds, q + 5, c >> 8);
  }
}

template <int NC, int FMT, bool EIGHT>
__device__ __forceinline__ void pack97_unit(const PackJob& job, int x0, int ys, int ye, int lane, uint32_t* rowbuf,
                                            Src97* tab, float IK) {
  constexpr int BPP = pack_bpp<FMT>();
  const int w = (int)job.w, h = (int)job.h;
  const int cx0 = (int)job.cx, cy0 = (int)job.cy, cx1 = cx0 + (int)job.cw, cy1 = cy0 + (int)job.ch;
  const uint32_t bd = job.bit_depth, reg = job.region_conv;
  const float shift = (float)(1u << (bd - 1));
  const bool ict = NC == 3 && job.mct;
  const int col = x0 - 4 + 4 * lane;
  const int xs = max(x0, cx0), xe = min(x0 + kStrip97, cx1);
  const int nbytes = (xe - xs) * BPP;
  auto emit = [&](int y, const float4* v) {
    if (y < cy0 || y >= cy1) return;  // warp-uniform
    uint32_t wds[BPP];
#pragma unroll
    for (int k = 0; k < BPP; ++k) wds[k] = 0;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      float c0 = lane_compf(v[0], p), c1 = 0.0f, c2 = 0.0f;
      if (NC == 3) {
        c1 = lane_compf(v[1], p);
        c2 = lane_compf(v[2], p);
        if (ict) {
          // mct.rs:80-115 with fused multiply-adds.
          const float r = fmaf(c2, 1.402f, c0);
          const float g = fmaf(c2, -0.71414f, fmaf(c1, -0.34413f, c0));
          const float bl = fmaf(c1, 1.772f, c0);
          c0 = r;
          c1 = g;
          c2 = bl;
        }
        c1 = __fadd_rn(c1, shift);
        c2 = __fadd_rn(c2, shift);
      }
      c0 = __fadd_rn(c0, shift);
      put_pixel97<FMT, EIGHT>(wds, p, c0, c1, c2, bd, reg);
    }
    // Lane k's words are columns x0 - 4 + 4k ..: the row starts at x0 - 4.
    store_row<BPP>(job.out + (uint64_t)(y - cy0) * job.pitch + (uint64_t)(xs - cx0) * BPP, x0 - 4, xs, nbytes,
                   lane, rowbuf, wds);
  };
  if (job.lifting) {
    // The components' band descriptors: read from the job once per unit into
    // the warp's shared table (RGB), or in registers (gray).
    const bool ll_band = job.ll_band != 0;
    auto src = [&](int c) {
      return Src97{job.ll[c], job.hl[c], job.lh[c], job.hh[c], {job.step[c][0], job.step[c][1], job.step[c][2], job.step[c][3]}};
    };
    const Src97 one = src(0);
    bool vec = vec97(one, w, x0 - 4);
    if (NC == 3) {
      vec = vec && vec97(src(1), w, x0 - 4) && vec97(src(2), w, x0 - 4);
      if (lane < 3) tab[lane] = src(lane);
      __syncwarp();
    }
    const Src97* S = NC == 3 ? tab : &one;
    if (vec) stream97<NC, true>(S, make_cols97<true>(col, w, h, ll_band), ys, ye, kKappa97, IK, emit);
    else stream97<NC, false>(S, make_cols97<false>(col, w, h, ll_band), ys, ye, kKappa97, IK, emit);
    if (NC == 3) __syncwarp();  // the table is rewritten by the warp's next unit
  } else {
    // Nothing to lift: the image is the LL band itself (dequantised).
    for (int y = ys; y < ye; ++y) {
      float4 v[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int32_t* rowp = job.ll[c] + (size_t)y * w;
        const float q = job.step[c][0];
        auto at = [&](int k) {
          const int x = col + k;
          return x >= 0 && x < w ? __fmul_rn(__int2float_rn(__ldg(rowp + x)), q) : 0.0f;
        };
        v[c] = make_float4(at(0), at(1), at(2), at(3));
      }
      emit(y, v);
    }
  }
}

}  // namespace

// Three CTAs per SM for RGB (152 registers, no spills), five for gray.
template <int FMT, bool QUEUE>
__global__ void __launch_bounds__(kWarps97 * 32, (FMT == PACK_GRAY8 || FMT == PACK_GRAY16) ? 5 : 3) pack97_kernel(const PackJob* __restrict__ jobs, uint32_t njobs,
                                                               uint32_t nunits, uint32_t* queue) {
  __shared__ __align__(16) uint32_t rowbufs[kWarps97][kRowWords];
  __shared__ Src97 tabs[kWarps97][3];
  const float IK = __fdiv_rn(1.0f, kKappa97);
  uint32_t* rowbuf = rowbufs[threadIdx.x >> 5];
  Src97* tab = tabs[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  auto one = [&](uint32_t unit) {
    const PackJob& job = find_job(jobs, njobs, unit);
    const uint32_t local = unit - job.unit_begin;
    const int x0 = (int)(job.cx - job.cx % kStrip97) + (int)(local % job.strips) * kStrip97;
    const int ys = (int)(job.cy & ~1u) + (int)(local / job.strips) * (int)job.seg;
    const int ye = min(ys + (int)job.seg, (int)(job.cy + job.ch));
    // RGB formats take RGB tiles, gray formats gray ones (the host maps them
    // so), so the format fixes the component count.
    constexpr int NC = (FMT == PACK_GRAY8 || FMT == PACK_GRAY16) ? 1 : 3;
    constexpr bool kU8 = FMT == PACK_GRAY8 || FMT == PACK_RGB8 || FMT == PACK_RGBA8;
    if (kU8 && job.bit_depth == 8) pack97_unit<NC, FMT, kU8>(job, x0, ys, ye, lane, rowbuf, tab, IK);
    else pack97_unit<NC, FMT, false>(job, x0, ys, ye, lane, rowbuf, tab, IK);
  };
  if (!QUEUE) {
    const uint32_t unit = blockIdx.x * kWarps97 + (threadIdx.x >> 5);
    if (unit < nunits) one(unit);
    return;
  }
  bool first = true;
  for (uint32_t unit; next_unit(queue, nunits, first, unit);) one(unit);
}

cudaError_t launch_idwt97_level(const IdwtJob* jobs, uint32_t njobs, uint32_t nunits, cudaStream_t stream,
                                uint32_t* queue, uint32_t persistent_ctas) {
  if (njobs == 0 || nunits == 0) return cudaSuccess;
  uint32_t ctas = (nunits + kIdwtWarps - 1) / kIdwtWarps;
  if (queue) ctas = std::max(1u, std::min(ctas, persistent_ctas));
  if (queue) idwt97_level_kernel<true><<<ctas, kIdwtWarps * 32, 0, stream>>>(jobs, njobs, nunits, queue);
  else idwt97_level_kernel<false><<<ctas, kIdwtWarps * 32, 0, stream>>>(jobs, njobs, nunits, nullptr);
  return cudaGetLastError();
}

cudaError_t launch_pack97(const PackJob* jobs, uint32_t njobs, uint32_t nunits, uint32_t fmt, cudaStream_t stream,
                          uint32_t* queue, uint32_t persistent_ctas) {
  if (njobs == 0 || nunits == 0) return cudaSuccess;
  uint32_t ctas = (nunits + kWarps97 - 1) / kWarps97;
  if (queue) ctas = std::max(1u, std::min(ctas, persistent_ctas));
  const dim3 grid(ctas), block(kWarps97 * 32);
#define SGN_PACK97_LAUNCH(F)                                                                   \
  case F:                                                                                       \
    if (queue) pack97_kernel<F, true><<<grid, block, 0, stream>>>(jobs, njobs, nunits, queue); \
    else pack97_kernel<F, false><<<grid, block, 0, stream>>>(jobs, njobs, nunits, nullptr);    \
    break;
  switch (fmt) {
    SGN_PACK97_LAUNCH(PACK_GRAY8)
    SGN_PACK97_LAUNCH(PACK_RGB8)
    SGN_PACK97_LAUNCH(PACK_RGBA8)
    SGN_PACK97_LAUNCH(PACK_GRAY16)
    SGN_PACK97_LAUNCH(PACK_RGB16)
    default: return cudaErrorInvalidValue;
  }
#undef SGN_PACK97_LAUNCH
  return cudaGetLastError();
}

cudaError_t launch_idwt_level(const IdwtJob* jobs, uint32_t njobs, uint32_t nunits, cudaStream_t stream,
                              uint32_t* queue, uint32_t persistent_ctas, bool lean) {
  if (njobs == 0 || nunits == 0) return cudaSuccess;
  uint32_t ctas = (nunits + kIdwtWarps - 1) / kIdwtWarps;
  if (queue) ctas = std::max(1u, std::min(ctas, persistent_ctas));
  if (queue) idwt_level_kernel<true><<<ctas, kIdwtWarps * 32, 0, stream>>>(jobs, njobs, nunits, queue);
  else if (lean) idwt_level_lean_kernel<<<ctas, kIdwtWarps * 32, 0, stream>>>(jobs, njobs, nunits);
  else idwt_level_kernel<false><<<ctas, kIdwtWarps * 32, 0, stream>>>(jobs, njobs, nunits, nullptr);
  return cudaGetLastError();
}

namespace {

template <int F, int NC, bool D>
cudaError_t launch_pack_variant(const PackJob* jobs, uint32_t njobs, uint32_t nunits, dim3 grid, cudaStream_t stream,
                                uint32_t* queue) {
  if (queue) pack_kernel<F, NC, D, true><<<grid, kIdwtWarps * 32, 0, stream>>>(jobs, njobs, nunits, queue);
  else pack_kernel<F, NC, D, false><<<grid, kIdwtWarps * 32, 0, stream>>>(jobs, njobs, nunits, nullptr);
  return cudaGetLastError();
}

// RGB formats take RGB tiles (variants 0, 1), gray formats gray ones (2, 3).
template <int F>
cudaError_t launch_pack_format(uint32_t variant, const PackJob* jobs, uint32_t njobs, uint32_t nunits, dim3 grid,
                               cudaStream_t stream, uint32_t* queue) {
  if constexpr (F == PACK_GRAY8 || F == PACK_GRAY16) {
    if (variant == 2) return launch_pack_variant<F, 1, true>(jobs, njobs, nunits, grid, stream, queue);
    if (variant == 3) return launch_pack_variant<F, 1, false>(jobs, njobs, nunits, grid, stream, queue);
  } else {
    if (variant == 0) return launch_pack_variant<F, 3, true>(jobs, njobs, nunits, grid, stream, queue);
    if (variant == 1) return launch_pack_variant<F, 3, false>(jobs, njobs, nunits, grid, stream, queue);
  }
  return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_pack(const PackJob* jobs, uint32_t njobs, uint32_t nunits, uint32_t fmt, uint32_t variant,
                        cudaStream_t stream, uint32_t* queue, uint32_t persistent_ctas) {
  if (njobs == 0 || nunits == 0) return cudaSuccess;
  uint32_t ctas = (nunits + kIdwtWarps - 1) / kIdwtWarps;
  if (queue) ctas = std::max(1u, std::min(ctas, persistent_ctas));
  const dim3 grid(ctas);
  switch (fmt) {
    case PACK_GRAY8: return launch_pack_format<PACK_GRAY8>(variant, jobs, njobs, nunits, grid, stream, queue);
    case PACK_RGB8: return launch_pack_format<PACK_RGB8>(variant, jobs, njobs, nunits, grid, stream, queue);
    case PACK_RGBA8: return launch_pack_format<PACK_RGBA8>(variant, jobs, njobs, nunits, grid, stream, queue);
    case PACK_GRAY16: return launch_pack_format<PACK_GRAY16>(variant, jobs, njobs, nunits, grid, stream, queue);
    case PACK_RGB16: return launch_pack_format<PACK_RGB16>(variant, jobs, njobs, nunits, grid, stream, queue);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t idwt_pack_occupancy(uint32_t fmt, int* idwt_ctas_per_sm, int* pack_ctas_per_sm) {
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(idwt_ctas_per_sm, idwt_level_kernel<true>,
                                                                kIdwtWarps * 32, 0);
  if (e != cudaSuccess) return e;
  // Every variant has the same launch bounds and shared memory; the direct
  // one of the format stands for them.
  switch (fmt) {
#define SGN_PACK_OCC(F)                                                                                    \
    case F:                                                                                                 \
      return cudaOccupancyMaxActiveBlocksPerMultiprocessor(                                                 \
          pack_ctas_per_sm, pack_kernel<F, (F == PACK_GRAY8 || F == PACK_GRAY16) ? 1 : 3, true, true>,     \
          kIdwtWarps * 32, 0);
    SGN_PACK_OCC(PACK_GRAY8)
    SGN_PACK_OCC(PACK_RGB8)
    SGN_PACK_OCC(PACK_RGBA8)
    SGN_PACK_OCC(PACK_GRAY16)
    SGN_PACK_OCC(PACK_RGB16)
#undef SGN_PACK_OCC
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace sgn
