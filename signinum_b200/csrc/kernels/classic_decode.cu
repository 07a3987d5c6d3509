// Classic JPEG 2000 Tier-1 (EBCOT) code-block decoding on sm_100a.
//
// The arithmetic follows the reference's CPU decoder exactly
// (crates/signinum-j2k-native/src/j2c/arithmetic_decoder.rs: the MQ decoder
// of Annex C with 0xFF past the end of a segment; bitplane.rs: the cleanup,
// significance propagation and magnitude refinement passes of Annex D with
// run-length and uniform contexts, vertically causal contexts, context reset,
// segmentation symbols, termination on every pass and arithmetic-coding
// bypass with raw sign bits).  Coefficients come out as int32 values
// (sign x magnitude, bit 0 the least significant decoded bit-plane), the
// layout the HT kernels write, so the IDWT and pack kernels run unchanged.
//
// Mapping: the MQ decoder is one serial chain per code block, so a lane
// decodes a block, `lanes` of them per warp, each taking blocks from a device
// counter.  The lanes of a warp are at different places of different blocks,
// so the decoder is one loop that every lane runs in step: an iteration steps
// to the next column when the current one is done, picks the next sample that
// the pass codes, decodes one binary decision (zero coding, sign, refinement,
// run length or uniform, whichever the lane's position asks for) through the
// one copy of the MQ decoder, and applies its bit.  Rare events (stripe, pass
// and block ends, raw segments) are branches; the rest is straight-line code
// under selects, whose independent parts (column step, probability update,
// renormalisation) overlap.
//
// A stripe column's state is one 16-bit word (significance, sign, refined and
// coded flags of its four samples) in shared memory, or, for plans of more
// blocks than that holds at once, in global scratch behind L1.  A column and its two
// neighbours, each joined with the samples above and below the stripe, hold
// the whole context window; they sit in registers while the column is coded,
// and the next column's words are loaded one column ahead.
//
// What bounds it: the chain of decisions of the plan's longest block, every
// iteration a fixed-latency path of table loads and selects in a warp that has
// its scheduler almost to itself.  In one 512 x 512 RGB tile of the uniform
// batch the longest block takes 33,302 iterations, 25,850 of them a decision
// (the others step over a column that the pass does not code): 13.7 ms, 810
// cycles for the 220 instructions of an iteration, with one block per warp
// (210 of them); 18.3 ms with all of them in seven warps.  64 tiles (13,440
// blocks): 41.6 ms with a thread per block and nested pass loops, whose 32
// lanes took turns at their branches (10.5 M warp instructions per warp), 21.1
// ms in this form with 16 blocks per warp.  The same loop with a branch per
// kind of decision took 27 ms (24 ms for one tile with 16 blocks per warp).
// 256 tiles (53,760 blocks, words in scratch) 66 -> 38 ms.
#include <algorithm>
#include <cstdint>

#include "../device_plan.h"
#include "../ebcot.h"
#include "kernels.h"

namespace sgn {
namespace {

using namespace ebcot;

// One warp per CTA; at most 32 blocks in flight per CTA, whose column words
// share one pool (16 blocks of 64 x 64).
constexpr uint32_t kClassicThreads = 32, kClassicBlocks = 32;
constexpr uint32_t kClassicPool = 16 * classic_slot_words(64, 64);

// Column word in shared memory: bits 0..3 significant, 4..7 refined, 8..11
// sign, 12..15 coded in this bit-plane (rows 0 .. 3 of the stripe).  In
// registers, joined with the rows above and below (join): bits 0..5
// significance of rows -1 .. 4, bits 8..13 their signs, 16..19 refined,
// 24..27 coded.
constexpr int kSgnBit = 8, kRefBit = 16, kCodBit = 24;
constexpr uint32_t kCodMask = 0xFu << kCodBit;

__device__ __forceinline__ uint32_t join(uint32_t above, uint32_t own, uint32_t below) {
  return ((own & 0x0F0Fu) << 1) | ((own & 0xF0F0u) << 12) | ((above >> 3) & 0x0101u) | ((below & 0x0101u) << 5);
}
__device__ __forceinline__ uint16_t own_word(uint32_t c) {
  return (uint16_t)(((c >> 1) & 0x0F0Fu) | ((c >> 12) & 0xF0F0u));
}

// The 3 x 3 significance window of row k from the columns' significance
// bits Q (left | centre << 9 | right << 18, rows -1 .. 4 from bit 0): the
// three rows k-1 .. k+1 of the left column in bits 0..2, of the centre in
// 3..5 (the sample itself bit 4), of the right in 6..8.
__device__ __forceinline__ uint32_t zc_index(uint32_t Q, uint32_t k) {
  const uint32_t t = (Q >> k) & 0x1C0E07u;
  return (t | (t >> 6) | (t >> 12)) & 0x1FFu;
}
constexpr uint32_t kCentre = 1u << 4;

// The neighbour-significance byte of ebcot.h for a window index.
__device__ __forceinline__ uint8_t window_byte(uint32_t i) {
  return (uint8_t)(((i & 1) << 7) | (((i >> 3) & 1) << 6) | (((i >> 6) & 1) << 5) | (((i >> 1) & 1) << 4) |
                   (((i >> 2) & 1) << 3) | (((i >> 7) & 1) << 2) | (((i >> 8) & 1) << 1) | ((i >> 5) & 1));
}

// Significance (bits 0..3) and signs (bits 4..7) of the left, right, upper
// and lower neighbours of row k from the column words.
__device__ __forceinline__ uint32_t sign_index(uint32_t L, uint32_t C, uint32_t R, uint32_t k) {
  const uint32_t l = (L >> (k + 1)) & 0x101u, r = (R >> (k + 1)) & 0x101u, c = C >> k;
  const uint32_t v = l | (r << 1) | ((c & 0x101u) << 2) | (((c >> 2) & 0x101u) << 3);
  return (v | (v >> 4)) & 0xFFu;
}
// Its byte of sc_context: two bits (negative, positive) per neighbour, top,
// left, right, bottom from the high end.
__device__ __forceinline__ uint8_t sign_byte(uint32_t i) {
  uint32_t m = 0;
  const uint32_t place[4] = {4, 2, 6, 0};  // left, right, upper, lower
  for (int n = 0; n < 4; ++n)
    if ((i >> n) & 1) m |= 1u << (place[n] + ((i >> (4 + n)) & 1));
  return (uint8_t)m;
}

// A context's adaptive state is its word of the probability table (Table
// C.2) for (index, MPS): qe, bits 16..22 the entry after an MPS, 23..29 the
// entry after an LPS (the MPS switched where the table says so), bit 31 the
// MPS; entry 2 * index + MPS.
template <uint32_t POOL>
struct Tables {
  uint32_t state[94];
  uint8_t zc[3][512];  // zero-coding label by window index (zc_index)
  uint8_t sc[256];     // sign label | xor << 7 by sign index (sign_index)
  uint32_t cx[19][kClassicBlocks];
  uint16_t cols[POOL];
};

// The MQ decoder of Annex C (C in the inverted form of the reference).  The
// current byte and the one after it are held, so that a refill never waits
// for the byte it appends.
struct MqDec {
  const uint8_t* d;
  uint32_t len, bp, b0, b1, c, a, ct;
  __device__ __forceinline__ uint32_t byte_at(uint32_t i) const { return i < len ? (uint32_t)__ldg(d + i) : 0xFFu; }
  __device__ __forceinline__ void bytein() {
    const uint32_t stuffed = b0 == 0xFF ? 1u : 0u;
    const bool end = stuffed && b1 > 0x8F;  // a marker: zeros (ones in the reference's form) from here on
    c += end ? 0u : 0xFF00u - (stuffed << 8) - (b1 << (8 + stuffed));
    ct = end ? 8 : 8 - stuffed;
    if (!end) {
      ++bp;
      b0 = b1;
      b1 = byte_at(bp + 1);
    }
  }
  __device__ __forceinline__ void init(const uint8_t* data, uint32_t n) {
    d = data;
    len = n;
    bp = 0;
    b0 = byte_at(0);
    b1 = byte_at(1);
    c = (b0 ^ 0xFFu) << 16;
    bytein();
    c <<= 7;
    ct -= 7;
    a = 0x8000;
  }
  // One decision with a context whose state is e; an e of 0 changes nothing
  // and gives 0.  *cx receives the context's next state.  (In a valid stream
  // C stays below A.  A byte 0x80 .. 0x8F after 0xFF can take bytein below
  // zero, as it does in the reference, so an e of 0 is told apart by its q and
  // not by C: A is then never 0, and the renormalisation shifts by at most 15.)
  __device__ __forceinline__ uint32_t decode(uint32_t e, uint32_t* cx, const uint32_t* state) {
    const uint32_t q = e & 0xFFFFu, rest = a - q;
    const bool low = q != 0 && (c >> 16) >= rest;  // the LPS sub-interval
    const bool lps = low != (rest < q);   // with the conditional exchange
    c -= low ? rest << 16 : 0u;
    a = low ? q : rest;
    // RENORMD (C.3.3), as many bits at once as A needs and the byte buffer
    // holds (as the reference's renormalize does); a decision seldom needs
    // more than one byte.
    uint32_t sh = (uint32_t)__clz(a) - 16;
    if (sh) *cx = state[(e >> (lps ? 23 : 16)) & 0x7Fu];
    a <<= sh;
    uint32_t s1 = min(sh, ct);
    c <<= s1;
    ct -= s1;
    sh -= s1;
    if (sh) bytein();
    s1 = min(sh, ct);
    c <<= s1;
    ct -= s1;
    sh -= s1;
    while (sh) {
      bytein();
      s1 = min(sh, ct);
      c <<= s1;
      ct -= s1;
      sh -= s1;
    }
    return (e >> 31) ^ (lps ? 1u : 0u);
  }
  // A bypassed segment: d, len, and bp as a bit position.
  __device__ __forceinline__ void init_raw(const uint8_t* data, uint32_t n) {
    d = data;
    len = n;
    bp = 0;
  }
};

// The raw bit at position p of a bypassed segment (bit 0 of the result, the
// next position above it): packet-header stuffing; 1 past the end or on a bad
// stuff bit (the reference's non-strict BypassDecoder).
__device__ __noinline__ uint32_t raw_bit(const uint8_t* d, uint32_t len, uint32_t p) {
  if ((p >> 3) >= len) return (p << 1) | 1u;
  const uint32_t byte = __ldg(d + (p >> 3));
  uint32_t b = (byte >> (7 - (p & 7))) & 1u;
  const bool stuff = (p & 7) == 7 && byte == 0xFF;
  ++p;
  if (stuff) {
    if ((p >> 3) >= len) return (p << 1) | 1u;
    b |= (__ldg(d + (p >> 3)) >> (7 - (p & 7))) & 1u;
    ++p;
  }
  return (p << 1) | b;
}

// What a lane's next decision is.
enum Step : uint32_t { kNext, kZero, kSign, kRefine, kRun, kUniform1, kUniform2, kSegSymbol };

}  // namespace

// Table C.2 packed per index: qe | nmps << 16 | nlps << 23 | switch << 30
// (built on the host from ebcot.h and passed by value).
struct QeTable {
  uint32_t e[47];
};

// slot_words: the 16-bit words of the plan's largest block
// (classic_slot_words); lanes: the blocks the CTA's warp has in flight.  Their
// column words are in the CTA's shared pool (lanes x slot_words at most
// kClassicPool), or with SCRATCH in `scratch`, one slot per lane.
template <bool SCRATCH>
__global__ void __launch_bounds__(kClassicThreads) classic_kernel(
    const ClassicJob* __restrict__ jobs, const ClassicSeg* __restrict__ segs, uint32_t njobs,
    const uint8_t* __restrict__ arena, const uint8_t* __restrict__ gather, int32_t* __restrict__ coef,
    uint16_t* scratch, uint32_t slot_words, uint32_t* queue, QeTable qt, uint32_t lanes) {
  __shared__ Tables<SCRATCH ? 2 : kClassicPool> t;
  for (uint32_t i = threadIdx.x; i < 94; i += blockDim.x) {
    const uint32_t e = qt.e[i >> 1], mps = i & 1;
    const uint32_t nm = 2 * ((e >> 16) & 0x7Fu) + mps, nl = 2 * ((e >> 23) & 0x7Fu) + (mps ^ (e >> 30));
    t.state[i] = (e & 0xFFFFu) | (nm << 16) | (nl << 23) | (mps << 31);
  }
  for (uint32_t i = threadIdx.x; i < 512; i += blockDim.x) {
    const uint8_t n = window_byte(i);
    t.zc[0][i] = zc_context(n, kLlLh);
    t.zc[1][i] = zc_context(n, kHl);
    t.zc[2][i] = zc_context(n, kHh);
  }
  for (uint32_t i = threadIdx.x; i < 256; i += blockDim.x) {
    uint8_t label, xr;
    sc_context(sign_byte(i), label, xr);
    t.sc[i] = (uint8_t)(label | (xr << 7));
  }
  __syncthreads();
  const uint32_t id = threadIdx.x;
  if (id >= lanes) return;
  uint16_t* const slot =
      SCRATCH ? scratch + ((size_t)blockIdx.x * lanes + id) * slot_words : t.cols + id * slot_words;

  // The lane's block.
  ClassicJob job;
  job.passes = job.bitplanes = job.style = 0;
  job.seg = 0;
  uint32_t w = 0, h = 0, stride = 0, vcut = 0;
  const uint8_t* data = nullptr;
  uint32_t* out = nullptr;
  const uint8_t* zc = t.zc[0];
  // Its segments: passes [.., seg_end) come from the open decoder.
  uint32_t nseg = 0, seg = 0, seg_end = 0, npasses = 0, off = 0;
  bool raw = false;
  MqDec dec;
  dec.init_raw(nullptr, 0);
  dec.c = dec.a = dec.ct = dec.b0 = dec.b1 = 0;
  // Its position: pass, stripe, column, row, and the column words around it.
  uint32_t pass = 0, kind = 0, one = 0, y0 = 0, x = 0, k = 0, rows = 0, cand = 0;
  uint32_t L = 0, C = 0, R = 0, N = 0, old = 0, Q = 0;
  int up = 0, down = 0;            // to the words above and below (0: none, or not to be seen)
  uint32_t upm = 0, downm = 0;     // all ones where there are such words
  uint32_t leave = 0;              // flags a column keeps when the pass leaves it
  uint16_t* f = slot;              // the current column's word
  uint32_t* col = nullptr;         // the current column's top sample
  uint32_t step = kNext, label = 0, flip = 0, symbols = 0;
  bool open = false;  // a block is being decoded
  auto reset_contexts = [&]() {
    for (int i = 0; i < 19; ++i) t.cx[i][id] = t.state[2 * initial_index(i)];
  };
  // The joined word of the column d after the current one (zero past the
  // block's right edge).
  auto column = [&](uint32_t d) -> uint32_t {
    const bool in = x + d < w;
    const uint16_t* p = f + (in ? d : 0);
    const uint32_t v = join(p[up] & upm, p[0], p[down] & downm);
    return in ? v : 0u;
  };
  auto stripe_begin = [&]() {
    f = slot + (y0 >> 2) * w;
    col = out + (size_t)y0 * stride;
    rows = (1u << min(4u, h - y0)) - 1;
    const bool above = y0 > 0, below = y0 + 4 < h && !vcut;
    up = above ? -(int)w : 0;
    upm = above ? ~0u : 0u;
    down = below ? (int)w : 0;
    downm = below ? ~0u : 0u;
    x = 0;
    L = 0;
    old = C = column(0);
    R = column(1);
    N = column(2);
  };
  auto pass_begin = [&]() {
    kind = pass % 3;
    one = 1u << ((uint32_t)job.bitplanes - 1 - (pass + 2) / 3);
    leave = kind == 0 ? ~kCodMask : ~0u;  // the cleanup pass ends the bit-plane
    y0 = 0;
    stripe_begin();
  };
  // The next pass, in its segment, or the next block's first pass; false
  // when there is no block left.
  auto next_pass = [&]() -> bool {
    symbols = 0;
    if (open) {
      if (job.style & kReset) reset_contexts();
      ++pass;
    }
    for (;;) {
      if (open && pass < npasses && pass < seg_end) break;
      if (open && seg < nseg && pass < npasses) {
        // (Only with one segment per terminated run of passes.)
        const ClassicSeg s = segs[job.seg + seg];
        raw = !segment_is_arithmetic(job.style, seg_end);
        if (raw) dec.init_raw(data + off, s.len);
        else dec.init(data + off, s.len);
        seg_end += s.passes;
        off += s.len;
        ++seg;
        continue;
      }
      open = false;
      const uint32_t j = atomicAdd(queue, 1u);
      if (j >= njobs) return false;
      job = jobs[j];
      w = job.w;
      h = job.h;
      stride = job.stride;
      out = reinterpret_cast<uint32_t*>(coef + job.dst);
      if (((job.dst | stride | w) & 3) == 0) {
        for (uint32_t y = 0; y < h; ++y)
          for (uint32_t i = 0; i < w; i += 4)
            *reinterpret_cast<uint4*>(out + (size_t)y * stride + i) = make_uint4(0, 0, 0, 0);
      } else {
        for (uint32_t y = 0; y < h; ++y)
          for (uint32_t i = 0; i < w; ++i) out[(size_t)y * stride + i] = 0;
      }
      if (job.passes == 0 || job.bitplanes == 0) continue;
      // The block's segments, in the input or (multi-layer) in the gather
      // area.
      data = (job.src & kClassicGathered) ? gather + (job.src & ~kClassicGathered) : arena + job.src;
      const uint32_t words = w * ((h + 3) >> 2);
      for (uint32_t i = 0; i < words; ++i) slot[i] = 0;
      vcut = (job.style & kVCausal) ? 1 : 0;  // a stripe does not see the row below it
      zc = t.zc[job.band_class];
      reset_contexts();
      npasses = 1 + 3 * ((uint32_t)job.bitplanes - 1);
      pass = 0;
      nseg = job.nseg;
      seg = 0;
      seg_end = 0;
      off = 0;
      raw = false;
      if (!(job.style & (kBypass | kTermAll))) {
        // One codeword for all passes.
        uint32_t total = 0;
        for (uint32_t i = 0; i < nseg; ++i) total += segs[job.seg + i].len;
        dec.init(data, total);
        npasses = min(npasses, (uint32_t)job.passes);
        seg_end = npasses;
        seg = nseg;
      }
      open = true;
    }
    pass_begin();
    return true;
  };

  for (;;) {
    // The next column of the stripe, when the current one is done.  (f stays
    // inside the slot: the last column's step is undone by stripe_begin or
    // next_pass, or reads nothing.)
    const bool turn = step == kNext && cand == 0;
    if (turn) {
      C &= leave;
      if (C != old) *f = own_word(C);
      L = C;
      old = C = R;
      R = N;
      ++x;
      ++f;
      ++col;
      if (x >= w) {
        // The next stripe, pass or block.
        f = slot;
        if (open && x == w && y0 + 4 < h) {
          y0 += 4;
          stripe_begin();
        } else if (open && kind == 0 && (job.style & kSegSym) && symbols < 4) {
          // Four uniform symbols end the cleanup pass.
          step = kSegSymbol;
          label = 18;
          rows = 0;
          old = C = 0;
        } else if (!next_pass()) {
          return;
        }
      } else {
        N = column(2);
      }
    }
    // The rows of this column that the pass codes.
    const uint32_t own = C >> 1, around = L | C | R, any = around | (around >> 2) | ((L | R) >> 1);
    const uint32_t all = (kind == 1 ? any : ~(C >> kCodBit)) & (kind == 2 ? own : ~own) & rows;
    cand = turn ? all : cand;
    Q = (L & 0x3Fu) | ((C & 0x3Fu) << 9) | ((R & 0x3Fu) << 18);
    const bool run = turn && kind == 0 && all == 0xFu && Q == 0;
    // The next sample of the column.
    const bool pick = step == kNext && !run && cand != 0;
    k = pick ? (uint32_t)__ffs((int)cand) - 1 : k;
    cand &= pick ? cand - 1 : ~0u;
    const uint32_t i = zc_index(Q, k);
    const uint32_t refine = ((C >> (kRefBit + k)) & 1u) ? 16u : (i & ~kCentre) ? 15u : 14u;
    const uint32_t zl = zc[i];
    label = run ? 17u : pick ? (kind == 2 ? refine : zl) : label;
    step = run ? (uint32_t)kRun : pick ? (kind == 2 ? (uint32_t)kRefine : (uint32_t)kZero) : step;
    // Its decision (none when the column codes no sample).
    uint32_t bit;
    if (raw) {
      bit = 0;
      if (step != kNext) {
        bit = raw_bit(dec.d, dec.len, dec.bp);
        dec.bp = bit >> 1;
        bit &= 1u;
      }
    } else {
      uint32_t* const cx = &t.cx[label][id];
      const uint32_t e = *cx;
      bit = dec.decode(step == kNext ? 0u : e, cx, t.state);
    }
    const bool zero = step == kZero, sign = step == kSign, refined = step == kRefine;
    const uint32_t s = bit ^ flip;  // (of a sign decision)
    // A sample's value: its first magnitude bit with its sign, then the
    // refinement bits added to it.
    const bool neg = sign ? s != 0 : ((C >> (kSgnBit + 1 + k)) & 1u) != 0;
    const uint32_t v = neg ? 0u - one : one;
    uint32_t* const px = col + (size_t)(k * stride);
    if (sign) *px = v;
    if (refined && bit) atomicAdd(px, v);
    const uint32_t set = sign ? 2u | (s << (kSgnBit + 1)) : refined ? 1u << kRefBit : zero && kind == 1 ? 1u << kCodBit : 0u;
    C |= set << k;
    // Significance propagation: the sample below has a neighbour now.
    cand |= sign && kind == 1 ? (2u << k) & ~(C >> 1) & rows : 0u;
    // The next step: a sign after a zero-coding 1 or the second uniform
    // symbol (the rows after that one are then coded one by one), a run's
    // uniform symbols, otherwise the next sample.
    const bool u1 = step == kUniform1, u2 = step == kUniform2, ran = step == kRun;
    k = u1 ? bit << 1 : u2 ? k | bit : k;
    cand = ran ? 0u : u2 ? 0xFu & ~((2u << k) - 1) : cand;
    symbols += step == kSegSymbol ? 1u : 0u;
    const bool to_sign = (zero && bit) || u2;
    const uint32_t next = ran && bit ? (uint32_t)kUniform1 : u1 ? (uint32_t)kUniform2 : (uint32_t)kNext;
    step = to_sign ? (uint32_t)kSign : step == kSegSymbol && symbols < 4 ? (uint32_t)kSegSymbol : next;
    const uint32_t e = t.sc[sign_index(L, C, R, k)];
    flip = raw ? 0u : e >> 7;
    label = to_sign ? e & 0x7Fu : 18u;
  }
}

cudaError_t launch_classic(const ClassicJob* jobs, const ClassicSeg* segs, uint32_t njobs, const uint8_t* arena,
                           const uint8_t* gather, int32_t* coef, uint16_t* scratch, uint32_t slot_words, uint32_t ctas,
                           uint32_t lanes, uint32_t* queue, cudaStream_t stream) {
  if (njobs == 0) return cudaSuccess;
  if (!queue || ctas == 0 || lanes == 0 || lanes > kClassicBlocks || (!scratch && lanes * slot_words > kClassicPool))
    return cudaErrorInvalidValue;
  QeTable qt;
  for (int i = 0; i < 47; ++i)
    qt.e[i] = kQe[i] | ((uint32_t)kNmps[i] << 16) | ((uint32_t)kNlps[i] << 23) | ((uint32_t)kSwitch[i] << 30);
  if (scratch)
    classic_kernel<true><<<ctas, kClassicThreads, 0, stream>>>(jobs, segs, njobs, arena, gather, coef, scratch,
                                                               slot_words, queue, qt, lanes);
  else
    classic_kernel<false><<<ctas, kClassicThreads, 0, stream>>>(jobs, segs, njobs, arena, gather, coef, nullptr,
                                                                slot_words, queue, qt, lanes);
  return cudaGetLastError();
}

uint32_t classic_max_lanes(uint32_t slot_words) {
  return std::max(1u, std::min(kClassicBlocks, kClassicPool / std::max(1u, slot_words)));
}

uint32_t classic_ctas_per_sm() {
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, classic_kernel<false>, kClassicThreads, 0) != cudaSuccess ||
      n < 1)
    n = 1;
  return (uint32_t)n;
}

uint32_t classic_scratch_ctas_per_sm() {
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, classic_kernel<true>, kClassicThreads, 0) != cudaSuccess ||
      n < 1)
    n = 1;
  return (uint32_t)n;
}

}  // namespace sgn
