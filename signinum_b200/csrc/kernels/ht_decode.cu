// HT code-block decoding on sm_100a.
//
// Decodes HTJ2K code blocks (T.814) into sign-magnitude coefficients and
// writes them as int32 sub-band samples, bit-exact with the reference's
// decode_impl (crates/signinum-j2k-native/src/j2c/ht_block_decode.rs:1563-1683)
// followed by coefficient_to_i32 (:225-234).
//
// Work mapping, in two passes over the blocks of a launch (ordered by coded
// length on the host, so neighbouring blocks carry similar work):
//  1. ht_vlc_kernel: one lane per code block runs the MEL / CxtVLC / UVLC
//     chain, the only inherently serial part of the cleanup pass, and writes
//     one 32-bit symbol per quad to a scratch table;
//  2. ht_magsgn_kernel: one warp per code block decodes magnitudes and signs,
//     a quad per lane, with a warp prefix scan of per-quad bit counts over the
//     block's unstuffed MagSgn stream staged in shared memory, and writes
//     whole rows with coalesced stores; blocks at most 32 wide without
//     refinement passes go two per warp, one per half-warp.
// Plans of few blocks run both passes in ht_cleanup_fused_kernel instead: a
// CTA per block, whose MagSgn warp follows the block's VLC chain row by row.
// Refinement passes (SigProp/MagRef) run in ht_refine_kernel for the few
// blocks that carry them.
#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "../device_plan.h"
#include "../ht_tables.h"
#include "kernels.h"

namespace sgn {

__device__ __align__(16) HtDecodeTables g_ht_tables;

namespace {

constexpr int kHtThreads = 128;
constexpr uint32_t kStatusDecode = 1u;

struct SmemTables {
  uint16_t vlc0[1024];
  uint16_t vlc1[1024];
  uint16_t uvlc0[320];
  uint16_t uvlc1[256];
};

__device__ __forceinline__ uint8_t ld8(const uint8_t* p) { return __ldg(p); }

// MEL bit-buffer refill, out of line (it runs once every several runs, and
// inlined its byte loop would sit in every step of the VLC chain): appends
// bytes until more than 56 bits are buffered.  After a 0xFF byte the next
// byte carries 7 bits; the last byte is ORed with 0x0F and the stream
// continues with 0xFF bytes.  State passed and returned by value, so it
// stays in registers.
struct MelFill {
  uint64_t buf;
  uint32_t pos, remaining, unstuff;
  int bits;
};
// The out-of-line refill loop.  While 32 bits or fewer are buffered, four
// bytes that are not the segment's last, after a byte that is not 0xFF and
// with no 0xFF among their first three (each then carries 8 bits) go in as
// one word from four independent loads; other bytes one at a time.  (The
// inline form keeps the byte loop alone: the word step measured slower
// inlined in the chain.)
__device__ __forceinline__ void mel_fill(const uint8_t* data, MelFill& f) {
  while (f.bits <= 56) {
    if (f.bits <= 32 && f.remaining >= 5 && !f.unstuff) {
      const uint8_t* p = data + f.pos;
      const uint32_t b0 = __ldg(p), b1 = __ldg(p + 1), b2 = __ldg(p + 2), b3 = __ldg(p + 3);
      if (b0 != 0xFF && b1 != 0xFF && b2 != 0xFF) {
        f.buf |= (uint64_t)((b0 << 24) | (b1 << 16) | (b2 << 8) | b3) << (32 - f.bits);
        f.bits += 32;
        f.pos += 4;
        f.remaining -= 4;
        f.unstuff = b3 == 0xFF;
        continue;
      }
    }
    uint32_t b;
    if (f.remaining > 0) {
      b = __ldg(data + f.pos);
      ++f.pos;
      --f.remaining;
    } else {
      b = 0xFF;
    }
    if (f.remaining == 0) b |= 0x0F;
    const int nb = 8 - (int)f.unstuff;
    f.buf |= (uint64_t)(b & ((1u << nb) - 1)) << (64 - f.bits - nb);
    f.bits += nb;
    f.unstuff = b == 0xFF;
  }
}
__device__ __noinline__ MelFill mel_refill(const uint8_t* data, MelFill f) {
  mel_fill(data, f);
  return f;
}

// MEL run decoder (ht_block_decode.rs:782-880).  The reference decodes runs
// into a small queue; here each run is decoded when it is needed, from a
// 64-bit buffer of unstuffed MEL bits (most significant bit first), with no
// inner loop: lanes of a warp decode different blocks, so a short fixed
// sequence per run diverges far less than a queue refill.
template <bool OUTLINE>
struct MelT {
  const uint8_t* data;
  uint32_t pos, remaining, unstuff;
  uint64_t buf;  // unread bits, left-aligned
  int bits, k;
  __device__ void init(const uint8_t* d, uint32_t lcup, uint32_t scup) {
    data = d;
    pos = lcup - scup;
    remaining = scup - 1;
    unstuff = 0;
    buf = 0;
    bits = 0;
    k = 0;
  }
  // OUTLINE: the refill is the out-of-line mel_refill; otherwise its loop
  // is inlined (which is faster depends on the batch: the autotuner picks).
  __device__ __forceinline__ void refill() {
    if constexpr (OUTLINE) {
      const MelFill f = mel_refill(data, MelFill{buf, pos, remaining, unstuff, bits});
      buf = f.buf;
      pos = f.pos;
      remaining = f.remaining;
      unstuff = f.unstuff;
      bits = f.bits;
    } else {
      while (bits <= 56) {
        uint32_t b;
        if (remaining > 0) {
          b = ld8(data + pos);
          ++pos;
          --remaining;
        } else {
          b = 0xFF;
        }
        if (remaining == 0) b |= 0x0F;
        const int nb = 8 - (int)unstuff;
        buf |= (uint64_t)(b & ((1u << nb) - 1)) << (64 - bits - nb);
        bits += nb;
        unstuff = b == 0xFF;
      }
    }
  }
  __device__ __forceinline__ int get_run() {
    if (bits < 6) refill();
    // MEL exponent table {0,0,0,1,1,1,2,2,2,3,3,4,5}, 3 bits per state.
    constexpr uint64_t kExp = (0ull << 0) | (0ull << 3) | (0ull << 6) | (1ull << 9) | (1ull << 12) | (1ull << 15) |
                              (2ull << 18) | (2ull << 21) | (2ull << 24) | (3ull << 27) | (3ull << 30) |
                              (4ull << 33) | (5ull << 36);
    const int e = (int)((kExp >> (3 * k)) & 7);
    const bool first = (buf >> 63) != 0;
    const uint32_t v = e ? (uint32_t)((buf << 1) >> (64 - e)) : 0u;
    const int used = first ? 1 : 1 + e;
    k = first ? min(k + 1, 12) : max(k - 1, 0);
    buf <<= used;
    bits -= used;
    return first ? ((1 << e) - 1) << 1 : (int)((v << 1) | 1);
  }
};

// Four bytes (highest address first) into the backward VLC reader's bit
// buffer one at a time, for words with a byte whose low 7 bits are all ones
// (after a byte above 0x8F such a byte loses its top bit to stuffing).  Out
// of line: it is the rare case of a refill.
struct VlcPush {
  uint64_t tmp;
  uint32_t bits, unstuff;
};
__device__ __noinline__ VlcPush vlc_push4(uint32_t wv, uint64_t tmp, uint32_t bits, uint32_t unstuff) {
#pragma unroll
  for (int k = 3; k >= 0; --k) {
    const uint32_t b = (wv >> (8 * k)) & 0xFF;
    const uint32_t db = 8 - ((unstuff && (b & 0x7F) == 0x7F) ? 1 : 0);
    tmp |= (uint64_t)b << bits;
    bits += db;
    unstuff = b > 0x8F;
  }
  return VlcPush{tmp, bits, unstuff};
}

// Backward VLC reader (ht_block_decode.rs:932-1000, new_vlc).
template <bool OUTLINE>
struct VlcT {
  const uint8_t* data;
  int pos;
  uint32_t remaining;
  uint64_t tmp;
  uint32_t bits, unstuff;
  // Word refills walk down 4 bytes at a time, so their two aligned words
  // are the previous refill's low word and the word below it: that one is
  // loaded a refill ahead (w_lo) and the refill itself never waits on memory.
  const uint32_t* wp;  // aligned word of the next refill's low half
  uint32_t w_lo, w_hi, sh8;
  __device__ void init(const uint8_t* d, uint32_t lcup, uint32_t scup) {
    data = d;
    uint32_t b = ld8(d + lcup - 2);
    tmp = b >> 4;
    bits = 4 - (((tmp & 7) == 7) ? 1 : 0);
    pos = (int)lcup - 3;
    remaining = scup - 2;
    unstuff = (b | 0x0F) > 0x8F;
    init_words();
  }
  // The MagRef reader (new_mrp, ht_block_decode.rs:1377-1433): the whole
  // refinement segment of n bytes from its last byte down, stuffing from the
  // start.
  __device__ void init_mrp(const uint8_t* d, uint32_t n) {
    data = d;
    tmp = 0;
    bits = 0;
    pos = (int)n - 1;
    remaining = n;
    unstuff = 1;
    init_words();
  }
  // Word-refill state for bytes pos - 3 .. pos; every initialiser calls it.
  __device__ __forceinline__ void init_words() {
    w_lo = w_hi = 0;
    wp = nullptr;
    sh8 = 0;
    if (remaining >= 4) {
      // Both words hold bytes of the segment (pos - 3 .. pos).
      const uintptr_t addr = (uintptr_t)(data + pos - 3);
      wp = reinterpret_cast<const uint32_t*>(addr & ~(uintptr_t)3);
      sh8 = (uint32_t)(addr & 3) * 8;
      w_lo = __ldg(wp);
      w_hi = sh8 ? __ldg(wp + 1) : 0u;
    }
  }
  __device__ __forceinline__ void push(uint32_t b) {
    const uint32_t db = 8 - ((unstuff && (b & 0x7F) == 0x7F) ? 1 : 0);
    tmp |= (uint64_t)b << bits;
    bits += db;
    unstuff = b > 0x8F;
  }
  // Appends bytes (walking backwards) until more than 32 bits are buffered;
  // past the segment the reader supplies zero bytes.  Four bytes at a time
  // come from one unaligned 32-bit read (two aligned loads inside the
  // segment), so the byte steps do not wait on one load each.
  __device__ __forceinline__ void fill() {
    while (bits <= 32) {
      if (remaining >= 4) {
        const uint32_t wv = __funnelshift_r(w_lo, w_hi, sh8);
        w_hi = w_lo;
        --wp;
        // The next word refill (when 4 more bytes remain) reads bytes down to
        // pos - 7, all inside the segment, so its low word is one of them.
        w_lo = remaining >= 8 ? __ldg(wp) : 0u;
        pos -= 4;
        remaining -= 4;
        if (__vcmpeq4(wv | 0x80808080u, 0xFFFFFFFFu) == 0) {
          // No byte has its low 7 bits all ones, so none loses a bit to
          // stuffing: the four bytes (highest address first) go in whole.
          tmp |= (uint64_t)__byte_perm(wv, 0, 0x0123) << bits;
          bits += 32;
          unstuff = (wv & 0xFF) > 0x8F;
        } else if constexpr (OUTLINE) {
          const VlcPush r = vlc_push4(wv, tmp, bits, unstuff);
          tmp = r.tmp;
          bits = r.bits;
          unstuff = r.unstuff;
        } else {
          push(wv >> 24);
          push((wv >> 16) & 0xFF);
          push((wv >> 8) & 0xFF);
          push(wv & 0xFF);
        }
      } else {
        uint32_t b = 0;
        if (remaining > 0) {
          b = ld8(data + pos);
          --pos;
          --remaining;
        }
        push(b);
      }
    }
  }
  __device__ __forceinline__ uint32_t fetch() {
    if (bits < 32) fill();
    return (uint32_t)tmp;
  }
  __device__ __forceinline__ uint32_t advance(uint32_t n) {
    tmp >>= n;
    bits -= n;
    return (uint32_t)tmp;
  }
};

// The refinement passes use the out-of-line forms.
using Mel = MelT<true>;
using Vlc = VlcT<true>;

// Forward reader with 0xFF stuffing (ht_block_decode.rs:888-930).
template <uint32_t PAD>
struct Fwd {
  const uint8_t* data;
  uint32_t len, pos;
  uint64_t tmp;
  uint32_t bits, unstuff;
  __device__ void init(const uint8_t* d, uint32_t n) {
    data = d;
    len = n;
    pos = 0;
    tmp = 0;
    bits = 0;
    unstuff = 0;
  }
  __device__ __forceinline__ void fill() {
    while (bits <= 32) {
      uint32_t b = pos < len ? (uint32_t)ld8(data + pos) : PAD;
      ++pos;
      tmp |= (uint64_t)b << bits;
      bits += 8 - unstuff;
      unstuff = b == 0xFF;
    }
  }
  __device__ __forceinline__ uint32_t fetch() {
    if (bits < 32) fill();
    return (uint32_t)tmp;
  }
  __device__ __forceinline__ void advance(uint32_t n) {
    tmp >>= n;
    bits -= n;
  }
};

__device__ __forceinline__ int32_t to_i32(uint32_t v, uint32_t nbp) {
  uint32_t shift = nbp >= 31 ? 0 : 31 - nbp;
  int32_t m = (int32_t)((v & 0x7FFFFFFFu) >> shift);
  return (v & 0x80000000u) ? -m : m;
}

// Row-above context of blocks at most 64 wide (REG): the significance of
// the two bottom samples of each quad (entry bits 5 and 7, the only part of
// a quad the row below takes its context from) in one 64-bit mask S, four
// bits per quad pair k at bits 4k .. 4k+3: {first quad's bit 5, second
// quad's bit 5, first quad's bit 7, second quad's bit 7}.  In that order a
// quad's two context bits from above (entry bits 7 and 9 of c_q: the left
// quad's bit 7 or its own bit 5; its own bit 7 or the right quad's bit 5)
// are ORs of adjacent bits of S: with Q = S | S >> 1, quad 2k takes
// Q[4k-1] and Q[4k+1], quad 2k+1 Q[4k+1] and Q[4k+3].
__device__ __forceinline__ uint32_t pair_nibble(uint32_t t0, uint32_t t1) {
  return (t0 & 0xA0u) | ((t1 & 0xA0u) << 1);  // the pair's four bits at bits 5 .. 8
}
// Appends a pair's nibble to the row mask under construction (pairs enter
// at the top and move down four bits per pair; the row's end aligns them).
__device__ __forceinline__ uint64_t push_nibble(uint64_t S, uint32_t nib) {
  return (S >> 4) | ((uint64_t)nib << 55);
}
// Context bit 8 of a quad from its left neighbour t in the same row (not
// the initial row): either of the neighbour's right-column samples.
__device__ __forceinline__ uint32_t left_ctx(uint32_t t) { return ((t & 0xC0u) + 0xC0u) & 0x100u; }

// CxtVLC / MEL / UVLC pass of one block (decode_cleanup_symbols,
// ht_block_decode.rs:1056-1205): the serial chain of the cleanup pass.  Writes
// one 32-bit symbol per quad (entry | u << 16) into the block's symbol table,
// quad rows of nq entries.  The row above gives the context: with REG (blocks
// at most 64 wide, nq <= 32) its two context bits per quad live in a 64-bit
// register, otherwise they are read back from the symbol table.
// After each quad row is in the symbol table, row_done(rows written so far)
// (the fused small-plan kernel publishes progress with it).  The row's pairs
// are staged at stage[pair * stage_stride + stage_slot].
struct NoRowHook {
  __device__ void operator()(uint32_t) const {}
};
template <bool REG, bool OUTLINE, typename RowHook = NoRowHook>
__device__ bool decode_vlc(const HtJob& job, const uint8_t* src, uint32_t* __restrict__ sym, const SmemTables& T,
                           uint2* __restrict__ stage, uint32_t stage_stride, uint32_t stage_slot,
                           RowHook row_done = RowHook()) {
  const uint32_t lcup = job.lcup, w = job.w, h = job.h;
  if (lcup < 2) return false;
  uint32_t scup = ((uint32_t)ld8(src + lcup - 1) << 4) + (ld8(src + lcup - 2) & 0x0F);
  if (scup < 2 || scup > lcup || scup > 4079) return false;
  MelT<OUTLINE> mel;
  mel.init(src, lcup, scup);
  VlcT<OUTLINE> vlc;
  vlc.init(src, lcup, scup);
  int run = mel.get_run();
  const uint32_t nq = (w + 1) / 2, qs = sym_row_stride(w);
  uint32_t* row = sym;
  // REG blocks whose rows hold a multiple of 4 symbols stage each row's
  // pairs in the lane's shared-memory column and write the row with 16-byte
  // stores (far fewer scattered store requests than one per pair).
  const bool staged = REG && (qs & 3) == 0;
  const uint32_t lanes = stage_stride, tid = stage_slot;
  auto put = [&](uint32_t q, uint32_t a, uint32_t b) {
    if (staged) stage[(q >> 1) * lanes + tid] = make_uint2(a, b);
    else *reinterpret_cast<uint2*>(row + q) = make_uint2(a, b);  // q even, rows padded to even
  };
  auto flush = [&]() {
    if constexpr (REG) {
      if (!staged) return;
      for (uint32_t k = 0; 2 * k < nq; k += 2) {
        const uint2 a = stage[k * lanes + tid];
        const uint2 b = 2 * (k + 1) < nq ? stage[(k + 1) * lanes + tid] : make_uint2(0, 0);
        *reinterpret_cast<uint4*>(row + 2 * k) = make_uint4(a.x, a.y, b.x, b.y);
      }
    }
  };
  // REG: the finished row's context mask S (pair_nibble); pairs enter it at
  // the top, so the row's end shifts it down by 4 bits per absent pair.
  uint64_t S = 0;
  const uint32_t row_align = 64 - 4 * ((nq + 1) / 2);
  // Initial quad row.
  {
    uint32_t c_q = 0;
    for (uint32_t q = 0; q < nq; q += 2) {
      uint32_t v = vlc.fetch();
      uint32_t t0 = T.vlc0[c_q + (v & 0x7F)];
      if (c_q == 0) {
        run -= 2;
        t0 = run == -1 ? t0 : 0;
        if (run < 0) run = mel.get_run();
      }
      c_q = ((t0 & 0x10) << 3) | ((t0 & 0xE0) << 2);
      // The pair's bits (at most 30) are read from the 32-bit window v with
      // 32-bit shifts; the reader advances once, by their sum, at the end.
      const uint32_t l0 = t0 & 7;
      v >>= l0;
      const bool hasB = q + 1 < nq;
      uint32_t t1 = T.vlc0[c_q + (v & 0x7F)];
      if (c_q == 0 && hasB) {
        run -= 2;
        t1 = run == -1 ? t1 : 0;
        if (run < 0) run = mel.get_run();
      }
      if (!hasB) t1 = 0;
      c_q = ((t1 & 0x10) << 3) | ((t1 & 0xE0) << 2);
      const uint32_t l1 = t1 & 7;
      v >>= l1;
      uint32_t mode = ((t0 & 8) << 3) | ((t1 & 8) << 4);
      if (mode == 0xC0) {
        run -= 2;
        if (run == -1) mode += 0x40;
        if (run < 0) run = mel.get_run();
      }
      uint32_t ue = T.uvlc0[mode + (v & 0x3F)];
      const uint32_t lp = ue & 7;
      v >>= lp;
      ue >>= 3;
      uint32_t len = ue & 0xF;
      uint32_t tmp = v & ((1u << len) - 1);
      vlc.advance(l0 + l1 + lp + len);
      ue >>= 4;
      len = ue & 7;
      ue >>= 3;
      put(q, t0 | ((1 + (ue & 7) + (tmp & ~(0xFFu << len))) << 16), t1 | ((1 + (ue >> 3) + (tmp >> len)) << 16));
      if (REG) S = push_nibble(S, pair_nibble(t0, t1));
    }
    if (REG) S >>= row_align;
    flush();
    row_done(1u);
  }
  // Other quad rows: context from the row above (quads q, q+1, q+2).
  for (uint32_t y = 2; y < h; y += 2) {
    const uint32_t* prev = row;
    row += qs;
    uint32_t c_q = 0;
    // REG: Qc = (S | S >> 1) >> (4k + 1) for pair k (bits 0 and 2: Q[4k+1],
    // Q[4k+3]); up7 = Q[4k-1] at bit 7 (Q[-1] = S[0]).
    uint64_t Qc = 0;
    uint32_t up7 = 0;
    uint32_t pq0 = 0, pq1 = 0;
    if (REG) {
      Qc = (S | (S >> 1)) >> 1;
      up7 = ((uint32_t)S & 1u) << 7;
      S = 0;
    } else {
      pq0 = prev[0] & 0xFFFF;
      pq1 = nq > 1 ? prev[1] & 0xFFFF : 0;
    }
    for (uint32_t q = 0; q < nq; q += 2) {
      uint32_t pq2 = 0, pq3 = 0, a1 = 0;
      if (REG) {
        const uint32_t qc = (uint32_t)Qc;
        c_q |= up7 | ((qc & 1u) << 9);  // quad q
        a1 = (qc & 5u) << 7;             // quad q + 1
        up7 = (qc & 4u) << 5;
        Qc >>= 4;
      } else {
        pq2 = q + 2 < nq ? prev[q + 2] & 0xFFFF : 0;
        pq3 = q + 3 < nq ? prev[q + 3] & 0xFFFF : 0;
        c_q |= (pq0 & 0xA0) << 2;
        c_q |= (pq1 & 0x20) << 4;
      }
      uint32_t v = vlc.fetch();
      uint32_t t0 = T.vlc1[c_q + (v & 0x7F)];
      if (c_q == 0) {
        run -= 2;
        t0 = run == -1 ? t0 : 0;
        if (run < 0) run = mel.get_run();
      }
      c_q = left_ctx(t0);
      if (REG) c_q |= a1;
      else c_q |= (pq0 & 0x80) | ((pq1 & 0xA0) << 2) | ((pq2 & 0x20) << 4);
      const uint32_t l0 = t0 & 7;
      v >>= l0;
      const bool hasB = q + 1 < nq;
      uint32_t t1 = T.vlc1[c_q + (v & 0x7F)];
      if (c_q == 0 && hasB) {
        run -= 2;
        t1 = run == -1 ? t1 : 0;
        if (run < 0) run = mel.get_run();
      }
      if (!hasB) t1 = 0;
      c_q = left_ctx(t1);
      if (!REG) c_q |= pq1 & 0x80;
      const uint32_t l1 = t1 & 7;
      v >>= l1;
      uint32_t mode = ((t0 & 8) << 3) | ((t1 & 8) << 4);
      uint32_t ue = T.uvlc1[mode + (v & 0x3F)];
      const uint32_t lp = ue & 7;
      v >>= lp;
      ue >>= 3;
      uint32_t len = ue & 0xF;
      uint32_t tmp = v & ((1u << len) - 1);
      vlc.advance(l0 + l1 + lp + len);
      ue >>= 4;
      len = ue & 7;
      ue >>= 3;
      put(q, t0 | (((ue & 7) + (tmp & ~(0xFFu << len))) << 16), t1 | (((ue >> 3) + (tmp >> len)) << 16));
      if (REG) {
        S = push_nibble(S, pair_nibble(t0, t1));
      } else {
        pq0 = pq2;
        pq1 = pq3;
      }
    }
    if (REG) S >>= row_align;
    flush();
    row_done(y / 2 + 1);
  }
  return true;
}

}  // namespace

// Pass 1: one lane per code block runs the VLC chain, `lanes` (a power of
// two up to 32) code blocks per warp: warp k takes blocks k * lanes ..
// k * lanes + lanes - 1 on its first lanes.  The lanes of a warp follow
// different blocks' branches, and a warp pays for every path any of its
// lanes takes at each step; fewer blocks per warp make each chain step
// shorter, which a plan with few blocks (one tile) wants, while a large
// batch fills the SMs with 32 blocks per warp.  OUTLINE: the bit readers'
// rare refill paths as out-of-line calls (MelT, VlcT).
template <bool OUTLINE>
__global__ void __launch_bounds__(kHtThreads) ht_vlc_kernel(const HtJob* __restrict__ jobs, uint32_t njobs,
                                                            const uint8_t* __restrict__ arena,
                                                            uint32_t* __restrict__ symbols, uint32_t lanes) {
  __shared__ SmemTables T;
  __shared__ uint2 stage[16 * kHtThreads];  // per lane: the pairs of one row of a 64-wide block
  {
    const uint32_t* src = reinterpret_cast<const uint32_t*>(&g_ht_tables);
    uint32_t* d = reinterpret_cast<uint32_t*>(&T);
    for (uint32_t i = threadIdx.x; i < sizeof(SmemTables) / 4; i += blockDim.x) d[i] = src[i];
  }
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31;
  if (lane >= lanes) return;
  const uint32_t j = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * lanes + lane;
  if (j >= njobs) return;
  const HtJob job = jobs[j];
  if (job.passes == 0) return;
  uint32_t* sym = symbols + job.sym;
  const bool ok = job.w <= 64 ? decode_vlc<true, OUTLINE>(job, arena + job.src, sym, T, stage, blockDim.x, threadIdx.x)
                              : decode_vlc<false, OUTLINE>(job, arena + job.src, sym, T, stage, blockDim.x, threadIdx.x);
  if (!ok) sym[0] = kSymFailed;
}

namespace {

constexpr int kMsWarps = 8;  // warps (code blocks in flight) per CTA of the MagSgn pass

// 0x80 in every byte of x that is 0xFF (exact in each byte).
__device__ __forceinline__ uint32_t ff_bytes(uint32_t x) {
  const uint32_t y = ~x;
  return ~(((y & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | y | 0x7F7F7F7Fu);
}

// Unstuffs the forward MagSgn byte stream [0, len) into a bit array W
// (bit k of the stream = bit k%32 of W[k/32]): each byte contributes 8 bits,
// or 7 after a 0xFF byte, ORed in at its offset exactly as the reference's
// ForwardBitReader accumulates it (ht_block_decode.rs:888-930).  Bits past
// the end, up to W[nwords - 1], read as ones (the reader pads with 0xFF).
//
// A group of G lanes (the warp, or each half-warp with its own stream; then
// both run the longer one's steps) takes 8 G bytes per step, eight aligned
// bytes per lane.  A lane removes the stuffed bits from its own bytes
// (events, below), so that its bits are one string of n bits at bit P of the
// stream, and writes the words of W whose first bit lies in its string, their
// ends completed from the next lane's string by a shuffle: no word is written
// twice but the first of a step, which lane 0 completes.  The pass issues
// instructions in 69 % of its cycles and waits for its loads in most others:
// eight bytes per lane instead of four, one 64-bit load instead of two
// unaligned words, plain stores instead of shared-memory atomics into a zeroed
// array, and fewer operations per sample in the row loops below took it from
// 2.70 to 2.17 ms on the uneven batch of 1,024 tiles and from 0.50 to 0.41 ms
// on 256 tiles of 512 x 512.
template <int G>
__device__ __forceinline__ void unstuff_magsgn(const uint8_t* src, uint32_t len, uint32_t* W, uint32_t nwords) {
  const uint32_t lane = threadIdx.x & 31, gl = lane & (G - 1), gsh = lane & (32 - G);
  const uint32_t lt = (1u << gl) - 1;
  const uint32_t lead = (uint32_t)((uintptr_t)src & 7);
  const uint8_t* const base = src - lead;
  const uint32_t span = lead + len;  // the stream is bytes [lead, span) from base
  uint32_t steps = len ? (span + 8 * G - 1) / (8 * G) : 0;
  if (G < 32) steps = max(steps, __shfl_xor_sync(0xFFFFFFFFu, steps, 16));
  // The lane's eight bytes at offset o, zero outside the stream: one aligned
  // load when all are in it, otherwise the aligned words that hold a byte of
  // it (so they lie inside its allocation).
  auto load = [&](uint32_t o) -> uint2 {
    uint2 x = make_uint2(0, 0);
    if (o >= lead && o + 8 <= span) {
      x = __ldg(reinterpret_cast<const uint2*>(base + o));
    } else if (o < span && len) {
      const uint32_t first = o < lead ? lead - o : 0, last = min(span - o, 8u);
      const uint32_t* wp = reinterpret_cast<const uint32_t*>(base + o);
      if (first < 4) x.x = __ldg(wp);
      if (last > 4) x.y = __ldg(wp + 1);
      uint64_t v = ((uint64_t)x.y << 32) | x.x;
      v = (v >> (8 * first)) << (8 * first);
      if (last < 8) v &= (1ull << (8 * last)) - 1;
      x = make_uint2((uint32_t)v, (uint32_t)(v >> 32));
    }
    return x;
  };
  uint32_t P = 0;     // stream bits before the step
  uint32_t info = 0;  // of the byte before the step: bit 0 it is 0xFF, bit 1 its stuffed top bit is set
  uint32_t end = 0;   // the lane's last string's end
  uint2 x = load(8 * gl);
  for (uint32_t k = 0; k < steps; ++k) {
    const uint32_t o = 8 * (k * G + gl);
    const uint2 nx = load(o + 8 * G);
    const uint32_t first = o < lead ? lead - o : 0;
    const uint32_t bytes = o < span ? min(span - o, 8u) - min(first, 8u) : 0u;
    uint64_t v = ((uint64_t)x.y << 32) | x.x;
    v >>= 8 * first;  // (first is not zero only on the lane that holds the stream's first byte)
    uint32_t n = 8 * bytes, at = P + 8 * (o - min(o, 8 * G * k + (k ? 0u : lead)));
    const uint32_t m0 = ff_bytes(x.x), m1 = ff_bytes(x.y);
    if (__any_sync(0xFFFFFFFFu, (m0 | m1 | info) != 0)) {
      // Positions: byte j of the stream is short when byte j - 1 is 0xFF, so
      // a lane's string starts one bit earlier per 0xFF byte among those
      // before the last byte before it.
      const uint32_t count = (uint32_t)(__popc(m0) + __popc(m1));
      uint32_t before = info & 1u;
      for (uint32_t t = 1;; ++t) {
        const uint32_t has = __ballot_sync(0xFFFFFFFFu, count >= t);
        if (has == 0) break;
        before += (uint32_t)__popc((has >> gsh) & lt);
      }
      const uint32_t mine = (m1 >> 31) | ((m1 >> 22) & (x.y >> 30) & 2u);
      uint32_t prev = __shfl_up_sync(0xFFFFFFFFu, mine, 1, G);
      if (gl == 0) prev = info;
      info = __shfl_sync(0xFFFFFFFFu, mine, G - 1, G);
      at -= before - (prev & 1u);
      // Events: a flag at each short byte of the lane's string.  Every bit
      // above a short byte moves down by one; the byte's own top bit stays
      // and is ORed with what arrives there.
      uint64_t ev = (((uint64_t)m1 << 32) | m0) >> (8 * first);
      ev = (ev << 8) | (prev & 1u ? 0x80u : 0u);
      if (bytes < 8) ev &= (1ull << (8 * bytes)) - 1;
      uint32_t drops = 0;
      while (ev) {
        const uint32_t top = (uint32_t)__ffsll((long long)ev) - drops;  // the short byte's end
        ev &= ev - 1;
        ++drops;
        if (top < 64) v = (v & ((1ull << top) - 1)) | ((v >> top) << (top - 1));
      }
      n -= drops;
      v |= (prev >> 1) & 1u;
    }
    uint32_t next = __shfl_down_sync(0xFFFFFFFFu, (uint32_t)v, 1, G);
    if (gl == G - 1) next = 0;
    __syncwarp();  // the previous step's words, before lane 0 completes the last of them
    if (bytes) {
      const uint32_t a = (0u - at) & 31u;  // bits of the string before its first own word
      uint32_t* wp = W + ((at + 31) >> 5);
      const uint64_t u = v >> a;
      if (gl == 0 && a) wp[-1] |= (uint32_t)v << (32 - a);
      if (a < n) wp[0] = (uint32_t)u | __funnelshift_lc(0u, next, n - a);
      if (a + 32 < n) wp[1] = (uint32_t)(u >> 32) | __funnelshift_lc(0u, next, n - a - 32);
      end = at + n;
    }
    P = __shfl_sync(0xFFFFFFFFu, at + n, G - 1, G);
    x = nx;
  }
  const uint32_t bits = __shfl_sync(0xFFFFFFFFu, end, len ? ((span - 1) >> 3) & (G - 1) : 0, G);
  __syncwarp();
  // Padding: every bit from there on is one.
  if (gl == 0 && (bits & 31) && (bits >> 5) < nwords) W[bits >> 5] |= 0xFFFFFFFFu << (bits & 31);
  for (uint32_t wi = ((bits + 31) >> 5) + gl; wi < nwords; wi += G) W[wi] = 0xFFFFFFFFu;
  __syncwarp();
}

__device__ __forceinline__ uint32_t bits_at(const uint32_t* W, uint32_t nwords, uint32_t off) {
  uint32_t wi = off >> 5, sh = off & 31;
  uint32_t lo = wi < nwords ? W[wi] : 0xFFFFFFFFu;
  uint32_t hi = wi + 1 < nwords ? W[wi + 1] : 0xFFFFFFFFu;
  return __funnelshift_r(lo, hi, sh);
}

// Per-quad magnitude/sign arithmetic of the row loops below, with the quad's
// four samples as the four bytes of one word (byte i = sample i, the order
// of the quad's bits in the stream: (0,0), (0,1), (1,0), (1,1) by column
// pairs).  A bit count m_n is at most 31 and a quad's total at most 124, so
// bytewise sums never carry and a multiply by 0x01010101 forms every
// sample's inclusive prefix inside the quad at once.

// Byte i = bit i of the nibble x.
__device__ __forceinline__ uint32_t spread4(uint32_t x) { return (x * 0x00204081u) & 0x01010101u; }

struct QuadBits {
  uint32_t m;    // m_n per sample: U - e_k when significant, else 0
  uint32_t incl; // per sample, the bits up to its own end in the quad
};

// U is the quad's u_q (plus the exponent bound kappa after the first row);
// U > mmsb + 2 marks an invalid stream, which the caller flags and whose
// block comes out as zeros, so clamping U to 31 here (the bytes then cannot
// carry) changes no valid result.  right: the quad's right column lies in the
// block; where it does not (the last quad of an odd width) a damaged stream
// can make its samples significant, and they take no bits of the stream.
__device__ __forceinline__ QuadBits quad_bits(uint32_t inf, uint32_t U, bool right) {
  const uint32_t sig = spread4((inf >> 4) & 0xFu), k = spread4(inf >> 12);
  const uint32_t m = (min(U, 31u) * 0x01010101u - k) & (sig * 0xFFu) & (right ? ~0u : 0xFFFFu);
  return QuadBits{m, m * 0x01010101u};
}

// Inclusive prefix sum over the calling group of G lanes (the warp or a
// half-warp): the shuffle's own in-range predicate guards each addition.
template <int G>
__device__ __forceinline__ uint32_t inclusive_scan(uint32_t x) {
#ifdef __CUDA_ARCH__
#pragma unroll
  for (int d = 1; d < G; d <<= 1)
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .u32 t;\n\t"
        "shfl.sync.up.b32 t|p, %0, %1, %2, 0xffffffff;\n\t"
        "@p add.u32 %0, %0, t;\n\t}"
        : "+r"(x)
        : "r"(d), "r"((32 - G) << 8));
#else
  const uint32_t gl = threadIdx.x & (G - 1);
  for (int d = 1; d < G; d <<= 1) {
    const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, x, d, G);
    if (gl >= (uint32_t)d) x += v;
  }
#endif
  return x;
}

// Sample i's coefficient from its bits msv (sign first, then the magnitude
// bits below the implied ones), bit count m (low five bits), known-1 bit e1
// and significance: decode_mag_sgn_sample_with_vn's v_n (ht_block_decode.rs:1010-1032)
// gives the sign-magnitude word sign << 31 | (v + 2) << (p - 1) in 32-bit
// arithmetic (whose top bit, in the largest valid magnitudes, the shift can
// set as well); RAW returns that word, otherwise coefficient_to_i32
// (:225-234) of it: (word & 0x7FFFFFFF) >> (31 - nbp), negated when the top
// bit is set, computed as (word << 1) >> rs with rs = 32 - nbp (1 when
// nbp >= 31; the shift clamps at 32).  E receives the position of v's top bit
// (one less than its bit length; 0 when insignificant), the exponent the row
// below needs.
template <bool RAW>
__device__ __forceinline__ int32_t sample_value(uint32_t msv, uint32_t m, uint32_t e1, bool sig, uint32_t p,
                                                uint32_t rs, uint32_t& E) {
  const uint32_t mask = __funnelshift_l(0xFFFFFFFFu, 0u, m);
  const uint32_t v = (msv & mask) | __funnelshift_l(0u, e1, m) | 1u;
  E = sig ? 31u - (uint32_t)__clz(v) : 0u;
  const uint32_t word = (msv << 31) | ((v + 2) << (p - 1));
  if (RAW) return sig ? (int32_t)word : 0;
  const int32_t mag = (int32_t)__funnelshift_rc(word << 1, 0u, rs);
  return sig ? ((int32_t)word < 0 ? -mag : mag) : 0;
}

// The four samples of a quad whose stream bits start at `off`: one clamped
// three-word window read serves all four when the quad holds fewer than 64
// bits, each sample's bits shifted out after it; otherwise each sample reads
// its own 32 bits.
template <bool RAW>
__device__ __forceinline__ void quad_samples(const uint32_t* W, uint32_t ms_words, uint32_t lim, uint32_t off,
                                             uint32_t inf, const QuadBits& qb, uint32_t p, uint32_t rs,
                                             int32_t val[4], uint32_t E[4]) {
  uint32_t lo, hi;
  {
    const uint32_t o = min(off, lim), wi = o >> 5;
    const uint32_t a0 = W[wi], a1 = W[wi + 1], a2 = W[wi + 2];
    lo = __funnelshift_r(a0, a1, o);
    hi = __funnelshift_r(a1, a2, o);
  }
  uint32_t msv[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    msv[i] = lo;
    // (Shift counts are taken modulo 32: the sample's byte of m.)
    lo = __funnelshift_r(lo, hi, qb.m >> (8 * i));
    hi = __funnelshift_r(hi, 0u, qb.m >> (8 * i));
  }
  if ((qb.incl >> 24) >= 64) {
#pragma unroll
    for (int i = 0; i < 4; ++i) msv[i] = bits_at(W, ms_words, off + (((qb.incl - qb.m) >> (8 * i)) & 0xFFu));
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
    val[i] = sample_value<RAW>(msv[i], qb.m >> (8 * i), (inf >> (8 + i)) & 1u, (inf >> (4 + i)) & 1u, p, rs, E[i]);
}


// The magnitude/sign rows of one block (decode_magnitude_sign_phase,
// ht_block_decode.rs:1435-1561) for the calling warp.  Per quad row the lanes
// take one quad each; a warp prefix scan of the per-quad bit counts gives each
// lane its bit offset in the unstuffed stream W, and the lane reads its bits
// through one 64-bit window.  The exponent bound kappa needs the bit lengths
// of v_n of the four samples above the quad: with NARROW (blocks at most 64
// wide, one quad per lane per row) they stay in registers and come from the
// neighbouring lanes by shuffles, otherwise they are kept per column in
// shared memory (Ebase, two rows of `cols` bytes).  Returns true (on every
// lane) when the stream is invalid.  ODD: the width may be odd (quad_bits); the
// usual even widths keep a loop without that test, which took 1 % of the
// uneven batch's pass (2.175 -> 2.195 ms).
// Rows are taken as they are: the two-pass form decodes symbols a kernel
// earlier.
struct NoRowWait {
  static constexpr bool kLive = false;
  __device__ bool operator()(uint32_t) const { return true; }
};
template <bool NARROW, bool RAW, bool ODD, typename RowWait = NoRowWait>
__device__ bool magsgn_rows(const HtJob& job, const uint32_t* W, uint32_t ms_words, uint8_t* Ebase, uint32_t cols,
                            const uint32_t* sym, int32_t* __restrict__ dst, RowWait row_ready = RowWait()) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t w = job.w, h = job.h, stride = job.stride;
  const uint32_t mmsb = job.mmsb, p = 30 - mmsb, mmsbp2 = mmsb + 2, nbp = job.nbp;
  const uint32_t rs = nbp >= 31 ? 1u : 32u - nbp;
  // Window reads start at most at bit `lim`, so that words wi .. wi + 2 lie
  // in the array (it holds at least 5 words).  The array ends with at least
  // 64 bits of ones past the stream (its padding), and `lim` lies beyond
  // those bits' start, so a clamped read returns the ones an unclamped one
  // would have seen past the end of the stream.
  const uint32_t lim = 32 * (ms_words - 3);
  const bool pairs = ((job.dst | stride) & 1) == 0;  // 8-byte aligned sample pairs
  const uint32_t nq = (w + 1) / 2, qs = sym_row_stride(w);
  uint8_t* Eprev = Ebase;  // wide blocks: top bit positions of v_n per column + 1, row above
  uint8_t* Ecur = Ebase + cols;
  if (!NARROW) {
    for (uint32_t c = lane; c < cols; c += 32) Eprev[c] = 0;
    __syncwarp();
  }
  uint32_t e_left = 0, e_right = 0;  // NARROW: bottom-row top bit positions of this lane's quad
  uint32_t rowbase = 0;
  bool bad = false;
  // Running pointers: sample row y of the block and quad row r of its symbols.
  int32_t* row0 = dst;
  const uint32_t* srow = sym;
  for (uint32_t y = 0; y < h; y += 2, row0 += 2 * (size_t)stride, srow += qs) {
    // The fused form waits for the quad row's symbols (warp-uniform result;
    // false: the chain failed or the wait ran out, and the block is invalid).
    if (!row_ready(y >> 1)) {
      bad = true;
      break;
    }
    const bool initial = y == 0, second = y + 1 < h;
    // NARROW rows have at most 32 quads: one pass, known at compile time.
    const uint32_t c0_end = NARROW ? 1u : nq;
    for (uint32_t c0 = 0; c0 < c0_end; c0 += 32) {
      const uint32_t q = c0 + lane;
      const bool active = q < nq;
      // Symbols written by the same CTA's chain lane: in shared memory, or
      // (wide blocks) read past L1.
      const uint32_t s = active ? (!RowWait::kLive ? srow[q]
                                   : NARROW        ? *const_cast<const volatile uint32_t*>(srow + q)
                                                   : __ldcg(srow + q))
                                : 0;
      const uint32_t inf = s & 0xFFFF;
      uint32_t U = s >> 16;
      if (!initial) {
        uint32_t e;
        if (NARROW) {
          // Columns 2q-1 and 2q+2 belong to the neighbouring lanes' quads
          // (lanes past nq hold zeros; the first and last lane's shuffles
          // give them their own samples, which the maximum has anyway).
          const uint32_t l = __shfl_up_sync(0xFFFFFFFFu, e_right, 1);
          const uint32_t rr = __shfl_down_sync(0xFFFFFFFFu, e_left, 1);
          e = max(max(l, e_left), max(e_right, rr));
        } else {
          // Columns 2q-1 .. 2q+2 of the row above live at Eprev[col + 1]
          // (index <= 2*nq + 1 <= w + 2 < max_w + 4 for an active lane).
          e = active ? max(max((uint32_t)Eprev[2 * q], (uint32_t)Eprev[2 * q + 1]),
                           max((uint32_t)Eprev[2 * q + 2], (uint32_t)Eprev[2 * q + 3]))
                     : 0;
        }
        // kappa: max(bit length, 2) - 1 of the samples above when at least
        // two of the quad's are significant, else 1.
        uint32_t gamma = inf & 0xF0;
        gamma &= gamma - 0x10;
        U += gamma != 0 ? max(e, 1u) : 1u;
      }
      // (A lane without a quad holds U of 0 or 1 and no significant sample.)
      bad |= U > mmsbp2;
      const QuadBits qb = quad_bits(inf, U, !ODD || 2 * q + 1 < w);
      const uint32_t tot = qb.incl >> 24;
      const uint32_t inc = inclusive_scan<32>(tot);
      const uint32_t off = rowbase + inc - tot;
      rowbase += __shfl_sync(0xFFFFFFFFu, inc, 31);
      int32_t val[4];
      uint32_t E[4];
      quad_samples<RAW>(W, ms_words, lim, off, inf, qb, p, rs, val, E);
      if (active) {
        const uint32_t x = 2 * q;
        int32_t* p0 = row0 + x;
        if (pairs && x + 1 < w) {
          *reinterpret_cast<int2*>(p0) = make_int2(val[0], val[2]);
          if (second) *reinterpret_cast<int2*>(p0 + stride) = make_int2(val[1], val[3]);
        } else {
          p0[0] = val[0];
          if (second) p0[stride] = val[1];
          if (x + 1 < w) {
            p0[1] = val[2];
            if (second) p0[stride + 1] = val[3];
          }
        }
        if (!NARROW) {
          // Bottom-row exponents of this quad for the next quad row.
          Ecur[x + 1] = (uint8_t)E[1];
          Ecur[x + 2] = x + 1 < w ? (uint8_t)E[3] : 0;
        }
      }
      if (NARROW) {
        e_left = active ? E[1] : 0;
        e_right = active && 2 * q + 1 < w ? E[3] : 0;
      }
    }
    if (!NARROW) {
      __syncwarp();
      // Columns outside [0, w) stay zero in both buffers.
      if (lane == 0) {
        Ecur[0] = 0;
        Ecur[w + 1] = 0;
        Ecur[w + 2] = 0;
      }
      __syncwarp();
      uint8_t* t = Eprev;
      Eprev = Ecur;
      Ecur = t;
    }
  }
  return __any_sync(0xFFFFFFFFu, bad);
}
}  // namespace

// Narrow blocks (at most 32 wide: 16 quads a row) would leave half of a
// warp idle, so a warp takes two of them, one per half-warp (lanes 0-15 and
// 16-31).  The function below is magsgn_rows for that case (and unstuff_magsgn
// has its half-warp form): every shuffle, ballot and scan runs on all 32 lanes with the
// half-warp as its segment, and both halves run the longer block's loop
// trip counts (a half past its own work idles), so no warp-synchronous
// operation sits in a branch that one half skips.

// magsgn_rows<true, false, ODD> for the calling half-warp's block (live) over
// hmax rows, the taller of the two blocks' heights.  Returns true on the
// half's lanes when its stream is invalid.
template <bool ODD>
__device__ bool magsgn_rows_half(const HtJob& job, bool live, const uint32_t* W, uint32_t ms_words, uint32_t hmax,
                                 const uint32_t* __restrict__ sym, int32_t* __restrict__ dst) {
  const uint32_t lane = threadIdx.x & 31, gl = lane & 15, gsh = lane & 16;
  const uint32_t w = live ? job.w : 0, h = live ? job.h : 0, stride = job.stride;
  const uint32_t mmsb = job.mmsb, p = 30 - mmsb, mmsbp2 = mmsb + 2, nbp = job.nbp;
  const uint32_t rs = nbp >= 31 ? 1u : 32u - nbp;
  // As in magsgn_rows: clamped window reads stay in the half's words.
  const uint32_t lim = live ? 32 * (ms_words - 3) : 0;
  const bool pairs = ((job.dst | stride) & 1) == 0;
  const uint32_t nq = (w + 1) / 2, qs = sym_row_stride(w);
  uint32_t e_left = 0, e_right = 0, rowbase = 0;
  bool bad = false;
  // Per lane, invariant over the rows: its quad column, whether it holds a
  // quad, whether the quad has a right column and whether the pair goes out
  // in one 8-byte store; running pointers to its samples and its symbols.
  const uint32_t q = gl;
  const bool lane_q = q < nq, has_right = 2 * q + 1 < w, pair_store = pairs && has_right;
  int32_t* lp = dst + 2 * q;
  const uint32_t* sp = sym + q;
  for (uint32_t y = 0; y < hmax; y += 2, lp += 2 * (size_t)stride, sp += qs) {
    const bool initial = y == 0, second = y + 1 < h;
    const bool active = y < h && lane_q;
    const uint32_t s = active ? *sp : 0;
    const uint32_t inf = s & 0xFFFF;
    uint32_t U = s >> 16;
    if (!initial) {
      const uint32_t l = __shfl_up_sync(0xFFFFFFFFu, e_right, 1, 16);
      const uint32_t rr = __shfl_down_sync(0xFFFFFFFFu, e_left, 1, 16);
      const uint32_t e = max(max(l, e_left), max(e_right, rr));
      uint32_t gamma = inf & 0xF0;
      gamma &= gamma - 0x10;
      U += gamma != 0 ? max(e, 1u) : 1u;
    }
    bad |= U > mmsbp2;
    const QuadBits qb = quad_bits(inf, U, !ODD || has_right);
    const uint32_t tot = qb.incl >> 24;
    const uint32_t inc = inclusive_scan<16>(tot);
    const uint32_t off = rowbase + inc - tot;
    rowbase += __shfl_sync(0xFFFFFFFFu, inc, 15, 16);
    int32_t val[4];
    uint32_t E[4];
    quad_samples<false>(W, ms_words, lim, off, inf, qb, p, rs, val, E);
    if (active) {
      if (pair_store) {
        *reinterpret_cast<int2*>(lp) = make_int2(val[0], val[2]);
        if (second) *reinterpret_cast<int2*>(lp + stride) = make_int2(val[1], val[3]);
      } else {
        lp[0] = val[0];
        if (second) lp[stride] = val[1];
        if (has_right) {
          lp[1] = val[2];
          if (second) lp[stride + 1] = val[3];
        }
      }
    }
    e_left = active ? E[1] : 0;
    e_right = active && has_right ? E[3] : 0;
  }
  return ((__ballot_sync(0xFFFFFFFFu, bad) >> gsh) & 0xFFFFu) != 0;
}

// Pass 2: one warp per code block decodes magnitudes and signs
// (decode_magnitude_sign_phase, ht_block_decode.rs:1435-1561).  Per quad row
// the lanes take one quad each: the exponent bound kappa comes from the four
// samples above (bit lengths of the previous row's v_n, kept per column in
// shared memory), each lane sums its samples' m_n, a warp prefix scan turns
// the sums into bit offsets inside the unstuffed MagSgn stream, and the row
// is written with coalesced stores.
namespace {

// Magnitudes and signs of one code block by the calling warp; W and Ebase
// are the warp's shared-memory bit array and exponent rows.
template <typename RowWait = NoRowWait>
__device__ void magsgn_block(const HtJob& job, const uint8_t* __restrict__ arena,
                             const uint32_t* symbols, int32_t* __restrict__ coef,
                             uint32_t* __restrict__ tile_status, uint32_t ms_words, uint32_t cols, uint32_t* W,
                             uint8_t* Ebase, RowWait row_ready = RowWait()) {
  const uint32_t lane = threadIdx.x & 31;
  int32_t* dst = coef + job.dst;
  const uint32_t w = job.w, h = job.h, stride = job.stride;
  if (job.passes == 0) {
    for (uint32_t y = 0; y < h; ++y)
      for (uint32_t x = lane; x < w; x += 32) dst[(size_t)y * stride + x] = 0;
    return;
  }
  const uint32_t* sym = RowWait::kLive ? symbols : symbols + job.sym;  // (live: the block's own table)
  const uint8_t* src = arena + job.src;
  // The block's cleanup bytes and quad symbols are requested from HBM before
  // the first of them is loaded: the unstuffing steps and the quad rows then
  // read them from L2.
  prefetch_l2_range(src, job.lcup, lane, 32);
  uint32_t lcup = job.lcup, scup = 0;
  bool ok;
  if constexpr (RowWait::kLive) {
    // The chain is still running: its failure arrives through row_ready, and
    // the segment checks it starts with are repeated here.
    ok = lcup >= 2;
    if (ok) {
      scup = ((uint32_t)ld8(src + lcup - 1) << 4) + (ld8(src + lcup - 2) & 0x0F);
      ok = scup >= 2 && scup <= lcup && scup <= 4079;
    }
  } else {
    prefetch_l2_range(sym, (size_t)sym_row_stride(w) * ((h + 1) / 2) * 4, lane, 32);
    ok = sym[0] != kSymFailed;
    if (ok) scup = ((uint32_t)ld8(src + lcup - 1) << 4) + (ld8(src + lcup - 2) & 0x0F);
  }
  if (ok) ok = (lcup - scup + 15) / 4 + 2 <= ms_words;
  if (ok) {
    const uint32_t ms_len = lcup - scup;
    // The block's own words of the bit array (at most ms_words, checked
    // above): they are written whole and padded with ones past the stream,
    // and reads beyond them return ones, so bits past the end still read as
    // the reference's 0xFF padding.
    const uint32_t words = (ms_len + 15) / 4 + 2;
    unstuff_magsgn<32>(src, ms_len, W, words);
    // Blocks with refinement passes keep the sign-magnitude words for them.
    const bool raw = job.passes > 1;
    auto rows = [&](auto narrow, auto raw_words, auto odd) {
      return magsgn_rows<decltype(narrow)::value, decltype(raw_words)::value, decltype(odd)::value>(
          job, W, words, Ebase, cols, sym, dst, row_ready);
    };
    using T = std::true_type;
    using F = std::false_type;
    // One loop for every width where the block is rare or waits for its chain.
    const bool narrow = job.w <= 64;
    bool bad;
    if (raw) bad = narrow ? rows(T{}, T{}, T{}) : rows(F{}, T{}, T{});
    else if (RowWait::kLive || (job.w & 1)) bad = narrow ? rows(T{}, F{}, T{}) : rows(F{}, F{}, T{});
    else if constexpr (!RowWait::kLive) bad = narrow ? rows(T{}, F{}, F{}) : rows(F{}, F{}, F{});
    ok = !bad;
  }
  if (!ok) {
    __syncwarp();
    for (uint32_t y = 0; y < h; ++y)
      for (uint32_t x = lane; x < w; x += 32) dst[(size_t)y * stride + x] = 0;
    if (lane == 0) atomicOr(&tile_status[job.tile], kStatusDecode);
  }
  __syncwarp();  // the warp's shared buffers are reused by its next block
}

// Two narrow blocks, jobs[a] on lanes 0-15 and jobs[b] on lanes 16-31 (b ==
// UINT32_MAX: none), each with half of the warp's bit array (half_words
// words); both at most 32 wide with no refinement passes (the host orders
// such blocks after the others).  Same results as magsgn_block on each.
__device__ void magsgn_pair(const HtJob* __restrict__ jobs, uint32_t a, uint32_t b, const uint8_t* __restrict__ arena,
                            const uint32_t* __restrict__ symbols, int32_t* __restrict__ coef,
                            uint32_t* __restrict__ tile_status, uint32_t half_words, uint32_t* W) {
  const uint32_t lane = threadIdx.x & 31, g = lane >> 4, gl = lane & 15;
  const bool present = g == 0 || b != 0xFFFFFFFFu;
  const HtJob job = jobs[present ? (g ? b : a) : a];
  uint32_t* Wg = W + g * half_words;
  int32_t* dst = coef + job.dst;
  const uint32_t* sym = symbols + job.sym;
  const uint8_t* src = arena + job.src;
  const bool coded = present && job.passes != 0;
  bool ok = coded;
  if (ok) {
    prefetch_l2_range(src, job.lcup, gl, 16);
    prefetch_l2_range(sym, (size_t)sym_row_stride(job.w) * ((job.h + 1) / 2) * 4, gl, 16);
    ok = sym[0] != kSymFailed;
  }
  uint32_t ms_len = 0, words = 0;
  if (ok) {
    const uint32_t lcup = job.lcup;
    const uint32_t scup = ((uint32_t)ld8(src + lcup - 1) << 4) + (ld8(src + lcup - 2) & 0x0F);
    ok = (lcup - scup + 15) / 4 + 2 <= half_words;
    if (ok) {
      ms_len = lcup - scup;
      words = (ms_len + 15) / 4 + 2;
    }
  }
  unstuff_magsgn<16>(src, ms_len, Wg, words);
  const uint32_t hh = ok ? job.h : 0;
  const uint32_t hmax = max(hh, __shfl_xor_sync(0xFFFFFFFFu, hh, 16));
  const bool odd = __any_sync(0xFFFFFFFFu, job.w & 1);
  const bool bad = odd ? magsgn_rows_half<true>(job, ok, Wg, words, hmax, sym, dst)
                       : magsgn_rows_half<false>(job, ok, Wg, words, hmax, sym, dst);
  if (present && (!ok || bad)) {
    // No coded passes: zeros; an invalid stream: zeros and the tile's status.
    for (uint32_t y = 0; y < job.h; ++y)
      for (uint32_t x = gl; x < job.w; x += 16) dst[(size_t)y * job.stride + x] = 0;
    if (coded && gl == 0) atomicOr(&tile_status[job.tile], kStatusDecode);
  }
  __syncwarp();  // the warp's shared buffers are reused by its next work item
}

}  // namespace

// Pass 2: one warp per code block decodes magnitudes and signs
// (decode_magnitude_sign_phase, ht_block_decode.rs:1435-1561).  Grid form
// (queue == nullptr): warp k of CTA c takes block c * warps + k.  Queue form:
// a persistent grid whose warps take `gran` consecutive blocks at a time
// from the device work queue (an atomic counter over the job table, which is
// ordered by coded length, longest first).
//
// Work items: jobs [0, nsingle) one per warp; the narrow jobs after them
// (at most 32 wide, no refinement passes) two per warp, item nsingle + k
// taking jobs nsingle + 2k and nsingle + 2k + 1.
template <bool QUEUE>
__global__ void __launch_bounds__(kMsWarps * 32) ht_magsgn_kernel(const HtJob* __restrict__ jobs, uint32_t njobs,
                                                                  const uint8_t* __restrict__ arena,
                                                                  const uint32_t* __restrict__ symbols,
                                                                  int32_t* __restrict__ coef,
                                                                  uint32_t* __restrict__ tile_status,
                                                                  uint32_t ms_words, uint32_t max_w, uint32_t* queue,
                                                                  uint32_t gran, uint32_t nsingle) {
  extern __shared__ __align__(16) uint8_t smem[];
  const uint32_t nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cols = max_w + 4;
  uint32_t* W = reinterpret_cast<uint32_t*>(smem) + (size_t)warp * ms_words;
  uint8_t* Ebase = smem + (size_t)nw * ms_words * 4 + (size_t)warp * 2 * cols;
  const uint32_t nitems = nsingle + (njobs - nsingle + 1) / 2;
  auto item = [&](uint32_t it) {
    if (it < nsingle) {
      magsgn_block(jobs[it], arena, symbols, coef, tile_status, ms_words, cols, W, Ebase);
    } else {
      const uint32_t a = nsingle + 2 * (it - nsingle);
      magsgn_pair(jobs, a, a + 1 < njobs ? a + 1 : 0xFFFFFFFFu, arena, symbols, coef, tile_status, ms_words / 2, W);
    }
  };
  if constexpr (!QUEUE) {
    const uint32_t it = blockIdx.x * nw + warp;
    if (it < nitems) item(it);
  } else {
    for (;;) {
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(queue, gran);
      base = __shfl_sync(0xFFFFFFFFu, base, 0);
      if (base >= nitems) break;
      const uint32_t end = min(base + gran, nitems);
      for (uint32_t it = base; it < end; ++it) item(it);
    }
  }
}

// Small plans: one CTA of two warps per code block runs both cleanup passes
// at once.  Lane 0 of warp 0 runs the block's VLC chain (decode_vlc) and
// publishes each finished quad row in shared memory; warp 1 unstuffs the
// MagSgn stream meanwhile and decodes each quad row's magnitudes and signs as
// soon as its symbols are out, so the block's MagSgn work hides behind its
// own chain instead of waiting for the slowest chain of the plan (a plan of
// one tile is as long as its longest block's chain).  Waits are bounded: a
// row that does not arrive within kFusedSpinLimit polls (tens of
// milliseconds, far beyond any chain) fails the block like an invalid
// stream.
namespace {

constexpr uint32_t kFusedThreads = 64;
constexpr uint32_t kRowsFailed = 0xFFFFFFFFu;
constexpr uint32_t kFusedSpinLimit = 1u << 20;

// The chain lane's row hook: the row's symbols, then its flag.
struct FusedPublish {
  volatile uint32_t* progress;
  __device__ void operator()(uint32_t rows) const {
    __threadfence_block();
    *progress = rows;
  }
};

struct FusedRowWait {
  static constexpr bool kLive = true;
  const volatile uint32_t* progress;  // quad rows published, or kRowsFailed
  __device__ bool operator()(uint32_t row) const {
    uint32_t ready = 1;
    if ((threadIdx.x & 31) == 0) {
      uint32_t p = *progress;
      for (uint32_t it = 0; p != kRowsFailed && p <= row && it < kFusedSpinLimit; ++it) {
        __nanosleep(32);
        p = *progress;
      }
      ready = p != kRowsFailed && p > row;
    }
    ready = __shfl_sync(0xFFFFFFFFu, ready, 0);
    __threadfence_block();  // the row's symbols are read after its flag
    return ready != 0;
  }
};

}  // namespace

// The chain of a block at most 64 wide has a warp of its own here, so it is
// bound by the latency of its dependent steps, not by instructions: it looks
// up entries that hold what the next step needs in place (HtChainTables),
// reads its bits from an array that the whole warp unstuffed beforehand, has
// no branch per quad but the one for MEL runs that end, and leaves its
// symbols in shared memory: one 512 x 512 RGB tile 0.111 -> 0.092 ms for the
// kernel (512 pairs of a 64 x 64 block at about 140 ns, 170 before).  The
// same entries and selects in the 32-blocks-per-warp VLC pass were slower
// (uneven batch 0.84 -> 0.87 ms, 256 tiles 0.25 -> 0.28): its warps share
// their issue slots, and the wider tables cost it CTAs.  Making a pair's
// symbols behind the next pair's first lookup was slower too (0.097 ms).
namespace {

constexpr uint32_t kChainPairs = 512;  // quad pairs of a block of at most 4096 samples, at most 64 wide
constexpr uint32_t kChainWords = kChainPairs * 30 / 32 + 8;  // their bits (at most 30 a pair), and words read ahead

// The block's VLC bits (the backward reader's order, VlcT) into B, as many as
// the chain can take, zeros behind them; by the calling warp.  d: the cleanup
// segment.  Bit order and overlaps as in unstuff_magsgn; a byte is short here
// when its low seven bits are all ones and the byte before it is above 0x8F.
__device__ void unstuff_vlc(const uint8_t* d, uint32_t lcup, uint32_t scup, uint32_t* B) {
  const uint32_t lane = threadIdx.x & 31;
  for (uint32_t i = lane; i < kChainWords; i += 32) B[i] = 0;
  __syncwarp();
  const uint32_t b0 = ld8(d + lcup - 2);
  uint32_t P = 4 - (((b0 >> 4) & 7) == 7 ? 1 : 0);  // bits before the step
  if (lane == 0) atomicOr(&B[0], b0 >> 4);
  uint32_t info = (b0 | 0x0F) > 0x8F ? 1u : 0u;  // bit 0: the byte before the step is above 0x8F
  // As many bytes as hold the chain's bits at seven bits a byte.
  const uint32_t n = min(scup - 2, 5 * kChainWords);
  static_assert(7 * 5 * kChainWords >= 32 * (kChainWords - 4), "seven bits a byte cover what the chain takes");
  for (uint32_t base = 0; base < n; base += 128) {
    // The lane's four bytes, the first one lowest.
    const uint32_t j = base + 4 * lane;
    const uint8_t* top = d + lcup - 3 - j;  // (formed only where j < n)
    uint32_t x = 0, bytes = 0;
    if (j + 4 <= n) {
      const uintptr_t addr = (uintptr_t)(top - 3);
      const uint32_t* wp = reinterpret_cast<const uint32_t*>(addr & ~(uintptr_t)3);
      const uint32_t sh = (uint32_t)(addr & 3);
      x = __byte_perm(__funnelshift_r(__ldg(wp), sh ? __ldg(wp + 1) : 0u, 8 * sh), 0, 0x0123);
      bytes = 4;
    } else if (j < n) {
      bytes = n - j;
      x = ld8(top);
      if (bytes > 1) x |= (uint32_t)ld8(top - 1) << 8;
      if (bytes > 2) x |= (uint32_t)ld8(top - 2) << 16;
    }
    const uint32_t low = x & 0x7F7F7F7Fu;
    const uint32_t ones = (low + 0x01010101u) & 0x80808080u;       // low seven bits all ones
    const uint32_t big = (low + 0x70707070u) & x & 0x80808080u;    // above 0x8F
    uint32_t prev = __shfl_up_sync(0xFFFFFFFFu, big >> 31, 1);
    if (lane == 0) prev = info;
    info = __shfl_sync(0xFFFFFFFFu, big >> 31, 31);
    uint32_t ev = ones & ((big << 8) | (prev << 7));  // short bytes
    uint32_t at = P + 8 * (j - base), bits = 8 * bytes;
    if (__any_sync(0xFFFFFFFFu, ev != 0)) {
      const uint32_t count = (uint32_t)__popc(ev);
      uint32_t before = 0, total = 0;
      for (uint32_t t = 1;; ++t) {
        const uint32_t has = __ballot_sync(0xFFFFFFFFu, count >= t);
        if (has == 0) break;
        before += (uint32_t)__popc(has & ((1u << lane) - 1));
        total += (uint32_t)__popc(has);
      }
      at -= before;
      P -= total;
      uint64_t v = x;
      for (uint32_t drops = 0; ev; ev &= ev - 1, ++drops) {
        const uint32_t end = (uint32_t)__ffs((int)ev) - drops;  // the short byte's end
        v = (v & ((1ull << end) - 1)) | ((v >> end) << (end - 1));
      }
      x = (uint32_t)v;
    }
    P += 8 * min(n - base, 128u);
    const uint32_t wi = at >> 5, sh = at & 31;
    if (bits && wi + 1 < kChainWords) {
      atomicOr(&B[wi], x << sh);
      if (sh) atomicOr(&B[wi + 1], x >> (32 - sh));
    }
  }
  __syncwarp();
}

// decode_vlc for a lane with a warp of its own: REG blocks, VLC bits from B,
// symbols into `sym` (shared memory), row_done as there.
template <bool OUTLINE, typename RowHook>
__device__ __forceinline__ void chain_vlc(const HtJob& job, const uint8_t* src, uint32_t scup, const HtChainTables& T,
                                          const uint32_t* B, uint32_t* sym, RowHook row_done) {
  const uint32_t nq = (job.w + 1u) / 2, qs = sym_row_stride(job.w), h = job.h;
  MelT<OUTLINE> mel;
  mel.init(src, job.lcup, scup);
  int run = mel.get_run();
  // The bit window: bit `pos` (< 32) of w0 on; w2 is loaded a word ahead.
  uint32_t w0 = B[0], w1 = B[1], w2 = B[2], pos = 0, next = 3;
  auto advance = [&](uint32_t n) {
    pos += n & 31u;
    const bool over = pos >= 32;
    w0 = over ? w1 : w0;
    w1 = over ? w2 : w1;
    if (over) w2 = B[min(next, kChainWords - 1)];
    next += over ? 1 : 0;
    pos &= 31u;
  };
  // A quad's entry with its MEL event when its context is zero.
  auto event = [&](bool zero, uint32_t t) -> uint32_t {
    if (zero) {
      run -= 2;
      if (run != -1) t = 0;
      if (run < 0) run = mel.get_run();
    }
    return t;
  };
  uint32_t* row = sym;
  uint64_t S = 0;
  const uint32_t row_align = 64 - 4 * ((nq + 1) / 2);
  // A pair's symbols from its entries and the window behind its codewords:
  // the packed entries with the u values above them.
  auto symbols = [&](uint32_t q, uint32_t v, uint32_t t0, uint32_t t1, uint32_t e, uint32_t base) {
    const uint32_t x = __funnelshift_r(v, 0u, e), y = __funnelshift_r(x, 0u, e >> 10);
    const uint32_t u0 = base + ((e >> 26) & 7u) + (x & (e >> 16) & 31u), u1 = base + (e >> 29) + (y & (e >> 21) & 31u);
    *reinterpret_cast<uint2*>(row + q) = make_uint2(__byte_perm(t0, u0, 0x5432), __byte_perm(t1, u1, 0x5432));
    S = push_nibble(S, pair_nibble(t0 >> 16, t1 >> 16));
  };
  {
    uint32_t c_q = 0;
    for (uint32_t q = 0; q < nq; q += 2) {
      uint32_t v = __funnelshift_r(w0, w1, pos);
      const uint32_t t0 = event(c_q == 0, T.vlc0[c_q + (v & 0x7F)]);
      c_q = t0 & 0x380u;
      v = __funnelshift_r(v, 0u, t0);
      const uint32_t t1 = q + 1 < nq ? event(c_q == 0, T.vlc0[c_q + (v & 0x7F)]) : 0u;
      c_q = t1 & 0x380u;
      v = __funnelshift_r(v, 0u, t1);
      uint32_t mode = (t0 & 0x40u) | ((t1 & 0x40u) << 1);
      if (mode == 0xC0) {
        run -= 2;
        if (run == -1) mode += 0x40;
        if (run < 0) run = mel.get_run();
      }
      const uint32_t e = T.uvlc0[mode + (v & 0x3F)];
      advance(t0 + t1 + (e >> 5));  // (three counts, at most 30 together, in the low five bits)
      symbols(q, v, t0, t1, e, 1u);
    }
    S >>= row_align;
    row_done(1u);
  }
  for (uint32_t y = 2; y < h; y += 2) {
    row += qs;
    uint32_t c_q = 0;
    uint64_t Qc = (S | (S >> 1)) >> 1;
    uint32_t up7 = ((uint32_t)S & 1u) << 7;
    S = 0;
    for (uint32_t q = 0; q < nq; q += 2) {
      const uint32_t qc = (uint32_t)Qc;
      const uint32_t c0 = c_q | up7 | ((qc & 1u) << 9), a1 = (qc & 5u) << 7;
      up7 = (qc & 4u) << 5;
      Qc >>= 4;
      const bool hasB = q + 1 < nq;
      const uint32_t v = __funnelshift_r(w0, w1, pos);
      // As if no MEL run ended in this pair: a quad with a zero context takes
      // no codeword.
      const bool z0 = c0 == 0;
      uint32_t t0 = T.vlc1[c0 + (v & 0x7F)];
      t0 = z0 ? 0u : t0;
      uint32_t c1 = (t0 & 0x380u) | a1;
      uint32_t v1 = __funnelshift_r(v, 0u, t0);
      const bool z1 = c1 == 0;
      uint32_t t1 = T.vlc1[c1 + (v1 & 0x7F)];
      t1 = z1 || !hasB ? 0u : t1;
      const int events = (z0 ? 2 : 0) + (z1 && hasB ? 2 : 0);
      if (run < events) {
        // One does: event by event.
        t0 = event(z0, T.vlc1[c0 + (v & 0x7F)]);
        c1 = (t0 & 0x380u) | a1;
        v1 = __funnelshift_r(v, 0u, t0);
        t1 = hasB ? event(c1 == 0, T.vlc1[c1 + (v1 & 0x7F)]) : 0u;
      } else {
        run -= events;
      }
      c_q = t1 & 0x380u;
      const uint32_t v2 = __funnelshift_r(v1, 0u, t1);
      const uint32_t mode = (t0 & 0x40u) | ((t1 & 0x40u) << 1);
      const uint32_t e = T.uvlc1[mode + (v2 & 0x3F)];
      advance(t0 + t1 + (e >> 5));
      symbols(q, v2, t0, t1, e, 0u);
    }
    S >>= row_align;
    row_done(y / 2 + 1);
  }
}

}  // namespace

template <bool OUTLINE>
__global__ void __launch_bounds__(kFusedThreads) ht_cleanup_fused_kernel(
    const HtJob* __restrict__ jobs, uint32_t njobs, const uint8_t* __restrict__ arena, uint32_t* __restrict__ symbols,
    int32_t* __restrict__ coef, uint32_t* __restrict__ tile_status, uint32_t ms_words, uint32_t max_w) {
  // The lookup tables: the chain's form for a block at most 64 wide, decode_vlc's
  // for a wider one.
  __shared__ __align__(16) uint32_t tables[sizeof(HtChainTables) / 4];
  __shared__ uint32_t vlc_bits[kChainWords];
  // The symbol table of a block at most 64 wide (rows padded to even counts);
  // a wider block's is in global memory.
  __shared__ __align__(16) uint32_t table[2 * kChainPairs];
  __shared__ uint32_t rows_done;
  extern __shared__ __align__(16) uint8_t smem[];
  if (blockIdx.x >= njobs) return;
  const HtJob job = jobs[blockIdx.x];
  const bool narrow = job.w <= 64;
  {
    static_assert(sizeof(HtChainTables) % 16 == 0 && sizeof(SmemTables) % 16 == 0 &&
                  sizeof(SmemTables) <= sizeof(HtChainTables), "copied by 16 bytes");
    const uint4* from = reinterpret_cast<const uint4*>(narrow ? reinterpret_cast<const uint8_t*>(&g_ht_tables.chain)
                                                              : reinterpret_cast<const uint8_t*>(&g_ht_tables));
    const uint32_t n = (narrow ? sizeof(HtChainTables) : sizeof(SmemTables)) / 16;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) reinterpret_cast<uint4*>(tables)[i] = from[i];
  }
  if (threadIdx.x == 0) rows_done = 0;
  __syncthreads();
  volatile uint32_t* progress = &rows_done;
  if (threadIdx.x < 32) {
    if (job.passes == 0) return;
    const uint8_t* src = arena + job.src;
    const FusedPublish publish{progress};
    bool ok;
    if (narrow) {
      // decode_vlc's checks of the segment.
      const uint32_t lcup = job.lcup;
      uint32_t scup = 0;
      ok = lcup >= 2;
      if (ok) {
        scup = ((uint32_t)ld8(src + lcup - 1) << 4) + (ld8(src + lcup - 2) & 0x0F);
        ok = scup >= 2 && scup <= lcup && scup <= 4079;
      }
      if (ok) unstuff_vlc(src, lcup, scup, vlc_bits);
      if (threadIdx.x != 0) return;
      if (ok)
        chain_vlc<OUTLINE>(job, src, scup, *reinterpret_cast<const HtChainTables*>(tables), vlc_bits, table, publish);
    } else {
      if (threadIdx.x != 0) return;
      ok = decode_vlc<false, OUTLINE>(job, src, symbols + job.sym, *reinterpret_cast<const SmemTables*>(tables),
                                      nullptr, 1, 0, publish);
    }
    if (!ok) {
      __threadfence_block();
      *progress = kRowsFailed;
    }
    return;
  }
  const uint32_t cols = max_w + 4;
  magsgn_block(job, arena, narrow ? table : symbols + job.sym, coef, tile_status, ms_words, cols,
               reinterpret_cast<uint32_t*>(smem), smem + (size_t)ms_words * 4, FusedRowWait{progress});
}

// ---------------------------------------------------------------------------
// Refinement passes for blocks with more than one coding pass.

namespace {

__device__ __forceinline__ uint32_t pair16(const uint16_t* v, uint32_t i) {
  return (uint32_t)v[i] | ((uint32_t)v[i + 1] << 16);
}

__device__ const uint32_t kSpread[16] = {0x33,   0x76,   0xEC,   0xC8,   0x330,   0x760,   0xEC0,   0xC80,
                                         0x3300, 0x7600, 0xEC00, 0xC800, 0x33000, 0x76000, 0xEC000, 0xC8000};

}  // namespace

// One thread per refinement block.  The block's cleanup result (raw
// sign-magnitude words written by ht_magsgn_kernel) gives the significance
// map; SigProp (ht_block_decode.rs:1254-1375) and MagRef (:1377-1433) then
// update the words in place, and the block is converted to int32.
__global__ void ht_refine_kernel(const HtJob* __restrict__ jobs, const uint32_t* __restrict__ list, uint32_t n,
                                 const uint8_t* __restrict__ arena, int32_t* __restrict__ coef,
                                 uint32_t* __restrict__ tile_status) {
  // sigma for blocks up to 4096 samples: rows (h/4 + 1) x stride ((w/4) + 2 + 7) & ~7.
  constexpr uint32_t kSigmaCap = 2560;
  uint16_t sigma[kSigmaCap];
  uint16_t prev_row[272];
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const HtJob job = jobs[list[k]];
    uint32_t* out = reinterpret_cast<uint32_t*>(coef + job.dst);
    const uint32_t w = job.w, h = job.h, stride = job.stride;
    const uint32_t mstr = (((w + 3) / 4) + 2 + 7) & ~7u;
    const uint32_t srows = (h + 3) / 4 + 1;
    bool ok = srows * mstr <= kSigmaCap && (w + 3) / 4 + 8 <= 272;
    const uint32_t p = 30 - job.mmsb;
    if (ok) {
      // Significance of the cleanup pass, 4-row stripes x 4-column groups
      // (build_sigma_from_cleanup_phase layout, :1207-1252).
      for (uint32_t i = 0; i < srows * mstr; ++i) sigma[i] = 0;
      for (uint32_t y = 0; y < h; ++y)
        for (uint32_t x = 0; x < w; ++x)
          if (out[(size_t)y * stride + x] != 0) {
            uint32_t idx = (y >> 2) * mstr + (x >> 2);
            sigma[idx] |= (uint16_t)(1u << (((x & 3) << 2) | (y & 3)));
          }
      const uint8_t* ref = arena + job.src + job.lcup;
      const uint32_t lref = job.lref;
      // SigProp.
      {
        uint32_t prl = (w + 3) / 4 + 8;
        for (uint32_t i = 0; i < prl; ++i) prev_row[i] = 0;
        Fwd<0> sp;
        sp.init(ref, lref);
        const bool causal = job.flags & 1;
        for (uint32_t y = 0; y < h; y += 4) {
          uint32_t pattern = 0xFFFF;
          if (h - y < 4) {
            pattern = 0x7777;
            if (h - y < 3) {
              pattern = 0x3333;
              if (h - y < 2) pattern = 0x1111;
            }
          }
          uint32_t prev = 0;
          uint32_t cur_row = (y >> 2) * mstr, next_row = cur_row + mstr;
          size_t dpp = (size_t)y * stride;
          for (uint32_t x = 0; x < w; x += 4) {
            uint32_t colp = pattern;
            int s = (int)x + 4 - (int)w;
            if (s < 0) s = 0;
            colp >>= (uint32_t)(s * 4);
            uint32_t idx = x >> 2;
            uint32_t ps = (uint32_t)prev_row[idx] | ((uint32_t)prev_row[idx + 1] << 16);
            uint32_t ns = pair16(sigma, next_row + idx);
            uint32_t u = (ps & 0x88888888u) >> 3;
            if (!causal) u |= (ns & 0x11111111u) << 3;
            uint32_t cs = pair16(sigma, cur_row + idx);
            uint32_t mbr = cs;
            mbr |= (cs & 0x77777777u) << 1;
            mbr |= (cs & 0xEEEEEEEEu) >> 1;
            mbr |= u;
            uint32_t t = mbr;
            mbr |= t << 4;
            mbr |= t >> 4;
            mbr |= prev >> 12;
            mbr &= colp;
            mbr &= ~cs;
            uint32_t new_sig = 0;
            if (mbr != 0) {
              uint32_t cwd = sp.fetch();
              uint32_t cnt = 0;
              uint32_t inv_sig = ~cs & colp;
              uint32_t cand = mbr, processed = 0;
              while (cand != 0) {
                uint32_t bit = __ffs(cand) - 1;
                uint32_t m = 1u << bit;
                cand &= ~m;
                processed |= m;
                if (cwd & 1) {
                  new_sig |= m;
                  cand |= kSpread[bit] & inv_sig & ~processed;
                }
                cwd >>= 1;
                ++cnt;
              }
              if (new_sig != 0) {
                uint32_t value = 3u << (p - 2);
                size_t bb = dpp + x;
                uint32_t sb = new_sig;
                while (sb != 0) {
                  uint32_t bit = __ffs(sb) - 1;
                  sb &= ~(1u << bit);
                  size_t off = (size_t)(bit >> 2) + (size_t)(bit & 3) * stride;
                  out[bb + off] = ((cwd & 1) << 31) | value;
                  cwd >>= 1;
                  ++cnt;
                }
              }
              sp.advance(cnt);
            }
            uint32_t comb = new_sig | cs;
            prev_row[idx] = (uint16_t)comb;
            if (idx + 1 < prl) prev_row[idx + 1] = (uint16_t)(comb >> 16);
            uint32_t np = comb;
            np |= (comb & 0x7777u) << 1;
            np |= (comb & 0xEEEEu) >> 1;
            prev = (np | u) & 0xF000;
          }
        }
      }
      // MagRef.
      if (job.passes > 2) {
        if (p < 2) {
          ok = false;
        } else {
          // Backward reader over the refinement segment (new_mrp).
          Vlc mr;
          mr.init_mrp(ref, lref);
          uint32_t half = 1u << (p - 2);
          for (uint32_t y = 0; y < h; y += 4) {
            uint32_t csi = (y >> 2) * mstr;
            size_t dpp = (size_t)y * stride;
            for (uint32_t i = 0; i < w; i += 8) {
              uint32_t cwd = mr.fetch();
              uint32_t sig = pair16(sigma, csi);
              csi += 2;
              uint32_t col_mask = 0xF;
              if (sig != 0) {
                for (uint32_t j = 0; j < 8; ++j) {
                  if (sig & col_mask) {
                    size_t dp = dpp + i + j;
                    uint32_t sm = 0x11111111u & col_mask;
                    for (int kk = 0; kk < 4; ++kk) {
                      if (sig & sm) {
                        uint32_t sym = cwd & 1;
                        sym = (1 - sym) << (p - 1);
                        sym |= half;
                        out[dp] ^= sym;
                        cwd >>= 1;
                      }
                      sm <<= 1;
                      dp += stride;
                    }
                  }
                  col_mask <<= 4;
                }
              }
              mr.advance(__popc(sig));
            }
          }
        }
      }
    }
    // Convert to int32 coefficients (or zero the block on failure).
    for (uint32_t y = 0; y < h; ++y)
      for (uint32_t x = 0; x < w; ++x) {
        uint32_t& v = out[(size_t)y * stride + x];
        v = ok ? (uint32_t)to_i32(v, job.nbp) : 0u;
      }
    if (!ok) atomicOr(&tile_status[job.tile], kStatusDecode);
  }
}

size_t ht_magsgn_smem_bytes(uint32_t ms_words, uint32_t max_w, uint32_t warps) {
  return (size_t)warps * ms_words * 4 + (size_t)warps * 2 * (max_w + 4);
}

cudaError_t ht_kernels_init() {
  // The VLC pass's lanes read their blocks' bytes a few at a time over the
  // whole chain, so its L1 hit rate matters more than a ninth resident CTA:
  // left to itself the driver sizes shared memory for the CTAs that the
  // registers allow (228 KB, 28 KB of L1); 72 % (164 KB, 7 CTAs of 21.6 KB)
  // leaves 92 KB of L1 (C2 VLC pass 0.96 -> 0.88 ms).
  for (const void* k : {(const void*)ht_vlc_kernel<true>, (const void*)ht_vlc_kernel<false>}) {
    const cudaError_t c = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 72);
    if (c != cudaSuccess) return c;
  }
  for (const void* k : {(const void*)ht_cleanup_fused_kernel<true>, (const void*)ht_cleanup_fused_kernel<false>}) {
    const cudaError_t c = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (c != cudaSuccess) return c;
  }
  cudaError_t e = cudaFuncSetAttribute(ht_magsgn_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(ht_magsgn_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
}

cudaError_t launch_ht_vlc(const HtJob* jobs, uint32_t njobs, const uint8_t* arena, uint32_t* symbols,
                          cudaStream_t stream, uint32_t threads, uint32_t lanes, bool outline) {
  if (njobs == 0) return cudaSuccess;
  if (threads == 0 || threads > kHtThreads || threads % 32) threads = kHtThreads;
  if (lanes == 0 || lanes > 32 || (lanes & (lanes - 1))) lanes = 32;
  const uint32_t warps = (njobs + lanes - 1) / lanes, per_cta = threads / 32;
  const uint32_t grid = (warps + per_cta - 1) / per_cta;
  if (outline) ht_vlc_kernel<true><<<grid, threads, 0, stream>>>(jobs, njobs, arena, symbols, lanes);
  else ht_vlc_kernel<false><<<grid, threads, 0, stream>>>(jobs, njobs, arena, symbols, lanes);
  return cudaGetLastError();
}

cudaError_t launch_ht_fused(const HtJob* jobs, uint32_t njobs, const uint8_t* arena, uint32_t* symbols, int32_t* coef,
                           uint32_t* tile_status, uint32_t ms_words, uint32_t max_w, cudaStream_t stream,
                           bool outline) {
  if (njobs == 0) return cudaSuccess;
  const size_t smem = ht_magsgn_smem_bytes(ms_words, max_w, 1);
  if (smem > 200 * 1024) return cudaErrorInvalidValue;
  if (outline)
    ht_cleanup_fused_kernel<true><<<njobs, kFusedThreads, smem, stream>>>(jobs, njobs, arena, symbols, coef,
                                                                          tile_status, ms_words, max_w);
  else
    ht_cleanup_fused_kernel<false><<<njobs, kFusedThreads, smem, stream>>>(jobs, njobs, arena, symbols, coef,
                                                                           tile_status, ms_words, max_w);
  return cudaGetLastError();
}

cudaError_t launch_ht_magsgn(const HtJob* jobs, uint32_t njobs, const uint8_t* arena, const uint32_t* symbols,
                             int32_t* coef, uint32_t* tile_status, uint32_t ms_words, uint32_t max_w,
                             cudaStream_t stream, uint32_t warps, uint32_t* queue, uint32_t gran,
                             uint32_t persistent_ctas, uint32_t nsingle) {
  if (njobs == 0) return cudaSuccess;
  if (warps == 0 || warps > kMsWarps) warps = kMsWarps;
  nsingle = std::min(nsingle, njobs);
  size_t smem = ht_magsgn_smem_bytes(ms_words, max_w, warps);
  if (smem > 227 * 1024) return cudaErrorInvalidValue;
  const uint32_t nitems = nsingle + (njobs - nsingle + 1) / 2;
  uint32_t ctas = (nitems + warps - 1) / warps;
  if (queue) {
    if (gran == 0) gran = 1;
    ctas = std::max(1u, std::min(ctas, persistent_ctas));
  }
  if (queue)
    ht_magsgn_kernel<true><<<ctas, warps * 32, smem, stream>>>(jobs, njobs, arena, symbols, coef, tile_status,
                                                               ms_words, max_w, queue, gran, nsingle);
  else
    ht_magsgn_kernel<false><<<ctas, warps * 32, smem, stream>>>(jobs, njobs, arena, symbols, coef, tile_status,
                                                                ms_words, max_w, nullptr, 0, nsingle);
  return cudaGetLastError();
}

cudaError_t ht_magsgn_occupancy(uint32_t ms_words, uint32_t max_w, uint32_t warps, int* ctas_per_sm) {
  if (warps == 0 || warps > kMsWarps) warps = kMsWarps;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas_per_sm, ht_magsgn_kernel<true>, warps * 32,
                                                       ht_magsgn_smem_bytes(ms_words, max_w, warps));
}

cudaError_t launch_ht_cleanup(const HtJob* jobs, uint32_t njobs, const uint8_t* arena, uint32_t* symbols,
                              int32_t* coef, uint32_t* tile_status, uint32_t ms_words, uint32_t max_w,
                              cudaStream_t stream) {
  cudaError_t e = launch_ht_vlc(jobs, njobs, arena, symbols, stream, kHtThreads);
  if (e != cudaSuccess) return e;
  return launch_ht_magsgn(jobs, njobs, arena, symbols, coef, tile_status, ms_words, max_w, stream, kMsWarps, nullptr,
                          0, 0, njobs);
}

cudaError_t launch_ht_refine(const HtJob* jobs, const uint32_t* list, uint32_t n, const uint8_t* arena, int32_t* coef,
                             uint32_t* tile_status, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  uint32_t threads = 64, blocks = (n + threads - 1) / threads;
  ht_refine_kernel<<<blocks, threads, 0, stream>>>(jobs, list, n, arena, coef, tile_status);
  return cudaGetLastError();
}

cudaError_t upload_ht_tables(const HtDecodeTables& host) {
  return cudaMemcpyToSymbol(g_ht_tables, &host, sizeof(HtDecodeTables));
}

}  // namespace sgn
