// Device-side building blocks of the NZR1 rANS decoder, shared by the decode
// kernels (nz_decode.cu) and the fused decode -> tensor-core GEMM (nz_linear.cu):
// PTX helpers, the per-symbol decode step, the merge of decoded exponents with the
// packed fractions, unit planning / staging / opening, and the decode-table build.
#pragma once

#include "nz_common.cuh"

namespace nz {

// A wait is a bounded number of tries; each may suspend the thread for up to kWaitHintNs, so
// that a warp that waits takes no issue slots from those that decode.  The hint is an upper
// limit only, a try may return at once: the number of tries is what a slow copy (a container in
// host memory) has to get by with, about a second at the most.
constexpr uint32_t kWaitHintNs = 1000;
constexpr uint32_t kMaxWaitIters = 1u << 20;

// ------------------------------------------------------------- PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t lds_u16(uint32_t a) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t lds_u8(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(kWaitHintNs)
      : "memory");
  return ok != 0;
}
// Bulk asynchronous copy global -> this CTA's shared memory (no multicast).
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes,
                                         uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(dst),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}

// Hint: bring a run of global memory (16-byte aligned, a multiple of 16 bytes) into L2.
__device__ __forceinline__ void bulk_prefetch_l2(const void *src, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}

// ------------------------------------------------------------------ decode
struct LaneState {
  uint32_t x;     // rANS state
  uint32_t p;     // shared address of the next unread stream word
  uint32_t w;     // that word, already loaded
};

// Per-lane constants of the replicated decode table.
struct LutView {
  uint32_t base;    // shared address of this lane's copy (table base + bank offset)
  uint32_t mask;    // 2^pb - 1
  uint32_t stride;  // bytes between slots (4 x copies)
  uint32_t pb;      // probability bits
  uint32_t k64k;    // 65536 in a register: keeps the shift-in an integer multiply-add
  uint32_t narrow;  // the table holds narrow entries
};

// Table entries, two layouts (`first` = first slot of the symbol):
//   wide    symbol << 23 | freq << 12 | (slot - first): any frequency up to 2047 (the
//           encoder's choice of resolution sees to that, the table build checks it).
//   narrow  (slot - first) << 23 | symbol << 15 | freq: frequencies up to 512, which a
//           9-bit table always has and weights at any resolution do too.
// Either way one byte permutation puts the symbols of two entries where the exponents of
// an output word's two bf16 go.  With the narrow layout frequency and offset are one
// operation each and the state update needs no correction term: 11 instead of 12
// instructions per symbol.  Measured on a B200 with units of 256 symbols, two chains a warp:
// 86 instead of 98 cycles a step in a lone warp, 226 instead of 242 with 20 warps (there the
// integer pipe and the memory are both nearly full).
constexpr uint32_t kEntSymShift = 23;
constexpr uint32_t kEntFreqShift = 12;
constexpr uint32_t kNarrowOffShift = 23;
constexpr uint32_t kNarrowSymShift = 15;
constexpr uint32_t kNarrowMaxFreq = 512;
// Resolution of the usual tables of a precision (up to 32 distinct exponents), the only one
// with a loop for narrow entries.
__host__ __device__ constexpr uint32_t usual_prob_bits(int precision) {
  return precision == 7 ? kMinProbBits : kDefaultLowProbBits;
}
__device__ __forceinline__ uint32_t entry_symbol(uint32_t ent) { return ent >> kEntSymShift; }

// One symbol.  Written in PTX so that the renormalisation stays predicated (no divergent
// branch) and the 16-bit stream word is loaded straight into a 32-bit register.
// ROW > 0: the table is narrow, has 2^PB slots and 2^ROW bytes between them (a constant
// factor folds into the address computation of the dependent chain x -> slot -> entry -> x
// that bounds a lane's rate); returns the narrow entry.
// ROW == 0: the table is wide; returns the wide entry.  The state update is
// f*(q - 4096) + (f*4096 + offset) = f*q + offset (mod 2^32), so that the entry's low 23
// bits serve as the addend unshifted.
// ROW == kNarrowRow: the table is narrow, its size is looked up (units decoded on their own);
// returns the entry with the symbol where the wide layout has it.
constexpr int kNarrowRow = -1;
template <int ROW, int PB = 0>
__device__ __forceinline__ uint32_t decode_step(LaneState &st, const LutView &lv) {
  uint32_t ent;
  if constexpr (ROW > 0) {
    asm volatile(
        "{\n\t"
        ".reg .b32 a, q, f, b;\n\t"
        ".reg .pred r;\n\t"
        "and.b32 a, %1, %6;\n\t"
        "mad.lo.u32 a, a, %8, %4;\n\t"         // slot * 2^ROW + lane's table base
        "ld.shared.u32 %0, [a];\n\t"
        "shr.u32 q, %1, %7;\n\t"
        "and.b32 f, %0, 0x7FFF;\n\t"
        "shr.u32 b, %0, 23;\n\t"
        "mad.lo.u32 %1, f, q, b;\n\t"
        "setp.lt.u32 r, %1, 65536;\n\t"
        "@r mad.lo.u32 %1, %1, %5, %3;\n\t"    // x = x * 65536 + w
        "@r add.u32 %2, %2, 2;\n\t"
        "@r ld.shared.u16 %3, [%2];\n\t"
        "}"
        : "=&r"(ent), "+r"(st.x), "+r"(st.p), "+r"(st.w)
        : "r"(lv.base), "r"(lv.k64k), "n"((1 << PB) - 1), "n"(PB), "n"(1 << ROW));
  } else if constexpr (ROW == kNarrowRow) {
    asm volatile(
        "{\n\t"
        ".reg .b32 a, q, f, b;\n\t"
        ".reg .pred r;\n\t"
        "and.b32 a, %1, %5;\n\t"
        "mad.lo.u32 a, a, %6, %4;\n\t"         // slot * stride + lane's table base
        "ld.shared.u32 %0, [a];\n\t"
        "shr.u32 q, %1, %7;\n\t"
        "and.b32 f, %0, 0x7FFF;\n\t"
        "shr.u32 b, %0, 23;\n\t"
        "mad.lo.u32 %1, f, q, b;\n\t"
        "setp.lt.u32 r, %1, 65536;\n\t"
        "@r mad.lo.u32 %1, %1, %8, %3;\n\t"    // x = x * 65536 + w
        "@r add.u32 %2, %2, 2;\n\t"
        "@r ld.shared.u16 %3, [%2];\n\t"
        "}"
        : "=&r"(ent), "+r"(st.x), "+r"(st.p), "+r"(st.w)
        : "r"(lv.base), "r"(lv.mask), "r"(lv.stride), "r"(lv.pb), "r"(lv.k64k));
    ent = (ent << (kEntSymShift - kNarrowSymShift)) & 0x7F800000u;
  } else {
    asm volatile(
        "{\n\t"
        ".reg .b32 a, q, f, b;\n\t"
        ".reg .pred r;\n\t"
        "and.b32 a, %1, %5;\n\t"
        "mad.lo.u32 a, a, %6, %4;\n\t"         // slot * stride + lane's table base
        "ld.shared.u32 %0, [a];\n\t"
        "shr.u32 q, %1, %7;\n\t"
        "add.s32 q, q, -4096;\n\t"
        "and.b32 b, %0, 0x7FFFFF;\n\t"         // freq << 12 | offset
        "shr.u32 f, b, 12;\n\t"
        "mad.lo.u32 %1, f, q, b;\n\t"
        "setp.lt.u32 r, %1, 65536;\n\t"
        "@r mad.lo.u32 %1, %1, %8, %3;\n\t"    // x = x * 65536 + w
        "@r add.u32 %2, %2, 2;\n\t"
        "@r ld.shared.u16 %3, [%2];\n\t"
        "}"
        : "=&r"(ent), "+r"(st.x), "+r"(st.p), "+r"(st.w)
        : "r"(lv.base), "r"(lv.mask), "r"(lv.stride), "r"(lv.pb), "r"(lv.k64k));
  }
  return ent;
}
// One symbol of either table, for code that runs too rarely to have a loop for each.
__device__ __forceinline__ uint32_t decode_step_any(LaneState &st, const LutView &lv) {
  return lv.narrow ? decode_step<kNarrowRow>(st, lv) : decode_step<0>(st, lv);
}
// Byte selector that joins the symbols of two entries (see the layouts above): from narrow
// entries when ROW > 0, from entries in the wide layout when ROW == 0.
template <int ROW>
__device__ __forceinline__ uint32_t join_symbols(uint32_t ea, uint32_t eb) {
  return __byte_perm(ea, eb, ROW > 0 ? 0x6521 : 0x7632);
}

// Merge two decoded symbols (table entries ea, eb) with their fields.
template <int S>
__device__ __forceinline__ uint32_t merge_pair_generic(uint32_t ea, uint32_t eb, uint32_t fa,
                                                       uint32_t fb, bool canon) {
  uint32_t out[2];
  const uint32_t e[2] = {entry_symbol(ea), entry_symbol(eb)};
  const uint32_t f[2] = {fa, fb};
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const uint32_t frac = (f[k] & ((1u << S) - 1u)) << (7 - S);
    const uint32_t sign = (f[k] >> S) & 1u;
    uint32_t v = (e[k] << 7) | frac | (sign << 15);
    if (canon && e[k] == 255u && frac != 0u) v = 0x7FFFu;
    out[k] = v;
  }
  return out[0] | (out[1] << 16);
}

// Lossless fast path: two entries + two fraction bytes -> one 32-bit word.
//   sel picks the two fraction bytes (a in both low bytes, b in both high).
// Two bytes of each entry hold its exponent in place.
template <int ROW>
__device__ __forceinline__ uint32_t merge_pair_s7(uint32_t ea, uint32_t eb, uint32_t fw,
                                                  uint32_t sel) {
  const uint32_t e = join_symbols<ROW>(ea, eb);
  const uint32_t g = __byte_perm(fw, 0, sel);            // fa fa fb fb
  return (e & 0x7F807F80u) | (g & 0x807F807Fu);
}

// A lane's packed fractions for one block (8 elements = s+1 bytes), streaming
// (evict-first) and volatile so that the loads stay where the code puts them:
// several blocks ahead of their use.
template <int S>
__device__ __forceinline__ uint64_t load_frac(const uint8_t *p) {
  if (S == 7) {
    uint32_t lo, hi;
    asm volatile("ld.global.cs.v2.u32 {%0, %1}, [%2];" : "=r"(lo), "=r"(hi) : "l"(p));
    return ((uint64_t)hi << 32) | lo;
  } else if (S == 3) {
    uint32_t v;
    asm volatile("ld.global.cs.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
  } else if (S == 1) {
    uint32_t v;
    asm volatile("ld.global.cs.u16 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
  } else {
    uint32_t v;
    asm volatile("ld.global.cs.u8 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
  }
}

// One output word (two elements) from two table entries and the lane's packed
// fractions of the block; `pair` is 0..3.
template <int S, int ROW = 0>
__device__ __forceinline__ uint32_t merge_word(uint32_t ea, uint32_t eb, uint64_t fbits, int pair) {
  if (S == 7) {
    const uint32_t half = (pair < 2) ? (uint32_t)fbits : (uint32_t)(fbits >> 32);
    return merge_pair_s7<ROW>(ea, eb, half, (pair & 1) ? 0x3322 : 0x1100);
  }
  // Lossy precisions: the pair's (s+1)-bit fields share one byte B of the packed
  // fractions.  One multiplication lays copies of B side by side (the shifts are
  // far enough apart that the copies never overlap, so nothing carries) such that
  // every sign and mantissa bit has a copy at its place in the output word; a mask
  // keeps those places.  The exponents come in place from the two entries, as in the
  // lossless path.
  const uint32_t e = join_symbols<ROW>(ea, eb) & 0x7F807F80u;
  const uint32_t f = (uint32_t)fbits;
  if (S == 3) {
    // B = [sa ma2 ma1 ma0 sb mb2 mb1 mb0]: ma -> bits 4..6 (shift 0), sa -> 15 (8),
    // mb -> 20..22 (20), sb -> 31 (28)
    const uint32_t B = __byte_perm(f, 0, 0x4440 | pair);
    return e | ((B * 0x10100101u) & 0x80708070u);
  }
  if (S == 1) {
    // B holds four 2-bit fields [s m]; the pair is the upper or the lower two of them
    const uint32_t B = __byte_perm(f, 0, 0x4440 | (pair >> 1));
    // upper two: sa bit 7 -> 15 (8), ma bit 6 -> 6 (0), sb bit 5 -> 31 (26), mb bit 4 -> 22 (18)
    // lower two: sa bit 3 -> 15 (12), ma bit 2 -> 6 (4), sb bit 1 -> 31 (30), mb bit 0 -> 22 (22)
    const uint32_t m = (pair & 1) ? 0x40401010u : 0x04040101u;
    return e | ((B * m) & 0x80408040u);
  }
  // B holds the block's eight sign bits, first element in bit 7:
  // sa bit 7-2p -> 15 (8+2p), sb bit 6-2p -> 31 (25+2p)
  const uint32_t B = f & 0xFFu;
  return e | ((B * ((1u << (8 + 2 * pair)) + (1u << (25 + 2 * pair)))) & 0x80008000u);
}
// NaN -> 0x7FFF in both halves of an output word (exponent 255, some mantissa bit).
__device__ __forceinline__ uint32_t canon_word(uint32_t w) {
  if ((w & 0x7FFFu) > 0x7F80u) w = (w & 0xFFFF0000u) | 0x7FFFu;
  if ((w & 0x7FFF0000u) > 0x7F800000u) w = (w & 0xFFFFu) | 0x7FFF0000u;
  return w;
}

struct DecodeArgs {
  const uint8_t *container;
  const uint8_t *frac;
  uint64_t n;
  uint32_t S;
  uint32_t n_units;
  uint32_t full_units;  // units that hold 32 * S elements (all but, perhaps, the last)
  uint64_t pay_off;     // byte offset of the payload in the container
  uint32_t max_words;   // 16-bit words of payload the buffer can hold (capped at 2^31 - 1)
  uint32_t slot_bytes;
  uint32_t lut_shift;   // log2 of the bytes per slot row for a 2^12-slot table (2..5)
  uint32_t lut_bytes;   // 4096 << lut_shift
  int canon;
  uint16_t *out_bf16;
  uint8_t *out_exp;
  uint32_t *status;
  const uint32_t *unit_list;   // units to decode, in output order (gather launches only)
  uint32_t n_work;             // units this launch decodes: n_units, or the length of the list
  const float *gx;             // matrix-vector launches: input vector (fp32, `in` entries)
  float *partial;              //   partial sums, `seg` places per unit
  uint32_t in;                 //   row length of the [out, in] matrix, a multiple of 256
  uint32_t seg;                //   rows a unit can touch
  uint32_t tile_cols;          // operand order: row length of the matrix (0 = the stream is the tensor)
  uint32_t segs;               //   units per row group, (tile_cols / 64) / (S / 8)
  // block normaliser: one stored byte per group of 2^norm_lg elements (null = none)
  const uint8_t *norm;
  uint32_t norm_lg;
  // update launches: gradient (bf16) and AdamW moments (bf16), indexed like the output tensor
  const uint16_t *grad;
  uint16_t *exp_avg, *exp_avg_sq;
  AdamArgs adam;
};

// Operand order.  A [rows, cols] matrix (rows % 4 == 0, cols % 64 == 0) may be stored
// with its elements permuted so that one 256-element block of the stream is a
// 4-row x 64-column patch of the matrix: stream element
//   e = ((g * (cols / 64) + kb) * 4 + r) * 64 + c
// is matrix element (4 g + r, 64 kb + c).  A lane's 8 consecutive stream elements
// are still 8 consecutive elements of one row (16 contiguous bytes), a quarter warp's
// 64 are 128 contiguous bytes; 32 consecutive row groups at one kb form the 128 x 64
// tensor-core operand tile.  Units hold whole blocks and never straddle a row group
// (lane_symbols / 8 divides cols / 64).
__device__ __forceinline__ uint64_t operand_index(uint64_t e, uint32_t cols) {
  const uint64_t block = e >> 8;
  const uint32_t w = (uint32_t)e & 255u;
  const uint32_t spr = cols >> 6;                       // blocks per row group
  const uint64_t g = block / spr;
  const uint32_t kb = (uint32_t)(block - g * spr);
  return (4 * g + (w >> 6)) * cols + kb * 64u + (w & 63u);
}
// Block normaliser on the way out (cuda/kernels.cuh:208-216 of the reference): a decoded
// bf16 value times the scale 1.<8 stored mantissa bits> of its group, rounded to bf16
// (nearest even) -- the arithmetic of nz_denormalize_bf16.
__device__ __forceinline__ float norm_scale(uint32_t stored_byte) {
  return __uint_as_float(0x3F800000u | (stored_byte << 15));
}
__device__ __forceinline__ uint32_t scale_bf16_bits(uint32_t bits16, float scale) {
  const float f = scale * __uint_as_float(bits16 << 16);
  uint32_t u = __float_as_uint(f);
  if ((u & 0x7F800000u) == 0x7F800000u && (u & 0x007FFFFFu)) return 0x7FFFu;    // NaN
  u += 0x7FFFu + ((u >> 16) & 1u);
  return u >> 16;
}
// The same for the two halves of an output word; the conversion writes 0x7FFF for NaN too.
__device__ __forceinline__ uint32_t scale_bf16_word(uint32_t w, float s0, float s1) {
  const float lo = s0 * __uint_as_float(w << 16), hi = s1 * __uint_as_float(w & 0xFFFF0000u);
  uint32_t out;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(out) : "f"(hi), "f"(lo));
  return out;
}
// Where stream element e goes in the output tensor.
__device__ __forceinline__ uint64_t out_index(const DecodeArgs &a, uint64_t e) {
  return a.tile_cols ? operand_index(e, a.tile_cols) : e;
}

// Where a lane's first element of unit u goes (all indices are below 2^32).
__device__ __forceinline__ uint32_t unit_out_index(const DecodeArgs &a, uint32_t u, uint32_t lane) {
  if (!a.tile_cols) return u * (32u * a.S) + lane * 8;
  const uint32_t g = u / a.segs, kb = (u - g * a.segs) * (a.S >> 3);
  return (4 * g + (lane >> 3)) * a.tile_cols + kb * 64u + (lane & 7u) * 8;
}

__device__ __forceinline__ void raise(uint32_t *status, uint32_t bits) {
  if (status) atomicOr(status, bits);
}

// Asynchronous per-lane copy of one block's packed fractions (4 or 8 bytes)
// from global to this lane's place in the warp's shared-memory ring.  Unlike a
// register load this occupies no register scoreboard while in flight, so the
// table and stream loads of the decode chain never wait behind it.
template <int S>
__device__ __forceinline__ void frac_async(uint32_t dst, const uint8_t *src) {
  if (S == 7)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void frac_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void frac_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
template <int S>
__device__ __forceinline__ uint64_t frac_from_ring(uint32_t addr) {
  if (S == 7) {
    uint32_t lo, hi;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(lo), "=r"(hi) : "r"(addr));
    return ((uint64_t)hi << 32) | lo;
  }
  return lds_u32(addr);
}

constexpr int kChains = 2;                       // units a warp decodes side by side

constexpr uint32_t kRingSlots = 4;               // blocks of fractions in flight per unit + 1
// Shared-memory ring of a warp for the packed fractions, by precision.  One unit's
// place holds, for precisions 7 and 3, one block (32 lanes x 8 or 4 bytes; four such
// slots) and, for precisions 1 and 0, a group of four blocks (32 lanes x 8 or 4
// bytes; two buffers).
__host__ __device__ constexpr uint32_t ring_unit_bytes(int precision) {
  return (precision == 7 || precision == 1) ? 256u : 128u;
}
__host__ __device__ constexpr uint32_t ring_warp_bytes(int precision) {
  return ((precision == 7 || precision == 3) ? kRingSlots : 2u) * kChains *
         ring_unit_bytes(precision);
}
// Precisions whose ring is filled block by block, per lane (the others: group by group).
__host__ __device__ constexpr bool ring_by_block(int s) { return s == 7 || s == 3; }

// What a warp knows about a unit it has planned.
struct UnitPlan {
  uint32_t kind;       // 0 = nothing to do, 1 = raw, 2 = coded
  uint32_t word0;      // first word of the unit in the payload
  uint32_t words;      // unit length in words
  uint32_t copy_bytes; // size of the widened bulk copy (coded)
  __device__ __forceinline__ uint64_t byte0() const { return (uint64_t)word0 * 2; }
  // byte offset of the unit inside its slot (the copy starts on a 16-byte boundary)
  __device__ __forceinline__ uint32_t head() const { return (word0 & 7u) * 2; }
};
constexpr uint32_t kUnitSkip = 0, kUnitRaw = 1, kUnitCoded = 2;

// The two entries of the offset table that bound unit u (zeros for no unit).
__device__ __forceinline__ void unit_offsets(const DecodeArgs &a, uint32_t u, uint32_t &off0,
                                             uint32_t &off1) {
  off0 = off1 = 0;
  if (u < a.n_units) {
    const uint32_t *offsets = reinterpret_cast<const uint32_t *>(a.container + kOffsetsOffset) + u;
    off0 = __ldg(offsets);
    off1 = __ldg(offsets + 1);
  }
}

// Validate unit u, bounded by the offset-table entries off0 and off1, against the buffer
// limits the host passed (not against anything read from the container).  All lanes return
// the same plan.
__device__ __forceinline__ UnitPlan plan_unit(const DecodeArgs &a, uint32_t u, uint32_t off0,
                                              uint32_t off1, uint32_t lane) {
  UnitPlan pl;
  pl.kind = kUnitSkip;
  pl.word0 = 0;
  pl.words = 0;
  pl.copy_bytes = 0;
  if (u >= a.n_units) return pl;
  const uint32_t w0 = off0 & ~kRawFlag, w1 = off1 & ~kRawFlag;
  pl.word0 = w0;
  pl.words = w1 - w0;
  bool good = w1 >= w0 && w1 <= a.max_words;
  if (off0 & kRawFlag) {
    const uint32_t U = 32u * a.S;
    const uint32_t count = u < a.full_units ? U : (uint32_t)a.n - u * U;
    good = good && pl.words * 2 >= count;      // a unit has at most 2^15 elements
    if (good) pl.kind = kUnitRaw;
  } else {
    // the copy is widened to 16-byte boundaries: it must still end inside the buffer (the
    // payload starts on such a boundary)
    const uint32_t c0 = w0 & ~7u, c1 = (w1 + 7u) & ~7u;
    const uint32_t bytes = (c1 - c0) * 2;
    good = good && pl.words >= 16 + 2 * 32 && pl.words <= 0xFFFFu && bytes <= a.slot_bytes &&
           c1 <= (a.max_words & ~7u);
    if (good) {
      pl.copy_bytes = bytes;
      pl.kind = kUnitCoded;
    }
  }
  if (!good && lane == 0) raise(a.status, NZ_STATUS_BAD_OFFSETS);
  return pl;
}

// Lane 0 arms the warp's mbarrier with the bytes of all copies and starts them.
// Returns true when at least one copy was issued.
__device__ __forceinline__ bool stage_units(const DecodeArgs &a, const UnitPlan (&pl)[kChains],
                                            uint32_t slot0, uint32_t bar, uint32_t lane) {
  uint32_t bytes = 0;
#pragma unroll
  for (int c = 0; c < kChains; ++c) bytes += pl[c].copy_bytes;
  if (bytes == 0) return false;
  if (lane == 0) {
    const uint8_t *payload = a.container + a.pay_off;
    mbar_expect_tx(bar, bytes);
#pragma unroll
    for (int c = 0; c < kChains; ++c)
      if (pl[c].copy_bytes)
        bulk_g2s(slot0 + c * a.slot_bytes, payload + (uint64_t)(pl[c].word0 & ~7u) * 2,
                 pl[c].copy_bytes, bar);
  }
  return true;
}

// Bounded wait for the warp's bulk copies.  Returns false when it ran out.
__device__ __forceinline__ bool wait_staged(uint32_t bar, uint32_t parity) {
  for (uint32_t it = 0; it < kMaxWaitIters; ++it)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

// Read the 32 lane lengths of a staged unit, check them against the unit
// length and set up this lane's state.  Returns false (same for all lanes)
// when the lengths are inconsistent.
__device__ __forceinline__ bool open_unit(const UnitPlan &pl, uint32_t slot, uint32_t lenq,
                                          uint32_t lane, LaneState &st) {
  const uint32_t ub = slot + pl.head();           // shared address of the unit
  const uint32_t q = lds_u8(ub + lane) * lenq;   // my stream length in words
  uint32_t incl = q;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= (uint32_t)o) incl += v;
  }
  const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
  if (__any_sync(0xFFFFFFFFu, q < 2) || 16u + total != pl.words) return false;
  const uint32_t sw = ub + 2 * (16 + incl - q);
  st.x = lds_u16(sw) | (lds_u16(sw + 2) << 16);
  st.p = sw + 4;
  st.w = lds_u16(st.p);
  return true;
}

// The same for two units at once: the lengths of both go through one packed scan (a unit's
// sum is at most 32 x 510, so the halves do not meet).
__device__ __forceinline__ bool open_pair(const UnitPlan (&pl)[kChains], uint32_t slot0,
                                          uint32_t slot_bytes, uint32_t lenq, uint32_t lane,
                                          LaneState (&st)[kChains]) {
  static_assert(kChains == 2, "two chains per warp");
  const uint32_t ub0 = slot0 + pl[0].head(), ub1 = slot0 + slot_bytes + pl[1].head();
  const uint32_t q0 = lds_u8(ub0 + lane) * lenq, q1 = lds_u8(ub1 + lane) * lenq;
  const uint32_t q = q0 | (q1 << 16);
  uint32_t incl = q;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= (uint32_t)o) incl += v;
  }
  const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
  if (__any_sync(0xFFFFFFFFu, q0 < 2 || q1 < 2) ||
      total + 0x00100010u != (pl[0].words | (pl[1].words << 16)))
    return false;
  const uint32_t before = incl - q + 0x00100010u;
  const uint32_t s0 = ub0 + 2 * (before & 0xFFFFu), s1 = ub1 + 2 * (before >> 16);
  st[0].x = lds_u16(s0) | (lds_u16(s0 + 2) << 16);
  st[1].x = lds_u16(s1) | (lds_u16(s1 + 2) << 16);
  st[0].p = s0 + 4;
  st[1].p = s1 + 4;
  st[0].w = lds_u16(s0 + 4);
  st[1].w = lds_u16(s1 + 4);
  return true;
}

// ---------------------------------------------------------------- decode table
// The table is built by all warps of a CTA in three steps with a __syncthreads()
// between them (the caller places the barriers):
//   table_scan     warp 0 scans the container's 256 frequencies into cum_sh[257]; one
//                  other thread checks the header against what the host passed
//   table_verdict  (after a barrier) every thread computes the same verdict
//   table_fill     warps take 32 slots in turn, look their symbols up and write the rows
// table_prefetch requests the frequencies that table_scan works on: called before anything
// that waits, so that their latency overlaps the first units' planning.
// flag_sh points at four words: header verdict, probability bits, "a frequency does
// not fit the table entry", "every frequency fits the narrow entry".
__device__ __forceinline__ uint4 table_prefetch(const DecodeArgs &a, uint32_t warp, uint32_t lane) {
  uint4 fv = make_uint4(0, 0, 0, 0);
  if (warp == 0) fv = __ldg(reinterpret_cast<const uint4 *>(a.container + kFreqOffset) + lane);
  return fv;
}
__device__ __forceinline__ void table_scan(const DecodeArgs &a, const Header *h, const uint4 fv,
                                           uint16_t *cum_sh, uint32_t *flag_sh, uint32_t warp,
                                           uint32_t lane, uint32_t n_warps) {
  uint32_t *pb_sh = flag_sh + 1;
  uint32_t *wide_sh = flag_sh + 2;
  if (warp == 0) {
    // inclusive scan of the 256 frequencies, 8 per lane
    const uint32_t fw[4] = {fv.x, fv.y, fv.z, fv.w};
    uint32_t f[8], sum = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      f[k] = (fw[k >> 1] >> ((k & 1) * 16)) & 0xFFFFu;
      sum += f[k];
    }
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= (uint32_t)o) incl += v;
    }
    uint32_t run = incl - sum;
    uint32_t widest = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) widest = max(widest, f[k]);
    const bool too_wide = __any_sync(0xFFFFFFFFu, widest >> (kEntSymShift - kEntFreqShift));
    const bool all_narrow = __all_sync(0xFFFFFFFFu, widest <= kNarrowMaxFreq);
    if (lane == 0) {
      cum_sh[0] = 0;
      *wide_sh = too_wide ? 1u : 0u;
      flag_sh[3] = all_narrow ? 1u : 0u;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      run += f[k];
      cum_sh[lane * 8 + k + 1] = (uint16_t)(run > 0xFFFF ? 0xFFFF : run);
    }
  }
  if (threadIdx.x == (n_warps > 1 ? 32u : 0u)) {
    const bool ok = h->magic == kMagic && h->version == 1 && h->n_symbols == a.n &&
                    h->lane_symbols == a.S && h->n_units == a.n_units &&
                    h->len_quantum == len_quantum(a.S) && h->payload_offset == a.pay_off &&
                    h->payload_words <= a.max_words && h->prob_bits >= kMinProbBits &&
                    h->prob_bits <= kMaxProbBits;
    *flag_sh = ok ? 0u : (uint32_t)NZ_STATUS_BAD_HEADER;
    *pb_sh = h->prob_bits;
  }
}

// Nothing writes the flags or cum_sh after the barrier that follows table_scan, so
// every thread computes the same verdict.  Returns status bits (0 = go on).
__device__ __forceinline__ uint32_t table_verdict(const uint16_t *cum_sh, const uint32_t *flag_sh,
                                                  uint32_t &pb) {
  pb = flag_sh[1];
  uint32_t bad = flag_sh[0];
  if (pb < kMinProbBits || pb > kMaxProbBits || cum_sh[256] != (1u << (pb & 15)) || flag_sh[2])
    bad |= NZ_STATUS_BAD_HEADER;
  return bad;
}

// Decode table at `smem`: warps take symbols in turn; a symbol's slot range is a run
// of rows (all copies of a slot hold the same word).  The host sized the table for
// 2^12 slots x 2^(lut_shift-2) copies; with fewer probability bits the spare room
// becomes more copies.  The entries are narrow when all frequencies fit, the table has
// 2^usual_pb slots and bit row_shift of `narrow_rows` is set: the caller has a loop for that.
__device__ __forceinline__ void table_fill(uint32_t lut_shift, uint32_t S, uint32_t pb,
                                           uint8_t *smem, const uint16_t *cum_sh,
                                           uint32_t narrow_rows, uint32_t usual_pb,
                                           const uint32_t *flag_sh,
                                           uint32_t warp, uint32_t lane, uint32_t n_warps,
                                           LutView &lv, uint32_t &row_shift) {
  lv.pb = pb;
  lv.mask = (1u << pb) - 1u;
  row_shift = lut_shift + (kMaxProbBits - pb);              // log2 of the bytes per slot row
  if (row_shift > 7) row_shift = 7;                         // 32 copies are enough
  lv.stride = 1u << row_shift;
  lv.narrow = flag_sh[3] && pb == usual_pb && ((narrow_rows >> row_shift) & 1u);
  lv.base = smem_u32(smem) + ((lane << 2) & (lv.stride - 1u));
  lv.k64k = S ? 65536u : 0u;        // S is never 0; the compiler cannot know
  const uint32_t lut = smem_u32(smem);
  // A warp takes 32 slots at a time: lane l finds the symbol that owns slot s0 + l (the
  // largest symbol whose cumulative count is not above the slot; symbols that do not occur
  // share their successor's count and are skipped by "largest"), then the warp writes the
  // 32 rows with 16-byte stores.  The cost does not depend on how the counts are spread over
  // the symbols.  The searches (eight dependent lookups) of up to four turns run side by
  // side, so that a CTA of one or two warps is not held up by them.
  const uint32_t n_slots = 1u << pb;
  constexpr int kTurns = 4;
  for (uint32_t s0 = warp * 32; s0 < n_slots; s0 += kTurns * n_warps * 32) {
    uint32_t sym[kTurns], entry[kTurns];
#pragma unroll
    for (int i = 0; i < kTurns; ++i) sym[i] = 0;
#pragma unroll
    for (uint32_t step = 128; step >= 1; step >>= 1)
#pragma unroll
      for (int i = 0; i < kTurns; ++i)
        if (cum_sh[sym[i] + step] <= s0 + i * n_warps * 32 + lane) sym[i] += step;
#pragma unroll
    for (int i = 0; i < kTurns; ++i) {
      const uint32_t start = cum_sh[sym[i]];
      const uint32_t freq = cum_sh[sym[i] + 1] - start, off = s0 + i * n_warps * 32 + lane - start;
      entry[i] = lv.narrow ? (off << kNarrowOffShift) | (sym[i] << kNarrowSymShift) | freq
                           : (sym[i] << kEntSymShift) | (freq << kEntFreqShift) | off;
    }
#pragma unroll
    for (int i = 0; i < kTurns; ++i) {
      const uint32_t first = s0 + i * n_warps * 32;
      if (first >= n_slots) break;
      if (row_shift < 4) {
        // one or two copies (12-bit tables beside long units): the lane's own row
        const uint32_t row = lut + ((first + lane) << row_shift);
        for (uint32_t k = 0; k < (1u << row_shift); k += 4)
          asm volatile("st.shared.u32 [%0], %1;" ::"r"(row + k), "r"(entry[i]) : "memory");
        continue;
      }
      const uint32_t dst = lut + (first << row_shift) + lane * 16;
      if (row_shift == 7) {
        uint32_t v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = __shfl_sync(0xFFFFFFFFu, entry[i], 4 * k + (lane >> 3));
#pragma unroll
        for (int k = 0; k < 8; ++k)
          asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(dst + 512 * k), "r"(v[k])
                       : "memory");
        continue;
      }
      for (uint32_t k = 0; k < (1u << row_shift); k += 16) {
        // store k / 16 of the 2^row_shift / 16 covers bytes [32 k, 32 k + 512) of the 32 rows
        const uint32_t v = __shfl_sync(0xFFFFFFFFu, entry[i], (32 * k + lane * 16) >> row_shift);
        asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(dst + 32 * k), "r"(v) : "memory");
      }
    }
  }
}

}  // namespace nz
