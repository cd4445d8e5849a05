// rANS decoder of the NZR1 container, fused with the bf16 merge: the kernel and its launch.
// One translation unit per precision instantiates it (nz_decode_s*.cu); nz_decode.cu holds
// the host side.
//
// Replaces nvcomp's ANS decompress followed by kernel_aligned_merge in the
// reference's read path (cuda/high_level.cu:184-201, cuda/kernels.cuh:158-217):
// the decoded exponent bytes stay in registers and are merged with the packed
// fractions straight into the bf16 output, so the exponent stream never makes
// the round trip through HBM.
//
// Work decomposition.  One CTA per SM; a warp decodes a run of units, two side by side (32
// lane streams of S symbols each: independent rANS chains hide one another's latency), or one
// where every unit of the CTA can have a warp of its own.  The units' coded bytes are staged
// into the warp's shared-memory slots with bulk asynchronous copies (cp.async.bulk + mbarrier,
// no multicast); each lane then walks its own stream with a private read
// pointer, so a renormalisation costs one predicated 16-bit shared load and no
// warp-wide vote.  A lane produces 8 consecutive tensor elements per block and
// writes them with one 128-bit store; the warp's stores are 512 contiguous
// bytes.  The same kernel, instantiated differently, decodes a list of units
// (gather), feeds the decoded words to a dot product or applies an optimiser step to them.
//
// Decode table.  One 32-bit entry per slot, built once per CTA from the container's
// frequency table, in one of two layouts (see decode_step): narrow entries where the
// frequencies allow it, wide ones otherwise.  Random table lookups by 32 lanes would collide
// in the 32 shared-memory banks (3.5 wavefronts per lookup on average, which made the
// shared-memory pipe the limiter), so the table is replicated across banks as
// far as the shared memory left by the slots allows (64 KB for lossless
// tensors: 32 copies of a 2^9-slot table, one per bank; 16 of a 2^10-slot one).
//
// Robustness.  Header, offset table and lane lengths are validated before
// use; a malformed container sets bits in the caller's status word and the
// affected units are skipped.  Reads of the coded stream are confined to the
// CTA's shared memory (a guard band behind the last slot absorbs run-away
// pointers), output and fraction addresses never depend on coded data, and
// the wait on the bulk copy is bounded.
#pragma once

#include <cuda_bf16.h>
#include <string.h>

#include <mutex>
#include <type_traits>

#include "nz_decode_core.cuh"

namespace nz {

// One launch decodes up to kMaxBatch tensors; each tensor gets its own range of
// CTAs (one CTA per SM), sized in proportion to its unit count, so a small
// tensor does not leave most of the machine idle.
constexpr uint32_t kMaxBatch = 8;
constexpr int kDecodeMaxWarps = 20;                  // 96 registers a thread: more of them would spill
struct BatchItem {
  const uint8_t *container;
  const uint8_t *frac;
  uint64_t n;
  uint16_t *out_bf16;
  uint8_t *out_exp;
  uint32_t n_units;
  uint32_t cta_begin;     // first CTA of this tensor
  uint32_t tile_cols;     // operand order: row length (0 = stream order)
  uint32_t segs;          //   units per row group
  uint32_t S;             // lane symbols of this tensor
  uint32_t groups_each;   // groups of `chains` units per warp (one more for the first groups_more)
  uint32_t groups_more;
  uint32_t chains;        // units a warp decodes side by side: 2, or 1 when there are few
  uint32_t warps;         // warps of a CTA that decode (the others leave once the table is built)
  uint32_t bufs;          // staging buffers per warp, 1 or 2
  uint32_t slot_bytes;    // one unit's place in a buffer
  uint32_t ring_offset;   // byte offset of the fraction rings in shared memory
  uint32_t full_units;    // units of 32 * S elements
  uint32_t max_words;     // words of payload the container's buffer can hold (capped)
  const uint8_t *norm;    // block normaliser bytes (null = none), log2 of the group size
  uint32_t norm_lg;
};
struct BatchArgs {
  BatchItem item[kMaxBatch];
  const uint32_t *unit_list;   // gather launches (count == 1): units of item[0] to decode
  uint32_t n_list;
  const float *gx;             // matrix-vector launches (count == 1), see DecodeArgs
  float *partial;
  uint32_t in, seg;
  const uint16_t *grad;        // update launches (count == 1): gradient, AdamW moments (bf16)
  uint16_t *exp_avg, *exp_avg_sq;
  AdamArgs adam;
  uint32_t inputs_stable;      // containers and fractions were complete before the previous kernel
  uint32_t count;
  uint32_t n_ctas;        // == gridDim.x
  uint32_t lut_shift, lut_bytes;
  int canon;
  uint32_t *status;
};

// Exponent-only output: the 8 symbols of a lane's block as one 64-bit store.
template <int ROW>
__device__ __forceinline__ void store_exp_block(const uint32_t (&ent)[8], uint8_t *exp) {
  uint32_t b[8];                                          // symbol in the top byte
#pragma unroll
  for (int k = 0; k < 8; ++k) b[k] = ent[k] << (24 - (ROW > 0 ? kNarrowSymShift : kEntSymShift));
  const uint32_t lo = __byte_perm(__byte_perm(b[0], b[1], 0x0073),
                                  __byte_perm(b[2], b[3], 0x0073), 0x5410);
  const uint32_t hi = __byte_perm(__byte_perm(b[4], b[5], 0x0073),
                                  __byte_perm(b[6], b[7], 0x0073), 0x5410);
  __stcs(reinterpret_cast<uint2 *>(exp), make_uint2(lo, hi));
}

// Scales of the 8 elements from e (a multiple of 8): one stored byte for groups of 8 and
// more elements, else 8 >> lg of them.
__device__ __forceinline__ uint64_t norm_bytes(const uint8_t *norm, uint32_t lg, uint32_t e) {
  const uint8_t *p = norm + (e >> lg);
  uint64_t b = __ldg(p);
  if (lg < 3)
    for (int i = 1; i < (8 >> lg); ++i) b |= (uint64_t)__ldg(p + i) << (8 * i);
  return b;
}
__device__ __forceinline__ void norm_words(uint32_t (&w)[4], uint64_t bytes, uint32_t lg) {
  if (lg >= 3) {
    const float s = norm_scale((uint32_t)bytes);
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = scale_bf16_word(w[j], s, s);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      w[j] = scale_bf16_word(w[j], norm_scale((uint32_t)(bytes >> (8 * ((2 * j) >> lg))) & 0xFFu),
                             norm_scale((uint32_t)(bytes >> (8 * ((2 * j + 1) >> lg))) & 0xFFu));
  }
}

// Decode blocks b0 .. n_blocks - 1 of one unit for this lane (units decoded on their own).  ROW
// is kNarrowRow or 0, by the table's layout: looked up once per unit and not per symbol, which
// costs a sixth of the rate.  `e` is the lane's first element of the unit.  The packed fractions
// are fetched a block ahead of their use.
template <int S, bool MERGE, int ROW>
__device__ __forceinline__ void decode_blocks(const DecodeArgs &a, LaneState &st, const LutView &lut,
                                              uint32_t b0, uint32_t n_blocks, uint32_t e,
                                              uint16_t *out_lane, uint8_t *exp_lane, uint32_t adv,
                                              bool canon) {
  constexpr uint32_t kFracStride = 32u * (S + 1);  // bytes of fractions per 256 elements
  const uint8_t *frac_lane = MERGE ? a.frac + ((uint64_t)e * (S + 1) >> 3) + (uint64_t)b0 * kFracStride
                                   : nullptr;
  if (MERGE) out_lane += (uint64_t)b0 * adv; else exp_lane += b0 * 256;
  uint64_t next = (MERGE && b0 < n_blocks) ? load_frac<S>(frac_lane) : 0;
#pragma unroll 1
  for (uint32_t b = b0; b < n_blocks; ++b) {
    const uint64_t bits = next;
    if (MERGE && b + 1 < n_blocks) next = load_frac<S>(frac_lane += kFracStride);
    const uint64_t scales = MERGE && a.norm ? norm_bytes(a.norm, a.norm_lg, e + b * 256) : 0;
    uint32_t ent[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) ent[t] = decode_step<ROW>(st, lut);
    if (MERGE) {
      uint32_t w[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        w[t] = merge_word<S>(ent[2 * t], ent[2 * t + 1], bits, t);
        if (canon) w[t] = canon_word(w[t]);
      }
      if (a.norm) norm_words(w, scales, a.norm_lg);
      __stcs(reinterpret_cast<uint4 *>(out_lane), make_uint4(w[0], w[1], w[2], w[3]));
      out_lane += adv;
    } else {
      store_exp_block<0>(ent, exp_lane);
      exp_lane += 256;
    }
  }
}

// One element with all guards, used for the partial block at the very end of
// the tensor and for raw units.
// `delta` is the distance (in elements) from an element's place in the tensor
// to its place in the output: 0 except in gather launches.
template <int S, bool MERGE>
__device__ __forceinline__ void emit_guarded(uint32_t sym, uint64_t e, int64_t delta,
                                             const DecodeArgs &a) {
  if (e >= a.n) return;
  if (MERGE) {
    const uint64_t bit = e * (S + 1);
    const uint32_t shift = 7 - S - (uint32_t)(bit & 7);
    const uint32_t field = ((uint32_t)a.frac[bit >> 3] >> shift) & ((2u << S) - 1u);
    uint32_t v = merge_pair_generic<S>(sym << kEntSymShift, 0, field, 0, a.canon != 0) & 0xFFFFu;
    if (a.norm) v = scale_bf16_bits(v, norm_scale(a.norm[e >> a.norm_lg]));
    a.out_bf16[out_index(a, e) + delta] = (uint16_t)v;
  } else {
    a.out_exp[e + delta] = (uint8_t)sym;
  }
}

constexpr int kFastRow = 7;                      // 128-byte table rows: one copy per bank
// Where the four words (8 bf16) that a lane produces per block and chain go.
// StoreSink writes them to the output tensor.
// ADV = elements between a lane's consecutive blocks: 256, or 64 in operand order (a
// compile-time constant, so that the offsets fold into the store instructions).
template <int ADV>
struct StoreSinkT {
  uint16_t *out[kChains];
  __device__ __forceinline__ void begin(int) {}
  __device__ __forceinline__ void put(int c, int k, const uint32_t (&w)[4]) {
    __stcs(reinterpret_cast<uint4 *>(out[c] + k * ADV), make_uint4(w[0], w[1], w[2], w[3]));
  }
  __device__ __forceinline__ void advance(int blocks) {
#pragma unroll
    for (int c = 0; c < kChains; ++c) out[c] += blocks * ADV;
  }
};
using StoreSink = StoreSinkT<256>;

// One lane's running dot product of a weight row with the input vector.  The
// tensor is a row-major [out, in] matrix with `in` a multiple of 256, so the 256
// elements of a block lie in one row and the end of a row is the same event for
// all lanes of the warp.  At the end of a row (and of the unit) the warp's sum
// goes to the next partial-sum place of the unit; a finishing kernel adds the
// partial sums of each row in unit order, so results do not depend on timing.
struct DotLane {
  const float *x;      // input vector, fp32
  uint32_t in;         // row length
  uint32_t col;        // this lane's column of the next block (block start + lane * 8)
  float acc;
  float *part;         // next partial-sum place of the unit
  __device__ __forceinline__ void start(const float *xv, uint32_t in_features, uint64_t first_elem,
                                        float *unit_part, uint32_t lane) {
    x = xv;
    in = in_features;
    col = (uint32_t)(first_elem % in_features) + lane * 8;
    acc = 0.f;
    part = unit_part;
  }
  __device__ __forceinline__ void emit(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    if ((threadIdx.x & 31) == 0) *part = v;
    ++part;
  }
  // The 8 input values of a block are requested before the block's symbols are
  // decoded and used after, so that their latency hides behind the decode steps.
  float4 xa, xb;
  __device__ __forceinline__ void begin() {
    xa = __ldg(reinterpret_cast<const float4 *>(x + col));
    xb = __ldg(reinterpret_cast<const float4 *>(x + col + 4));
  }
  __device__ __forceinline__ void put(const uint32_t (&w)[4]) {
    float a = acc;
    a = fmaf(__uint_as_float(w[0] << 16), xa.x, a);
    a = fmaf(__uint_as_float(w[0] & 0xFFFF0000u), xa.y, a);
    a = fmaf(__uint_as_float(w[1] << 16), xa.z, a);
    a = fmaf(__uint_as_float(w[1] & 0xFFFF0000u), xa.w, a);
    a = fmaf(__uint_as_float(w[2] << 16), xb.x, a);
    a = fmaf(__uint_as_float(w[2] & 0xFFFF0000u), xb.y, a);
    a = fmaf(__uint_as_float(w[3] << 16), xb.z, a);
    a = fmaf(__uint_as_float(w[3] & 0xFFFF0000u), xb.w, a);
    acc = a;
    col += 256;
    if (col >= in) {          // same verdict in every lane: in - (col - lane*8) is a multiple of 256
      emit(acc);
      acc = 0.f;
      col -= in;
    }
  }
  // end of the unit: a row that is still open gives its partial sum
  __device__ __forceinline__ void finish() {
    if (col & ~255u) emit(acc);
  }
};
struct DotSink {
  DotLane lane[kChains];
  __device__ __forceinline__ void begin(int c) { lane[c].begin(); }
  __device__ __forceinline__ void put(int c, int, const uint32_t (&w)[4]) { lane[c].put(w); }
  __device__ __forceinline__ void advance(int) {}
};

// A sink in front of another: tensors written with a block normaliser are multiplied by
// their group's scale as they are produced (8 elements of a lane share one stored byte for
// groups of 8 and more, else each run of `group` elements has its own).
template <class Inner>
struct NormSink {
  Inner inner;
  const uint8_t *norm;
  uint32_t lg;
  uint32_t e0[kChains];       // tensor index of the lane's first element of the unit
  int blk[kChains];
  uint64_t bytes[kChains];
  __device__ __forceinline__ void begin(int c) {
    inner.begin(c);
    bytes[c] = norm_bytes(norm, lg, e0[c] + ((uint32_t)blk[c] << 8));
  }
  __device__ __forceinline__ void put(int c, int k, const uint32_t (&w)[4]) {
    uint32_t o[4] = {w[0], w[1], w[2], w[3]};
    norm_words(o, bytes[c], lg);
    inner.put(c, k, o);
    ++blk[c];
  }
  __device__ __forceinline__ void advance(int n) { inner.advance(n); }
};

// Update launches: the four decoded words of a block (8 weights of one row) take an
// AdamW step against the gradient and the moments at the same place of their (row-major)
// tensors and go, rounded to bf16 once, to the output tensor; the moments are updated in
// place.  Gradient and moments of a block are requested before its symbols are decoded.
__device__ __forceinline__ void adamw_words(const uint32_t (&w)[4], const uint4 &gv, uint4 &mv,
                                            uint4 &vv, const AdamArgs &a, uint4 &out) {
  const uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w};
  uint32_t mw[4] = {mv.x, mv.y, mv.z, mv.w}, vw[4] = {vv.x, vv.y, vv.z, vv.w}, ow[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    uint32_t res = 0, mres = 0, vres = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t sh = 16 * h;
      float m = __bfloat162float(__ushort_as_bfloat16((unsigned short)(mw[k] >> sh)));
      float v = __bfloat162float(__ushort_as_bfloat16((unsigned short)(vw[k] >> sh)));
      const float x = adamw_element(
          __bfloat162float(__ushort_as_bfloat16((unsigned short)(w[k] >> sh))),
          __bfloat162float(__ushort_as_bfloat16((unsigned short)(gw[k] >> sh))), m, v, a);
      res |= (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(x)) << sh;
      mres |= (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(m)) << sh;
      vres |= (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v)) << sh;
    }
    ow[k] = res;
    mw[k] = mres;
    vw[k] = vres;
  }
  out = make_uint4(ow[0], ow[1], ow[2], ow[3]);
  mv = make_uint4(mw[0], mw[1], mw[2], mw[3]);
  vv = make_uint4(vw[0], vw[1], vw[2], vw[3]);
}

template <int ADV>
struct UpdateSinkT {
  uint16_t *out[kChains];
  const uint16_t *g[kChains];
  uint16_t *m[kChains], *v[kChains];
  uint4 gv[kChains], mv[kChains], vv[kChains];
  int blk[kChains];
  AdamArgs adam;
  __device__ __forceinline__ void begin(int c) {
    const int o = blk[c] * ADV;
    gv[c] = __ldcs(reinterpret_cast<const uint4 *>(g[c] + o));
    mv[c] = __ldcs(reinterpret_cast<const uint4 *>(m[c] + o));
    vv[c] = __ldcs(reinterpret_cast<const uint4 *>(v[c] + o));
  }
  __device__ __forceinline__ void put(int c, int, const uint32_t (&w)[4]) {
    uint4 res;
    adamw_words(w, gv[c], mv[c], vv[c], adam, res);
    const int o = blk[c] * ADV;
    __stcs(reinterpret_cast<uint4 *>(out[c] + o), res);
    __stcs(reinterpret_cast<uint4 *>(m[c] + o), mv[c]);
    __stcs(reinterpret_cast<uint4 *>(v[c] + o), vv[c]);
    ++blk[c];
  }
  __device__ __forceinline__ void advance(int) {}
};

// Start the copies of a group's first packed fractions into the warp's ring.  They depend on
// nothing that is decoded, so the caller issues them before it waits for the coded units:
// the two latencies overlap.  `ring` carries the lane's offset in a block (8 or 4 bytes).
template <int S, int C>
__device__ __forceinline__ void group_async(uint32_t ring, const uint8_t *(&frac)[kChains],
                                            uint32_t g) {
  // s = 0 and 1: four blocks of a unit are 128 or 256 contiguous bytes, copied by the whole
  // warp (4 or 8 bytes per lane)
  constexpr uint32_t kLaneBytes = 4u * (S + 1);          // per lane and group
  constexpr uint32_t kGroupBytes = 32u * kLaneBytes;     // per unit and group
  constexpr uint32_t kRingUnitBytes = ring_unit_bytes(S);
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t dst = ring - lane * 4 + (g & 1) * (kChains * kRingUnitBytes) + lane * kLaneBytes;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const uint8_t *src = frac[c] - lane * (S + 1) + (uint64_t)g * kGroupBytes + lane * kLaneBytes;
    if (S == 1)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + c * kRingUnitBytes),
                   "l"(src)
                   : "memory");
    else
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + c * kRingUnitBytes),
                   "l"(src)
                   : "memory");
  }
  frac_commit();
}
template <int S, int C>
__device__ __forceinline__ void ring_prologue(uint32_t ring, const uint8_t *(&frac)[kChains],
                                              uint32_t n_blocks) {
  if (ring_by_block(S)) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if ((uint32_t)k < n_blocks) {
#pragma unroll
        for (int c = 0; c < C; ++c)
          frac_async<S>(ring + k * (kChains * ring_unit_bytes(S)) + c * ring_unit_bytes(S),
                        frac[c] + k * 32u * (S + 1));
      }
      frac_commit();
    }
  } else if (n_blocks >= 4) {
    group_async<S, C>(ring, frac, 0);
  }
}

// C units (1 or 2) interleaved in one lane: the rANS chains are independent, so
// each hides the shared-memory and multiply latency of the others.  For
// precisions 3 and 7 the packed fractions travel through a small ring in shared
// memory, fetched three blocks ahead with per-lane asynchronous copies; the
// narrower fractions of precisions 0 and 1 (1 and 2 bytes per lane and block)
// are fetched four blocks at a time by the whole warp.  The caller has started the
// first copies (ring_prologue); returns true when the next group's first copies are under
// way in their place.
//
// CANON: the tensor has NaN to rewrite (tables in the wide layout only); a template parameter,
// because the test at run time costs a fifth of the loop's rate (116 instead of 98 cycles a step
// in a lone warp).
template <int S, bool MERGE, int ROW, bool CANON, int C, typename Sink>
__device__ __forceinline__ bool decode_blocks_multi(LaneState (&st)[kChains], const LutView &lut,
                                                    uint32_t n_blocks,
                                                    const uint8_t *(&frac)[kChains],
                                                    const uint8_t *(&next_frac)[kChains], Sink &sink,
                                                    uint8_t *(&exp)[kChains], uint32_t ring) {
  constexpr uint32_t kFracStride = 32u * (S + 1);
  constexpr uint32_t kRingUnitBytes = ring_unit_bytes(S);
  constexpr uint32_t kRingSlotBytes = kChains * kRingUnitBytes;
  // Blocks per trip of the loop over the ring.  Two: the code of a trip (about 4 KB a block) is
  // fetched once per SM, which a call that decodes one group per warp pays for in full.
  constexpr int kTrip = 2;
  if (!MERGE) {
#pragma unroll 1
    for (uint32_t b = 0; b < n_blocks; ++b) {
      uint32_t e[kChains][8];
#pragma unroll
      for (int t = 0; t < 8; ++t)
#pragma unroll
        for (int c = 0; c < C; ++c) e[c][t] = decode_step<ROW, usual_prob_bits(S)>(st[c], lut);
#pragma unroll
      for (int c = 0; c < C; ++c) {
        store_exp_block<ROW>(e[c], exp[c]);
        exp[c] += 256;
      }
    }
    return false;
  }
  // One block of every unit with its packed fractions at hand: two symbols of each chain,
  // then their output words (the table entries do not stay live for the whole block).
  auto decode_block = [&](const uint64_t (&bits)[kChains], int k) {
#pragma unroll
    for (int c = 0; c < C; ++c) sink.begin(c);
    uint32_t w[kChains][4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      uint32_t e0[kChains], e1[kChains];
#pragma unroll
      for (int c = 0; c < C; ++c) e0[c] = decode_step<ROW, usual_prob_bits(S)>(st[c], lut);
#pragma unroll
      for (int c = 0; c < C; ++c) e1[c] = decode_step<ROW, usual_prob_bits(S)>(st[c], lut);
#pragma unroll
      for (int c = 0; c < C; ++c) {
        w[c][t] = merge_word<S, ROW>(e0[c], e1[c], bits[c], t);
        if (CANON) w[c][t] = canon_word(w[c][t]);
      }
    }
#pragma unroll
    for (int c = 0; c < C; ++c) sink.put(c, k, w[c]);
  };
  if (ring_by_block(S)) {
    auto ring_read = [&](uint32_t at, uint64_t (&bits)[kChains]) {
      frac_commit();
      frac_wait<3>();
#pragma unroll
      for (int c = 0; c < C; ++c)
        bits[c] = frac_from_ring<S>(ring + at + c * kRingUnitBytes);
    };
    // Block b starts the copy of block b + 3 into the ring slot that block b - 1 has left
    // (`fetch`: where that block's fractions are).  When the group fills the ring a whole
    // number of times, the copies go on after its last block with the first three of the next
    // group (next_frac, unless null), which finds them where ring_prologue would put them.
    const bool carry = n_blocks && n_blocks % kRingSlots == 0 && next_frac[0] != nullptr;
    uint32_t b = 0;
    const uint8_t *fetch[kChains];
#pragma unroll
    for (int c = 0; c < C; ++c) fetch[c] = frac[c] + 3 * kFracStride;
    const uint32_t fetch_end = carry ? ~0u : n_blocks;
    uint32_t half = 0;                       // byte offset of the trip's two ring slots
#pragma unroll 1
    for (; b + kTrip <= n_blocks; b += kTrip) {
      uint64_t bits[kChains];
      if (b + 3 < fetch_end) {
#pragma unroll
        for (int c = 0; c < C; ++c)
          frac_async<S>(ring + (half ^ (2 * kRingSlotBytes)) + kRingSlotBytes + c * kRingUnitBytes,
                        fetch[c]);
      }
      ring_read(half, bits);
      decode_block(bits, 0);
#pragma unroll
      for (int c = 0; c < C; ++c) {
        fetch[c] += kFracStride;
        if (carry && b + 4 == n_blocks) fetch[c] = next_frac[c];
      }
      if (b + 4 < fetch_end) {
#pragma unroll
        for (int c = 0; c < C; ++c)
          frac_async<S>(ring + half + c * kRingUnitBytes, fetch[c]);
      }
      ring_read(half + kRingSlotBytes, bits);
      decode_block(bits, 1);
#pragma unroll
      for (int c = 0; c < C; ++c) fetch[c] += kFracStride;
      half ^= 2 * kRingSlotBytes;
      sink.advance(kTrip);
    }
#pragma unroll 1
    for (; b < n_blocks; ++b) {
      if (b + 3 < n_blocks) {
#pragma unroll
        for (int c = 0; c < C; ++c)
          frac_async<S>(ring + ((b + 3) % kRingSlots) * kRingSlotBytes + c * kRingUnitBytes,
                        fetch[c]);
      }
      uint64_t bits[kChains];
      ring_read((b % kRingSlots) * kRingSlotBytes, bits);
      decode_block(bits, 0);
#pragma unroll
      for (int c = 0; c < C; ++c) fetch[c] += kFracStride;
      sink.advance(1);
    }
    return carry;
  }
  // Narrow fractions: a double-buffered ring filled one group of four blocks ahead; lanes
  // then read their own 1 or 2 bytes.  Only the one to three blocks behind the last whole group
  // (43 blocks a unit in matrices with 11008 columns) are loaded into registers: the chain's
  // lookups wait for such loads.
  const uint32_t lane_id = threadIdx.x & 31;
  const uint32_t ring0 = ring - lane_id * 4;               // `ring` carries lane*4 for s<7
  const uint32_t n_groups = n_blocks >> 2;
#pragma unroll 1
  for (uint32_t g = 0; g < n_groups; ++g) {
    __syncwarp();                         // everyone is done with the buffer about to be refilled
    if (g + 1 < n_groups) {
      group_async<S, C>(ring, frac, g + 1);
      frac_wait<1>();
    } else {
      frac_wait<0>();
    }
    __syncwarp();                         // all lanes' copies of group g have landed
    const uint32_t src = ring0 + (g & 1) * kRingSlotBytes + lane_id * (S + 1);
    // one block per trip: with two, the lone warp's step takes 119 instead of 85 cycles at
    // precision 0, and 115 instead of 87 at precision 1
#pragma unroll 1
    for (int at = 0; at < 4; ++at) {
      uint64_t bits[kChains];
#pragma unroll
      for (int c = 0; c < C; ++c)
        bits[c] = (S == 1) ? lds_u16(src + c * kRingUnitBytes + at * 64)
                           : lds_u8(src + c * kRingUnitBytes + at * 32);
      decode_block(bits, 0);
      sink.advance(1);
    }
  }
#pragma unroll 1
  for (uint32_t b = n_groups * 4; b < n_blocks; ++b) {
    uint64_t bits[kChains];
#pragma unroll
    for (int c = 0; c < C; ++c) bits[c] = load_frac<S>(frac[c] + b * kFracStride);
    decode_block(bits, 0);
    sink.advance(1);
  }
  return false;
}

// Decode what is left of a unit from block b0 on: its full blocks, then the partial block
// that ends the tensor.
template <int S, bool MERGE>
__device__ __forceinline__ void decode_rest(const DecodeArgs &a, LaneState &st, uint32_t u,
                                            uint32_t b0, int64_t delta, const LutView &lv, bool canon,
                                            uint32_t lane) {
  const uint32_t U = 32u * a.S, first = u * U, e_lane = first + lane * 8;
  const uint32_t count = u < a.full_units ? U : (uint32_t)a.n - first;
  const uint32_t full_blocks = count >> 8;
  // in operand order a lane's blocks are 64 elements apart in its row (units never
  // straddle a row group); the exponent-only output is always in stream order
  uint16_t *out_lane = MERGE ? a.out_bf16 + ((int64_t)unit_out_index(a, u, lane) + delta) : nullptr;
  uint8_t *exp_lane = MERGE ? nullptr : a.out_exp + ((int64_t)e_lane + delta);
  const uint32_t adv = (MERGE && a.tile_cols) ? 64u : 256u;
  if (lv.narrow)
    decode_blocks<S, MERGE, kNarrowRow>(a, st, lv, b0, full_blocks, e_lane, out_lane, exp_lane, adv, canon);
  else
    decode_blocks<S, MERGE, 0>(a, st, lv, b0, full_blocks, e_lane, out_lane, exp_lane, adv, canon);
  if (count == U) {
    if (__any_sync(0xFFFFFFFFu, st.x != kStateLow) && lane == 0)
      raise(a.status, NZ_STATUS_BAD_STATE);
  } else if (count & 255) {
    const uint64_t e0 = e_lane + (uint64_t)full_blocks * 256;
#pragma unroll 1
    for (int t = 0; t < 8; ++t) {
      const uint32_t ent = decode_step_any(st, lv);
      emit_guarded<S, MERGE>(entry_symbol(ent), e0 + t, delta, a);
    }
  }
}

// A raw unit: its exponent bytes are stored as they are, from any 16-bit word of the payload on.
// Block by block like a coded unit, bytes and fractions fetched a block ahead; what is left of
// a ragged one element by element.  (All of it element by element: 282 us for 11008 x 4096
// elements with raw rows; units next to one another, as those of a row are, meet in one warp.)
// A function of its own, given what it needs one by one, so that the registers and the code of
// the loops above stay as they are.  `e` is the unit's first element in the tensor, `out` where
// the lane's first element goes (bf16, or bytes without MERGE), `adv` the distance between its
// blocks.
template <int S, bool MERGE>
__device__ __noinline__ void emit_raw_unit(const uint8_t *src, const uint8_t *frac, void *out, uint32_t e,
                                           uint32_t count, uint32_t adv, bool canon,
                                           const uint8_t *norm, uint32_t norm_lg) {
  constexpr uint32_t kFracStride = 32u * (S + 1);
  const uint32_t lane = threadIdx.x & 31, full_blocks = count >> 8;
  uint16_t *out_lane = reinterpret_cast<uint16_t *>(out);
  uint8_t *exp_lane = reinterpret_cast<uint8_t *>(out);
  const uint16_t *raw = reinterpret_cast<const uint16_t *>(src) + lane * 4;
  const uint8_t *frac_lane = MERGE ? frac + ((uint64_t)(e + lane * 8) * (S + 1) >> 3) : nullptr;
  uint32_t lo = 0, hi = 0;
  uint64_t bits = 0;
  auto fetch = [&]() {
    lo = __ldg(raw) | ((uint32_t)__ldg(raw + 1) << 16);
    hi = __ldg(raw + 2) | ((uint32_t)__ldg(raw + 3) << 16);
    raw += 128;
    if (MERGE) {
      bits = load_frac<S>(frac_lane);
      frac_lane += kFracStride;
    }
  };
  if (full_blocks) fetch();
#pragma unroll 1
  for (uint32_t b = 0; b < full_blocks; ++b) {
    const uint32_t sym[2] = {lo, hi};
    const uint64_t now = bits;
    if (b + 1 < full_blocks) fetch();
    if (MERGE) {
      uint32_t w[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const uint32_t pair = sym[t >> 1] >> (16 * (t & 1));
        w[t] = merge_word<S>((pair & 0xFFu) << kEntSymShift, (pair << (kEntSymShift - 8)) & 0x7F800000u, now, t);
        if (canon) w[t] = canon_word(w[t]);
      }
      if (norm) norm_words(w, norm_bytes(norm, norm_lg, e + lane * 8 + b * 256), norm_lg);
      __stcs(reinterpret_cast<uint4 *>(out_lane), make_uint4(w[0], w[1], w[2], w[3]));
      out_lane += adv;
    } else {
      __stcs(reinterpret_cast<uint2 *>(exp_lane), make_uint2(sym[0], sym[1]));
      exp_lane += 256;
    }
  }
}

// Decode one unit on its own (raw units, odd counts).
template <int S, bool MERGE>
__device__ __forceinline__ void decode_single(const DecodeArgs &a, const UnitPlan &pl, uint32_t u,
                                              int64_t delta, uint32_t slot, const LutView &lv, bool canon,
                                              const uint8_t *payload, uint32_t lenq,
                                              uint32_t lane) {
  if (pl.kind == kUnitRaw) {
    const uint32_t U = 32u * a.S, first = u * U;
    const uint32_t count = u < a.full_units ? U : (uint32_t)a.n - first;
    const uint8_t *src = payload + pl.byte0();
    const int64_t o = (int64_t)unit_out_index(a, u, lane) + delta;      // (exponents: stream order)
    emit_raw_unit<S, MERGE>(src, a.frac, MERGE ? (void *)(a.out_bf16 + o) : (void *)(a.out_exp + o), first,
                            count, a.tile_cols ? 64u : 256u, a.canon != 0, a.norm, a.norm_lg);
#pragma unroll 1
    for (uint32_t i = (count & ~255u) + lane; i < count; i += 32)
      emit_guarded<S, MERGE>(src[i], (uint64_t)first + i, delta, a);
    return;
  }
  if (pl.kind != kUnitCoded) return;
  LaneState st;
  if (!open_unit(pl, slot, lenq, lane, st)) {
    if (lane == 0) raise(a.status, NZ_STATUS_BAD_LANES);
    return;
  }
  decode_rest<S, MERGE>(a, st, u, 0, delta, lv, canon, lane);
}

template <int ADV>
__device__ __forceinline__ void init_sink(StoreSinkT<ADV> &sk, int c, const DecodeArgs &a, uint32_t,
                                          uint64_t out_elem, uint32_t) {
  // out_elem is the place of the lane's first element of the unit in the output
  sk.out[c] = a.out_bf16 + out_elem;
}
__device__ __forceinline__ void init_sink(DotSink &sk, int c, const DecodeArgs &a, uint32_t unit,
                                          uint64_t, uint32_t lane) {
  sk.lane[c].start(a.gx, a.in, (uint64_t)unit * (32ull * a.S), a.partial + (uint64_t)unit * a.seg,
                   lane);
}
template <int ADV>
__device__ __forceinline__ void finish_sink(StoreSinkT<ADV> &) {}
template <int ADV>
__device__ __forceinline__ void init_sink(UpdateSinkT<ADV> &sk, int c, const DecodeArgs &a, uint32_t,
                                          uint64_t o, uint32_t) {
  sk.out[c] = a.out_bf16 + o;
  sk.g[c] = a.grad + o;
  sk.m[c] = a.exp_avg + o;
  sk.v[c] = a.exp_avg_sq + o;
  sk.blk[c] = 0;
  sk.adam = a.adam;
}
template <int ADV>
__device__ __forceinline__ void finish_sink(UpdateSinkT<ADV> &) {}
template <class Inner>
__device__ __forceinline__ void init_sink(NormSink<Inner> &sk, int c, const DecodeArgs &a,
                                          uint32_t unit, uint64_t out_elem, uint32_t lane) {
  init_sink(sk.inner, c, a, unit, out_elem, lane);
  sk.norm = a.norm;
  sk.lg = a.norm_lg;
  sk.e0[c] = unit * (32u * a.S) + lane * 8;
  sk.blk[c] = 0;
}
template <class Inner>
__device__ __forceinline__ void finish_sink(NormSink<Inner> &sk) { finish_sink(sk.inner); }

// Update launches, units that do not take the fast path: the unit has just been decoded
// into the output tensor the ordinary way; its elements take their step there.
__device__ __forceinline__ void update_decoded_unit(const DecodeArgs &a, uint32_t u, uint32_t lane) {
  if (u >= a.n_units) return;
  const uint64_t U = 32ull * a.S;
  const uint64_t first = (uint64_t)u * U;
  const uint64_t count = (a.n - first < U) ? (a.n - first) : U;
  __syncwarp();
  for (uint64_t i = lane; i < count; i += 32) {
    const uint64_t o = out_index(a, first + i);
    float m = __bfloat162float(__ushort_as_bfloat16(a.exp_avg[o]));
    float v = __bfloat162float(__ushort_as_bfloat16(a.exp_avg_sq[o]));
    const float x = adamw_element(__bfloat162float(__ushort_as_bfloat16(a.out_bf16[o])),
                                  __bfloat162float(__ushort_as_bfloat16(a.grad[o])), m, v, a.adam);
    a.out_bf16[o] = __bfloat16_as_ushort(__float2bfloat16_rn(x));
    a.exp_avg[o] = __bfloat16_as_ushort(__float2bfloat16_rn(m));
    a.exp_avg_sq[o] = __bfloat16_as_ushort(__float2bfloat16_rn(v));
  }
}
__device__ __forceinline__ void finish_sink(DotSink &sk) {
#pragma unroll
  for (int c = 0; c < kChains; ++c) sk.lane[c].finish();
}

// Matrix-vector launches, units that do not take the fast path (raw units, the
// tensor's last unit, units whose neighbour in the group is one of those).  The
// partial sums of unit u go to partial[u * seg ...], one per row the unit
// touches, in row order -- the same places the fast path fills.
template <int S>
__device__ __forceinline__ void dot_single(const DecodeArgs &a, const UnitPlan &pl, uint32_t u,
                                           uint32_t slot, const LutView &lv, bool canon,
                                           const uint8_t *payload, uint32_t lenq, uint32_t lane) {
  if (u >= a.n_units) return;
  const uint64_t U = 32ull * a.S;
  const uint64_t first = (uint64_t)u * U;
  const uint64_t count = (a.n - first < U) ? (a.n - first) : U;
  float *part = a.partial + (uint64_t)u * a.seg;
  const uint64_t row0 = first / a.in, row1 = (first + count - 1) / a.in;
  bool filled = false;
  if (pl.kind == kUnitRaw) {
    const uint8_t *src = payload + pl.byte0();
    for (uint64_t r = row0; r <= row1; ++r) {
      const uint64_t lo = r * a.in > first ? r * a.in : first;
      const uint64_t hi = (r + 1) * a.in < first + count ? (r + 1) * a.in : first + count;
      float acc = 0.f;
      for (uint64_t e = lo + lane; e < hi; e += 32) {
        const uint64_t bit = e * (S + 1);
        const uint32_t shift = 7 - S - (uint32_t)(bit & 7);
        const uint32_t field = ((uint32_t)a.frac[bit >> 3] >> shift) & ((2u << S) - 1u);
        const uint32_t v = merge_pair_generic<S>((uint32_t)src[e - first] << kEntSymShift, 0, field,
                                                 0, a.canon != 0);
        acc = fmaf(__uint_as_float(v << 16), a.gx[e - r * a.in], acc);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
      if (lane == 0) part[r - row0] = acc;
    }
    filled = true;
  } else if (pl.kind == kUnitCoded) {
    LaneState st;
    if (open_unit(pl, slot, lenq, lane, st)) {
      // the row length is a multiple of 256, so is the element count: whole blocks only
      const uint32_t n_blocks = (uint32_t)(count / 256);
      const uint8_t *frac_lane = a.frac + (first + lane * 8) * (S + 1) / 8;
      DotLane d;
      d.start(a.gx, a.in, first, part, lane);
      auto blocks = [&](auto row) {
        uint64_t next = load_frac<S>(frac_lane);
#pragma unroll 1
        for (uint32_t b = 0; b < n_blocks; ++b) {
          const uint64_t fbits = next;
          if (b + 1 < n_blocks) next = load_frac<S>(frac_lane += 32u * (S + 1));
          uint32_t ent[8], w[4];
          d.begin();
#pragma unroll
          for (int t = 0; t < 8; ++t) ent[t] = decode_step<decltype(row)::value>(st, lv);
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            w[t] = merge_word<S>(ent[2 * t], ent[2 * t + 1], fbits, t);
            if (canon) w[t] = canon_word(w[t]);
          }
          d.put(w);
        }
      };
      if (lv.narrow) blocks(std::integral_constant<int, kNarrowRow>());
      else blocks(std::integral_constant<int, 0>());
      d.finish();
      if (count == U && __any_sync(0xFFFFFFFFu, st.x != kStateLow) && lane == 0)
        raise(a.status, NZ_STATUS_BAD_STATE);
      filled = true;
    } else if (lane == 0) {
      raise(a.status, NZ_STATUS_BAD_LANES);
    }
  }
  if (!filled && lane == 0)          // a unit that could not be decoded contributes zeros
    for (uint64_t r = row0; r <= row1; ++r) part[r - row0] = 0.f;
}

// MODE kModeList: gather launch -- the launch decodes the units named in
// batch.unit_list (of the single tensor item[0]) and writes them one after the other.
// MODE kModeDot: matrix-vector launch -- nothing is written back; every unit's
// elements are multiplied with the input vector as they are decoded.
constexpr int kModeTensor = 0, kModeList = 1, kModeDot = 2, kModeUpdate = 3;
constexpr int kUpdateMaxWarps = 16;                 // the update's operands want registers
constexpr int kDotMaxWarps = kDecodeMaxWarps;   // 16 warps and 128 registers measured slower
template <int S, bool MERGE, int MODE>
__global__ void __launch_bounds__((MODE == kModeDot ? kDotMaxWarps : MODE == kModeUpdate ? kUpdateMaxWarps : kDecodeMaxWarps) * 32, 1)
decode_kernel(const BatchArgs batch) {
  constexpr bool LIST = MODE == kModeList;
  constexpr bool DOT = MODE == kModeDot;
  constexpr bool UPDATE = MODE == kModeUpdate;
  extern __shared__ __align__(128) uint8_t smem[];
  // which tensor this CTA works on, and its rank among that tensor's CTAs
  uint32_t ti = 0;
#pragma unroll
  for (uint32_t t = 1; t < kMaxBatch; ++t)
    if (t < batch.count && blockIdx.x >= batch.item[t].cta_begin) ti = t;
  const uint32_t cta_first = batch.item[ti].cta_begin;
  const uint32_t cta_end = (ti + 1 < batch.count) ? batch.item[ti + 1].cta_begin : batch.n_ctas;
  const uint32_t cta_rank = blockIdx.x - cta_first, cta_count = cta_end - cta_first;
  DecodeArgs a;
  a.container = batch.item[ti].container;
  a.frac = batch.item[ti].frac;
  a.n = batch.item[ti].n;
  a.S = batch.item[ti].S;
  a.n_units = batch.item[ti].n_units;
  a.full_units = batch.item[ti].full_units;
  a.pay_off = payload_offset(a.n_units);
  a.max_words = batch.item[ti].max_words;
  a.slot_bytes = batch.item[ti].slot_bytes;
  a.lut_shift = batch.lut_shift;
  a.lut_bytes = batch.lut_bytes;
  a.canon = batch.canon;
  a.out_bf16 = batch.item[ti].out_bf16;
  a.out_exp = batch.item[ti].out_exp;
  a.status = batch.status;
  a.unit_list = LIST ? batch.unit_list : nullptr;
  a.n_work = LIST ? batch.n_list : a.n_units;
  a.gx = DOT ? batch.gx : nullptr;
  a.partial = DOT ? batch.partial : nullptr;
  a.in = DOT ? batch.in : 0;
  a.seg = DOT ? batch.seg : 0;
  a.tile_cols = ((MODE == kModeTensor || UPDATE) && MERGE) ? batch.item[ti].tile_cols : 0;
  a.segs = batch.item[ti].segs;
  a.norm = (MERGE && (MODE == kModeTensor || LIST)) ? batch.item[ti].norm : nullptr;
  a.norm_lg = batch.item[ti].norm_lg;
  a.grad = UPDATE ? batch.grad : nullptr;
  a.exp_avg = UPDATE ? batch.exp_avg : nullptr;
  a.exp_avg_sq = UPDATE ? batch.exp_avg_sq : nullptr;
  if (UPDATE) a.adam = batch.adam;
  const uint32_t all_warps = blockDim.x >> 5;
  const uint32_t n_warps = batch.item[ti].warps, bufs = batch.item[ti].bufs;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + a.lut_bytes);
  uint16_t *cum_sh = reinterpret_cast<uint16_t *>(smem + a.lut_bytes + 8 * 32);  // 257 entries
  uint32_t *flag_sh = reinterpret_cast<uint32_t *>(smem + a.lut_bytes + 8 * 32 + 520);  // 4 words
  uint8_t *slots = smem + a.lut_bytes + 1024;
  const uint32_t bar = smem_u32(&bars[warp]);
  const uint32_t chains = (DOT || UPDATE) ? kChains : batch.item[ti].chains;
  const uint32_t buf_bytes = chains * a.slot_bytes;
  const uint32_t slot0 = smem_u32(slots) + warp * bufs * buf_bytes;
  // per-warp ring for the packed fractions, behind all slots and their guard band
  const uint32_t ring =
      smem_u32(smem) + batch.item[ti].ring_offset + warp * ring_warp_bytes(S) + lane * (S == 7 ? 8 : 4);

  // Each warp owns one mbarrier; its lane 0 initialises it and is the only
  // thread that ever arms it.
  if (lane == 0) {
    mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncwarp();
  // Programmatic dependent launch: let the next kernel of the stream start its
  // own launch now, and do not touch global memory before the previous kernel
  // of the stream has completed.  When the caller vouches that the compressed
  // inputs were complete before that kernel was launched, only the outputs (and
  // the input vector of a matrix-vector launch) depend on it: the wait then
  // moves behind the table build, which overlaps the previous kernel's tail.
  // Both instructions are no-ops for an ordinary launch.
  const bool early = MODE != kModeList && batch.inputs_stable != 0;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (!early) asm volatile("griddepcontrol.wait;" ::: "memory");

  // ---- this warp's share: a run of consecutive work items (units, or entries of the list)
  const Header *h = reinterpret_cast<const Header *>(a.container);
  const uint4 freqs = table_prefetch(a, warp, lane);
  const uint8_t *payload = a.container + a.pay_off;
  const uint32_t U = 32u * a.S;
  const uint32_t n_blocks = a.S >> 3;
  uint32_t it, it_end;         // items left, in groups of `chains`
  {
    // groups_each for every warp and one more for the first groups_more of them, counted
    // across the CTAs first, so that every CTA gets its part of the longer runs
    const uint32_t me = warp * cta_count + cta_rank;
    const uint32_t each = batch.item[ti].groups_each, more = batch.item[ti].groups_more;
    it = chains * (each * me + (me < more ? me : more));
    it_end = it + chains * (each + (me < more ? 1u : 0u));
    if (it_end > a.n_work) it_end = a.n_work;
    if (warp >= n_warps) it = it_end = 0;
  }
  // A window of 32 items, one per lane: what the lane found out about its item.  Planning is
  // done for 32 units at once; a group takes its two from the window with a few shuffles.
  UnitPlan mine;
  uint32_t my_unit, my_out;
  uint32_t coded_mask, win;    // items of the window that are coded units; its first item
  auto load_window = [&](uint32_t first) {
    win = first;
    my_unit = first + lane < it_end ? first + lane : a.n_units;
    if (LIST && first + lane < it_end) {
      my_unit = __ldg(a.unit_list + first + lane);
      if (my_unit >= a.n_units) {
        raise(a.status, NZ_STATUS_BAD_UNIT);
        my_unit = a.n_units;
      }
    }
    uint32_t off0, off1;
    unit_offsets(a, my_unit, off0, off1);
    my_out = (MERGE && my_unit < a.n_units) ? unit_out_index(a, my_unit, 0) : 0u;
    mine = plan_unit(a, my_unit, off0, off1, 0);
    coded_mask = __ballot_sync(0xFFFFFFFFu, mine.kind == kUnitCoded);
  };
  // The units of group `at` (its first item) and their plans.
  auto take_group = [&](uint32_t at, uint32_t (&unit)[kChains], UnitPlan (&pl)[kChains]) {
    if (at - win >= 32) load_window(at);
#pragma unroll
    for (int c = 0; c < kChains; ++c) {
      if (c && chains == 1) {
        unit[c] = a.n_units;
        pl[c].kind = kUnitSkip;
        pl[c].word0 = pl[c].words = pl[c].copy_bytes = 0;
        continue;
      }
      const int k = (int)(at - win) + c;         // below 32: windows hold whole groups
      unit[c] = LIST ? __shfl_sync(0xFFFFFFFFu, my_unit, k) : (at + c < it_end ? at + c : a.n_units);
      pl[c].word0 = __shfl_sync(0xFFFFFFFFu, mine.word0, k);
      pl[c].words = __shfl_sync(0xFFFFFFFFu, mine.words, k);
      pl[c].copy_bytes = __shfl_sync(0xFFFFFFFFu, mine.copy_bytes, k);
      pl[c].kind = pl[c].copy_bytes ? kUnitCoded
                                    : (coded_mask == 0xFFFFFFFFu ? kUnitSkip
                                                                 : __shfl_sync(0xFFFFFFFFu, mine.kind, k));
    }
  };
  uint32_t parity = 0, buf = 0;
  UnitPlan pl[kChains];
  uint32_t real[kChains];      // the units behind work items it .. it+kChains-1
  bool staged = false;
  if (it < it_end) {
    load_window(it);
    take_group(it, real, pl);
    staged = stage_units(a, pl, slot0, bar, lane);
  }

  // ---- build the decode table while the first units arrive
  table_scan(a, h, freqs, cum_sh, flag_sh, warp, lane, all_warps);
  __syncthreads();
  uint32_t pb;
  const uint32_t bad = table_verdict(cum_sh, flag_sh, pb);
  if (bad) {
    // Every exit path orders itself behind the previous kernel of the stream first: the
    // status word is shared with it, and a kernel that retired without waiting would let
    // the next programmatically serialised launch overtake that kernel's reads.
    if (early) asm volatile("griddepcontrol.wait;" ::: "memory");
    // copies may be in flight into this warp's slots: let them land before leaving
    if (staged) wait_staged(bar, parity);
    if (threadIdx.x == 0 && cta_rank == 0) raise(a.status, bad);
    return;
  }
  LutView lv;
  uint32_t row_shift;
  const bool canon = MERGE && a.canon && (cum_sh[256] != cum_sh[255]);
  // Row sizes that have a loop for narrow entries: 32 copies of the table, one per bank, and
  // for the lossy precisions, whose tables have twice the slots, also 16.  Tensors with NaN
  // to rewrite take the wide loop.
  const uint32_t narrow_rows = canon ? 0u : (1u << kFastRow) | (S != 7 ? 1u << (kFastRow - 1) : 0u);
  table_fill(a.lut_shift, a.S, pb, smem, cum_sh, narrow_rows, usual_prob_bits(S), flag_sh, warp, lane,
             all_warps, lv, row_shift);
  __syncthreads();
  if (early) asm volatile("griddepcontrol.wait;" ::: "memory");

  // ---- units, kChains at a time
  const uint32_t lenq = len_quantum(a.S);
  auto frac_of = [&](uint32_t unit) {
    return a.frac + (((uint64_t)unit * U + lane * 8) * (S + 1) >> 3);
  };
  bool primed = false;         // the ring holds (or is receiving) the group's first fractions
  while (it < it_end) {
    // Both units (the one unit) coded: decoded side by side as far as both have full blocks
    // (all of them, but for the tensor's last unit).  Matrix-vector and update launches only
    // take whole units this way.
    bool pair = true;
    uint32_t common = n_blocks;
#pragma unroll
    for (int c = 0; c < kChains; ++c) {
      if (c && chains == 1) continue;
      pair = pair && pl[c].kind == kUnitCoded;
      if (real[c] >= a.full_units) {
        if (DOT || UPDATE || real[c] >= a.n_units) pair = false;
        else common = ((uint32_t)a.n - real[c] * U) >> 8;
      }
    }
    if (common == 0) pair = false;
    const uint8_t *fr[kChains];
#pragma unroll
    for (int c = 0; c < kChains; ++c) fr[c] = MERGE ? frac_of(real[c]) : nullptr;
    if (MERGE) {
      if (pair && !primed) {
        if (chains == 1) ring_prologue<S, 1>(ring, fr, common);
        else ring_prologue<S, kChains>(ring, fr, common);
      } else if (!pair && primed) {
        frac_wait<0>();
      }
      primed = false;
    }
    if (staged) {
      const bool arrived = wait_staged(bar, parity);
      parity ^= 1;
      if (!__all_sync(0xFFFFFFFFu, arrived)) {
        // The copies may still be in flight, so the slots cannot be reused: flag it,
        // give them one more bounded chance to land and leave.
        if (lane == 0) raise(a.status, NZ_STATUS_TIMEOUT);
        if (!arrived) wait_staged(bar, parity ^ 1);
        frac_wait<0>();
        return;
      }
    }
    const uint32_t slot = slot0 + buf * buf_bytes;
    LaneState st[kChains];
    if (pair && !(chains == 1 ? open_unit(pl[0], slot, lenq, lane, st[0])
                              : open_pair(pl, slot, a.slot_bytes, lenq, lane, st))) {
      pair = false;
      frac_wait<0>();          // the ring is used again
    }
    uint32_t out0[kChains];    // output element of the units' first elements
#pragma unroll
    for (int c = 0; c < kChains; ++c)      // (with one chain the second is not used)
      out0[c] = a.tile_cols ? __shfl_sync(0xFFFFFFFFu, my_out, ((int)(it - win) + c) & 31) : real[c] * U;

    // The next group: copied into the other buffer now, where there is one (the whole group
    // then hides the latency of its copies), else brought into L2 and copied at the end.
    uint32_t nreal[kChains] = {a.n_units, a.n_units};
    UnitPlan npl[kChains];
    const bool more = it + chains < it_end;
    if (more) {
      take_group(it + chains, nreal, npl);
      if (bufs > 1) {
        staged = stage_units(a, npl, slot0 + (buf ^ 1) * buf_bytes, bar, lane);
      } else if (lane == 0) {
#pragma unroll
        for (int c = 0; c < kChains; ++c)
          if (npl[c].copy_bytes)
            bulk_prefetch_l2(payload + (uint64_t)(npl[c].word0 & ~7u) * 2, npl[c].copy_bytes);
      }
    }
    if (pair) {
      uint8_t *xb[kChains];
      const uint8_t *nfr[kChains] = {nullptr, nullptr};
      if (MERGE && more && npl[0].copy_bytes && (chains == 1 || npl[1].copy_bytes) &&
          common == n_blocks && nreal[0] < a.full_units && (chains == 1 || nreal[1] < a.full_units)) {
#pragma unroll
        for (int c = 0; c < kChains; ++c) nfr[c] = frac_of(nreal[c]);
      }
      auto run = [&](auto &sink) {
#pragma unroll
        for (int c = 0; c < kChains; ++c) {
          // place of the lane's first element: in a gather launch by work item
          const uint64_t o = LIST ? (uint64_t)(it + c) * U + lane * 8
                                  : (uint64_t)(out0[c] + (a.tile_cols ? (lane >> 3) * a.tile_cols + (lane & 7u) * 8
                                                                      : lane * 8));
          xb[c] = MERGE ? nullptr : a.out_exp + o;
          init_sink(sink, c, a, real[c], o, lane);
        }
        auto with = [&](auto cc) {
          constexpr int C = decltype(cc)::value;
#define NZ_LOOP(ROW, CANON) decode_blocks_multi<S, MERGE, ROW, CANON, C>(st, lv, common, fr, nfr, sink, xb, ring)
          if (lv.narrow && row_shift == kFastRow) primed = NZ_LOOP(kFastRow, false);
          else if (S != 7 && lv.narrow) primed = NZ_LOOP(kFastRow - 1, false);     // see narrow_rows
          else if (MERGE && canon) primed = NZ_LOOP(0, true);
          else primed = NZ_LOOP(0, false);
#undef NZ_LOOP
        };
        if (DOT || UPDATE || chains == kChains) with(std::integral_constant<int, kChains>());
        else with(std::integral_constant<int, 1>());
        finish_sink(sink);
      };
      if (DOT) {
        typename std::conditional<DOT, DotSink, StoreSink>::type sink;
        run(sink);
      } else if (UPDATE) {
        if (a.tile_cols) {
          typename std::conditional<UPDATE, UpdateSinkT<64>, StoreSink>::type sink;
          run(sink);
        } else {
          typename std::conditional<UPDATE, UpdateSinkT<256>, StoreSink>::type sink;
          run(sink);
        }
      } else if (MODE == kModeTensor && MERGE && a.tile_cols) {
        typename std::conditional<DOT, DotSink, StoreSinkT<64>>::type sink;     // operand order
        run(sink);
      } else if (MERGE && !UPDATE && a.norm) {
        typename std::conditional<DOT || UPDATE || !MERGE, StoreSink, NormSink<StoreSink>>::type sink;
        run(sink);
      } else {
        typename std::conditional<DOT, DotSink, StoreSink>::type sink;
        run(sink);
      }
      if (common == n_blocks) {
        bool low = st[0].x == kStateLow;
        if (chains > 1) low = low && st[kChains - 1].x == kStateLow;
        if (__any_sync(0xFFFFFFFFu, !low) && lane == 0) raise(a.status, NZ_STATUS_BAD_STATE);
      } else if (!DOT && !UPDATE) {
#pragma unroll 1
        for (uint32_t c = 0; c < chains; ++c) {
          const int64_t delta = LIST ? ((int64_t)(it + c) - (int64_t)(c ? real[1] : real[0])) * (int64_t)U : 0;
          LaneState one = c ? st[1] : st[0];
          decode_rest<S, MERGE>(a, one, c ? real[1] : real[0], common, delta, lv, canon, lane);
        }
      }
    } else {
#pragma unroll 1
      for (uint32_t c = 0; c < chains; ++c) {
        const uint32_t u = c ? real[1] : real[0];
        const UnitPlan p = c ? pl[1] : pl[0];
        if (DOT) {
          dot_single<S>(a, p, u, slot + c * a.slot_bytes, lv, canon, payload, lenq, lane);
        } else {
          const int64_t delta = LIST ? ((int64_t)(it + c) - (int64_t)u) * (int64_t)U : 0;
          decode_single<S, MERGE>(a, p, u, delta, slot + c * a.slot_bytes, lv, canon, payload, lenq,
                                  lane);
          if (UPDATE) update_decoded_unit(a, u, lane);
        }
      }
    }
    // every lane is done reading the slots
    __syncwarp();
    it += chains;
    if (it < it_end) {
      take_group(it, real, pl);
      if (bufs > 1) buf ^= 1;
      else staged = stage_units(a, pl, slot0, bar, lane);
    }
  }
}

template <int S, bool MERGE, int MODE = kModeTensor>
static int launch_decode(const BatchArgs &b, uint32_t warps, uint32_t smem_bytes, cudaStream_t st) {
  auto kern = decode_kernel<S, MERGE, MODE>;
  // The opt-in to large dynamic shared memory is per kernel and device.  It is made once
  // per (instantiation, device), for the most a CTA can have, under a lock: concurrent
  // callers can then never leave the attribute below what a launch needs.
  {
    static std::mutex mu;
    static bool opted[kMaxDeviceOrdinals] = {};
    int dev = 0;
    NZ_CUDA_TRY(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    if (dev < 0 || dev >= kMaxDeviceOrdinals || !opted[dev]) {
      NZ_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kMaxDynamicSmem));
      if (dev >= 0 && dev < kMaxDeviceOrdinals) opted[dev] = true;
    }
  }
  // Programmatic stream serialisation: this launch may begin while the previous
  // kernel of the stream drains; the kernel itself waits (griddepcontrol.wait)
  // before it reads or writes global memory, so ordering is preserved.
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(b.n_ctas);
  cfg.blockDim = dim3(warps * 32);
  cfg.dynamicSmemBytes = smem_bytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  NZ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, b));
  return NZ_OK;
}

// The launch of one precision, for every mode; each precision is a translation unit of its own.
template <int S>
int launch_decode_precision(int mode, const BatchArgs &b, uint32_t warps, uint32_t smem_bytes,
                            cudaStream_t st) {
  switch (mode) {
    case kModeList: return launch_decode<S, true, kModeList>(b, warps, smem_bytes, st);
    case kModeUpdate: return launch_decode<S, true, kModeUpdate>(b, warps, smem_bytes, st);
    case kModeDot: return launch_decode<S, true, kModeDot>(b, warps, smem_bytes, st);
    default: return launch_decode<S, true>(b, warps, smem_bytes, st);
  }
}
// Exponent bytes only.
int launch_decode_exponents(const BatchArgs &b, uint32_t warps, uint32_t smem_bytes, cudaStream_t st);
extern template int launch_decode_precision<0>(int, const BatchArgs &, uint32_t, uint32_t, cudaStream_t);
extern template int launch_decode_precision<1>(int, const BatchArgs &, uint32_t, uint32_t, cudaStream_t);
extern template int launch_decode_precision<3>(int, const BatchArgs &, uint32_t, uint32_t, cudaStream_t);
extern template int launch_decode_precision<7>(int, const BatchArgs &, uint32_t, uint32_t, cudaStream_t);

}  // namespace nz
