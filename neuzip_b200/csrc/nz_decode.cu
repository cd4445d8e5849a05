// Host side of the decoder (nz_decode_kernel.cuh): launch geometry, batching, argument
// checks, the row gather around it and the C entry points.
#include <string.h>

#include "nz_decode_kernel.cuh"

namespace nz {

// Adds the partial sums of each output row in unit order, adds the bias and
// rounds to bf16 (round to nearest even, like the library GEMM's epilogue).
__global__ void dot_finish_kernel(const float *__restrict__ partial, uint32_t seg, uint64_t U,
                                  uint32_t in, uint32_t out_features,
                                  const uint16_t *__restrict__ bias, uint16_t *__restrict__ y) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= out_features) return;
  const uint64_t e_lo = (uint64_t)r * in, e_hi = e_lo + in - 1;
  float sum = 0.f;
  for (uint64_t u = e_lo / U; u <= e_hi / U; ++u)
    sum += partial[u * seg + (r - (uint32_t)(u * U / in))];
  if (bias) sum += __uint_as_float((uint32_t)bias[r] << 16);
  uint32_t bits = __float_as_uint(sum);
  if ((bits & 0x7F800000u) == 0x7F800000u && (bits & 0x007FFFFFu))
    bits = 0x7FFF0000u;                                  // NaN
  else
    bits += 0x7FFFu + ((bits >> 16) & 1u);               // round to nearest even
  y[r] = (uint16_t)(bits >> 16);
}

// ------------------------------------------------------------------- host
struct HostItem {
  const void *container;
  uint64_t container_bytes;
  const void *frac;
  uint64_t n;
  uint32_t max_unit_words;
  void *out_bf16;
  void *out_exp;
  const uint32_t *unit_list;   // gather: device array of unit numbers (else null)
  uint32_t n_list;
  const float *gx;             // matrix-vector: input vector (else null), partial sums,
  float *partial;              //   row length and partial-sum places per unit
  uint32_t in, seg;
  uint32_t flags;              // NZ_ITEM_* of the C interface
  uint32_t tile_cols;          // operand order: row length of the matrix (0 = stream order)
  uint32_t S;                  // lane symbols of this tensor
  const uint16_t *grad;        // update: gradient and AdamW moments (bf16, else null)
  uint16_t *exp_avg, *exp_avg_sq;
  AdamArgs adam;
  const uint8_t *norm;         // block normaliser bytes (else null) and log2 of the group size
  uint32_t norm_lg;
};

// Units a launch decodes for an item (a tensor has fewer than 2^24).
static inline uint32_t work_units(const HostItem &it) {
  return it.unit_list ? it.n_list : (uint32_t)unit_count(it.n, it.S);
}

// Cycles per symbol step of a CTA with `w` warps of `chains` units each, as measured on a B200
// (units of 256 to 512 symbols, one warp to twenty): the latency of the dependent chains while
// a scheduler has one warp or two, then what the schedulers' integer pipes need.  Without a
// loop for narrow rows (`narrow` false) a step has one instruction more and a longer chain, and
// beside the smallest table (`smallest`) more of its lookups meet in a bank.  The merge of
// precisions 0 and 1 is the cheapest.
static uint32_t step_cycles(uint32_t w, uint32_t chains, bool narrow, bool smallest, int precision) {
  uint32_t t;
  if (chains == 1) {
    t = (narrow ? 65 : 75) + (w > 8 ? 5 * (w - 8) : 0);
  } else if (w <= 4) {
    t = narrow ? 90 : 98;
  } else {
    const uint32_t slope10 = precision < 3 ? 84 : narrow ? 95 : 104;
    t = (narrow || precision < 3 ? 111 : 119) + (w > 8 ? slope10 * (w - 8) / 10 : 0);
  }
  return smallest ? t + t / 20 : t;
}

// Grid geometry of one launch over `count` tensors.  One CTA per SM.  Every
// warp decodes whole units, so a tensor is only as fast as its busiest CTA.  A tensor with so
// few units that every one can have a warp of its own is decoded with one chain per warp: a
// step then takes the latency of one chain (65 cycles instead of 90 in a lone warp).  Others are
// decoded kChains units at a time, by no more warps than make the rounds even (14 groups and 13
// warps: two rounds of 7).  Tensors of one launch differ in size and in unit length: each gets its
// own number of warps and of CTAs -- in proportion to the symbols first, then moved one at a time
// from the tensor that finishes first to the one that finishes last, by the estimate of
// step_cycles.  The number of table copies is the one with the lowest estimate for the busiest
// CTA: more copies than one per two banks do not speed a step up, but they take the place of
// warps, and with fewer there is no loop for narrow rows (8192 x 8192 elements at precision 0: 14
// warps beside 8 copies 48 us, 7 warps twice beside 16 copies 58).
static int decode_geometry(const HostItem *items, uint32_t count, int precision, uint32_t ring_bytes,
                           BatchArgs &b, uint32_t &warps, uint32_t &smem_bytes) {
  const uint32_t sm_smem = 227u * 1024u;
  const uint32_t max_warps = items[0].gx ? (uint32_t)kDotMaxWarps
                             : items[0].grad ? (uint32_t)kUpdateMaxWarps : (uint32_t)kDecodeMaxWarps;
  uint64_t total_work = 0, total_units = 0;
  uint32_t units[kMaxBatch], groups[kMaxBatch], guard[kMaxBatch], per_warp[kMaxBatch];
  for (uint32_t t = 0; t < count; ++t) {
    const uint64_t U = 32ull * items[t].S;
    uint64_t ub = items[t].max_unit_words ? (uint64_t)items[t].max_unit_words * 2 : U;
    if (ub > U) ub = U;
    if (ub < 160) ub = 160;
    b.item[t].slot_bytes = (uint32_t)((ub + 32 + 15) & ~uint64_t(15));
    guard[t] = 1024 + (((items[t].S + 8) * 2 + 127) & ~127u);
    per_warp[t] = kChains * b.item[t].slot_bytes + ring_bytes;
    if (16 * 1024 + guard[t] + per_warp[t] > sm_smem) {
      set_error("decode: a warp's units of %u symbols do not fit in shared memory", (unsigned)U);
      return NZ_E_ARG;
    }
    units[t] = work_units(items[t]);         // at least one
    groups[t] = (units[t] - 1) / kChains + 1;
    total_units += units[t];
    total_work += (uint64_t)groups[t] * items[t].S;
  }
  // CTAs per tensor: one per SM (fewer when there is not enough work to give every SM a
  // unit), in proportion to the symbols, at least one
  uint32_t n_ctas = (uint32_t)sm_count();
  if (total_units < n_ctas) n_ctas = (uint32_t)total_units;
  if (n_ctas < count) n_ctas = count;
  uint32_t share[kMaxBatch], used = 0;
  for (uint32_t t = 0; t < count; ++t) {
    uint64_t c = total_work ? (uint64_t)groups[t] * items[t].S * n_ctas / total_work : 1;
    if (c > units[t]) c = units[t];
    if (c < 1) c = 1;
    share[t] = (uint32_t)c;
    used += share[t];
  }
  // units of a CTA, and whether each of them gets a warp beside a table of 4096 << sh bytes
  // (matrix-vector and update launches always decode two units per warp)
  const bool pairs_only = items[0].gx || items[0].grad;
  auto own = [&](uint32_t t, uint32_t c) { return (units[t] - 1) / c + 1; };
  auto alone = [&](uint32_t t, uint32_t each, uint32_t sh) {
    return !pairs_only && each <= max_warps &&
           (4096u << sh) + guard[t] + each * (b.item[t].slot_bytes + ring_bytes) <= sm_smem;
  };
  bool hidden = true;          // every tensor's inputs are stable: the set-up overlaps the kernel before
  for (uint32_t t = 0; t < count; ++t) hidden = hidden && (items[t].flags & NZ_ITEM_INPUTS_STABLE);
  hidden = hidden || (precision == 7 && !items[0].out_exp);    // (exponent streams have 10 bits)
  const uint32_t pb = usual_prob_bits(precision);
  uint64_t best = ~0ull;
  uint32_t ctas[kMaxBatch] = {};
  b.lut_shift = 2;
  // a table of 2^12 slots x 2^(sh-2) copies; 32 copies at the expected resolution are enough
  for (uint32_t sh = pb == kMinProbBits ? 4 : 5; sh >= 2; --sh) {
    const uint32_t copies = (1024u << sh) >> pb;
    const bool narrow = copies >= (precision == 7 ? 32u : 16u);
    uint32_t cap[kMaxBatch];
    bool fits = true;
    for (uint32_t t = 0; t < count; ++t) {
      const uint32_t fixed = (4096u << sh) + guard[t];
      cap[t] = fixed + per_warp[t] <= sm_smem ? (sm_smem - fixed) / per_warp[t] : 0;
      if (cap[t] > max_warps) cap[t] = max_warps;
      if (cap[t] == 0) fits = false;
    }
    if (!fits) continue;
    auto cost = [&](uint32_t t, uint32_t c) -> uint64_t {
      const uint32_t each = own(t, c);
      if (alone(t, each, sh)) return (uint64_t)items[t].S * step_cycles(each, 1, narrow, sh == 2, precision);
      const uint32_t g = (groups[t] + c - 1) / c, rounds = (g + cap[t] - 1) / cap[t];
      // between two rounds a warp opens its next units
      constexpr uint32_t kRoundCycles = 1500;
      const uint32_t step = step_cycles((g + rounds - 1) / rounds, kChains, narrow, sh == 2, precision);
      return (uint64_t)rounds * (items[t].S * step + kRoundCycles);
    };
    uint32_t now[kMaxBatch], sum = used;
    for (uint32_t t = 0; t < count; ++t) now[t] = share[t];
    if (count == 1) {
      now[0] = n_ctas;
    } else {
      for (uint32_t it = 0; it < 6 * kMaxBatch; ++it) {
        uint32_t hi = 0, lo = kMaxBatch;
        for (uint32_t t = 1; t < count; ++t)
          if (cost(t, now[t]) > cost(hi, now[hi])) hi = t;
        if (sum < n_ctas) {
          if (now[hi] >= units[hi]) break;
          ++now[hi];
          ++sum;
          continue;
        }
        for (uint32_t t = 0; t < count; ++t)
          if (now[t] > 1 && (sum > n_ctas || t != hi) &&
              (lo == kMaxBatch || cost(t, now[t] - 1) < cost(lo, now[lo] - 1)))
            lo = t;
        if (lo == kMaxBatch) break;
        if (sum > n_ctas) {                      // many tiny tensors were given one each
          --now[lo];
          --sum;
          continue;
        }
        if (now[hi] >= units[hi] || cost(lo, now[lo] - 1) >= cost(hi, now[hi])) break;
        --now[lo];
        ++now[hi];
      }
    }
    // The table has to be written first, 16 bytes per lane and store.  A small launch has few warps
    // for that, and it shows where the launch does not overlap the kernel before it (fresh inputs)
    // and the table does not have the 32 copies whose stores are unrolled, as precision 7 does
    // beside 64 KB.  Reads of 444 x 1600 and 512 x 1024 elements, one unit per CTA, in us beside 16
    // and 64 KB: precision 7 overlapped 9.71, 9.22 and 6.93, 6.55, fresh 14.34, 13.19 and 11.53, 10.73;
    // precision 3 overlapped 9.85, 9.54 and 7.04, 6.76, but fresh 16.3, 19.4 and 13.4, 16.8.
    uint64_t worst = 0;
    for (uint32_t t = 0; t < count; ++t) {
      const uint32_t each = own(t, now[t]), writers = each < 4 && !hidden ? each : 4;
      const uint64_t c = cost(t, now[t]) + (4096u << sh) / (16 * writers);
      if (c > worst) worst = c;
    }
    if (worst < best) {
      best = worst;
      b.lut_shift = sh;
      for (uint32_t t = 0; t < count; ++t) {
        ctas[t] = now[t];
        b.item[t].warps = cap[t];
      }
    }
  }
  b.lut_bytes = 4096u << b.lut_shift;
  warps = 1;
  smem_bytes = 0;
  uint32_t begin = 0;
  for (uint32_t t = 0; t < count; ++t) {
    BatchItem &it = b.item[t];
    // no more warps than make the rounds even, and a second staging buffer per warp where
    // there is more than one round and room for it
    const uint32_t fixed0 = b.lut_bytes + guard[t], each = own(t, ctas[t]);
    if (alone(t, each, b.lut_shift)) {
      it.chains = 1;
      it.warps = each;
      it.bufs = 1;
      it.groups_each = units[t] / (ctas[t] * it.warps);
      it.groups_more = units[t] % (ctas[t] * it.warps);
    } else {
      const uint32_t g = (groups[t] + ctas[t] - 1) / ctas[t];
      const uint32_t rounds = (g + it.warps - 1) / it.warps;
      it.chains = kChains;
      it.warps = (g + rounds - 1) / rounds;
      it.bufs = rounds > 1 && fixed0 + it.warps * (ring_bytes + 2 * kChains * it.slot_bytes) <= sm_smem
                    ? 2u : 1u;
      it.groups_each = groups[t] / (ctas[t] * it.warps);
      it.groups_more = groups[t] % (ctas[t] * it.warps);
    }
    it.ring_offset = fixed0 + it.bufs * it.warps * it.chains * it.slot_bytes;
    const uint32_t need = it.ring_offset + it.warps * ring_bytes;
    if (need > smem_bytes) smem_bytes = need;
    if (it.warps > warps) warps = it.warps;
    it.cta_begin = begin;
    begin += ctas[t];
  }
  b.n_ctas = begin;
  return NZ_OK;
}

// Decode `count` tensors (same precision and lane_symbols), kMaxBatch per launch.
int decode_many(const HostItem *items, uint32_t count, int precision, uint32_t S, int canon,
                bool merge, void *status, cudaStream_t st) {
  HostItem live[kMaxBatch];
  uint32_t n_live = 0;
  auto flush = [&]() -> int {
    if (n_live == 0) return NZ_OK;
    BatchArgs b;
    memset(&b, 0, sizeof(b));
    uint32_t warps = 0, smem_bytes = 0;
    // the exponent-only kernel is the precision-7 instantiation
    int rc = decode_geometry(live, n_live, precision, ring_warp_bytes(merge ? precision : 7), b,
                             warps, smem_bytes);
    if (rc) return rc;
    b.count = n_live;
    b.canon = canon;
    b.status = (uint32_t *)status;
    for (uint32_t t = 0; t < n_live; ++t) {
      b.item[t].container = (const uint8_t *)live[t].container;
      b.item[t].frac = (const uint8_t *)live[t].frac;
      b.item[t].n = live[t].n;
      b.item[t].out_bf16 = (uint16_t *)live[t].out_bf16;
      b.item[t].out_exp = (uint8_t *)live[t].out_exp;
      b.item[t].n_units = (uint32_t)unit_count(live[t].n, live[t].S);
      b.item[t].tile_cols = live[t].tile_cols;
      b.item[t].S = live[t].S;
      b.item[t].segs = live[t].tile_cols ? (live[t].tile_cols / 64) / (live[t].S / 8) : 0;
      b.item[t].full_units = (uint32_t)(live[t].n / (32ull * live[t].S));
      const uint64_t words =
          (live[t].container_bytes - payload_offset(b.item[t].n_units)) / 2;   // checked: not negative
      b.item[t].max_words = words < 0x7FFFFFFFull ? (uint32_t)words : 0x7FFFFFFFu;
      b.item[t].norm = live[t].norm;
      b.item[t].norm_lg = live[t].norm_lg;
    }
    const bool gather = live[0].unit_list != nullptr;   // gather calls pass a single item
    b.unit_list = live[0].unit_list;
    b.n_list = live[0].n_list;
    const bool dot = live[0].gx != nullptr;             // so do matrix-vector calls
    b.gx = live[0].gx;
    b.partial = live[0].partial;
    b.in = live[0].in;
    b.seg = live[0].seg;
    const bool update = live[0].grad != nullptr;        // and update calls
    b.grad = live[0].grad;
    b.exp_avg = live[0].exp_avg;
    b.exp_avg_sq = live[0].exp_avg_sq;
    b.adam = live[0].adam;
    b.inputs_stable = 1;
    for (uint32_t t = 0; t < n_live; ++t)
      if (!(live[t].flags & NZ_ITEM_INPUTS_STABLE)) b.inputs_stable = 0;
    n_live = 0;
    if (!merge) return launch_decode_exponents(b, warps, smem_bytes, st);
    const int mode = gather ? kModeList : update ? kModeUpdate : dot ? kModeDot : kModeTensor;
    switch (precision) {
      case 0: return launch_decode_precision<0>(mode, b, warps, smem_bytes, st);
      case 1: return launch_decode_precision<1>(mode, b, warps, smem_bytes, st);
      case 3: return launch_decode_precision<3>(mode, b, warps, smem_bytes, st);
      default: return launch_decode_precision<7>(mode, b, warps, smem_bytes, st);
    }
  };
  for (uint32_t i = 0; i < count; ++i) {
    if (items[i].n == 0) continue;
    const uint64_t nu = unit_count(items[i].n, items[i].S ? items[i].S : S);
    if (items[i].container_bytes < payload_offset(nu)) {
      set_error("decode: container %u of %llu bytes is too short for %llu units", i,
                (unsigned long long)items[i].container_bytes, (unsigned long long)nu);
      return NZ_E_FORMAT;
    }
    live[n_live] = items[i];
    if (!live[n_live].S) live[n_live].S = S;
    ++n_live;
    if (n_live == kMaxBatch) {
      int rc = flush();
      if (rc) return rc;
    }
  }
  return flush();
}

int decode_common(const void *container, uint64_t container_bytes, const void *frac, uint64_t n,
                  int precision, uint32_t S, uint32_t max_unit_words, int canon, void *out_bf16,
                  void *out_exp, void *status, cudaStream_t st) {
  HostItem it;
  it.container = container;
  it.container_bytes = container_bytes;
  it.frac = frac;
  it.n = n;
  it.max_unit_words = max_unit_words;
  it.out_bf16 = out_bf16;
  it.out_exp = out_exp;
  it.unit_list = nullptr;
  it.n_list = 0;
  it.gx = nullptr;
  it.partial = nullptr;
  it.in = it.seg = 0;
  it.flags = 0;
  it.tile_cols = 0;
  it.S = 0;
  it.grad = nullptr;
  it.exp_avg = it.exp_avg_sq = nullptr;
  it.norm = nullptr;
  it.norm_lg = 0;
  return decode_many(&it, 1, precision, S, canon, out_bf16 != nullptr, status, st);
}

// A [rows, cols] matrix stored in operand order, decoded to row-major.
int decode_operand(const void *container, uint64_t container_bytes, const void *frac, uint64_t rows,
                   uint64_t cols, int precision, uint32_t S, uint32_t max_unit_words, int canon,
                   void *out_bf16, void *status, cudaStream_t st) {
  HostItem it;
  memset(&it, 0, sizeof(it));
  it.container = container;
  it.container_bytes = container_bytes;
  it.frac = frac;
  it.n = rows * cols;
  it.max_unit_words = max_unit_words;
  it.out_bf16 = out_bf16;
  it.tile_cols = (uint32_t)cols;
  return decode_many(&it, 1, precision, S, canon, true, status, st);
}

// Decode a tensor and apply an AdamW step to it on the way out: out_bf16 receives the
// updated (row-major) weights, the moments (bf16) are updated in place.
int decode_update(const void *container, uint64_t container_bytes, const void *frac, uint64_t n,
                  uint64_t operand_cols, int precision, uint32_t S, uint32_t max_unit_words,
                  int canon, const void *grad, void *exp_avg, void *exp_avg_sq, const AdamArgs &adam,
                  void *out_bf16, void *status, cudaStream_t st) {
  HostItem it;
  memset(&it, 0, sizeof(it));
  it.container = container;
  it.container_bytes = container_bytes;
  it.frac = frac;
  it.n = n;
  it.max_unit_words = max_unit_words;
  it.out_bf16 = out_bf16;
  it.tile_cols = (uint32_t)operand_cols;
  it.grad = (const uint16_t *)grad;
  it.exp_avg = (uint16_t *)exp_avg;
  it.exp_avg_sq = (uint16_t *)exp_avg_sq;
  it.adam = adam;
  return decode_many(&it, 1, precision, S, canon, true, status, st);
}

}  // namespace nz

static int check_decode_args(const char *who, const void *container, uint64_t n, uint32_t S) {
  if (!nz::valid_lane_symbols(S)) {
    nz::set_error("%s: lane_symbols must be a multiple of 8 in [8, %u] (got %u)", who,
                  nz::kMaxLaneSymbols, S);
    return NZ_E_ARG;
  }
  if (n >= (1ull << 32)) {
    nz::set_error("%s: tensors of 2^32 or more elements are not supported", who);
    return NZ_E_ARG;
  }
  if (n && (!container || ((uintptr_t)container & 15))) {
    nz::set_error("%s: container must be a 16-byte aligned device pointer", who);
    return NZ_E_ARG;
  }
  return NZ_OK;
}

extern "C" int nz_decode_exponents(const void *container, uint64_t container_bytes, uint64_t n,
                                   uint32_t lane_symbols, uint32_t max_unit_words, void *exp_out,
                                   void *status, void *stream) {
  int rc = check_decode_args("nz_decode_exponents", container, n, lane_symbols);
  if (rc) return rc;
  if (n && (!exp_out || ((uintptr_t)exp_out & 7))) {
    nz::set_error("nz_decode_exponents: output must be an 8-byte aligned device pointer");
    return NZ_E_ARG;
  }
  return nz::decode_common(container, container_bytes, nullptr, n, 7, lane_symbols,
                           max_unit_words, 0, nullptr, exp_out, status, (cudaStream_t)stream);
}

extern "C" int nz_decompress_bf16(const void *container, uint64_t container_bytes,
                                  const void *frac_in, uint64_t n, int precision,
                                  uint32_t lane_symbols, uint32_t max_unit_words,
                                  int canonical_nan, void *out_bf16, void *status, void *stream) {
  if (!nz::valid_precision(precision)) {
    nz::set_error("nz_decompress_bf16: precision must be 0, 1, 3 or 7 (got %d)", precision);
    return NZ_E_ARG;
  }
  int rc = check_decode_args("nz_decompress_bf16", container, n, lane_symbols);
  if (rc) return rc;
  if (n && (!out_bf16 || !frac_in || ((uintptr_t)out_bf16 & 15) || ((uintptr_t)frac_in & 7))) {
    nz::set_error("nz_decompress_bf16: output must be 16-byte, fractions 8-byte aligned");
    return NZ_E_ARG;
  }
  return nz::decode_common(container, container_bytes, frac_in, n, precision, lane_symbols,
                           max_unit_words, canonical_nan, out_bf16, nullptr, status,
                           (cudaStream_t)stream);
}

extern "C" int nz_decompress_bf16_batch(const nz_decompress_item *items, uint32_t count,
                                        int precision, uint32_t lane_symbols, int canonical_nan,
                                        void *status, void *stream) {
  if (!nz::valid_precision(precision)) {
    nz::set_error("nz_decompress_bf16_batch: precision must be 0, 1, 3 or 7 (got %d)", precision);
    return NZ_E_ARG;
  }
  if (count == 0) return NZ_OK;
  if (!items) {
    nz::set_error("nz_decompress_bf16_batch: null item array");
    return NZ_E_ARG;
  }
  constexpr uint32_t kChunk = 64;
  nz::HostItem host[kChunk];
  for (uint32_t base = 0; base < count; base += kChunk) {
    const uint32_t m = count - base < kChunk ? count - base : kChunk;
    for (uint32_t i = 0; i < m; ++i) {
      const nz_decompress_item &it = items[base + i];
      int rc = check_decode_args("nz_decompress_bf16_batch", it.container, it.n, lane_symbols);
      if (rc) return rc;
      if (it.n && (!it.out_bf16 || !it.frac_in || ((uintptr_t)it.out_bf16 & 15) ||
                   ((uintptr_t)it.frac_in & 7))) {
        nz::set_error("nz_decompress_bf16_batch: item %u: output must be 16-byte, fractions "
                      "8-byte aligned", base + i);
        return NZ_E_ARG;
      }
      host[i].container = it.container;
      host[i].container_bytes = it.container_bytes;
      host[i].frac = it.frac_in;
      host[i].n = it.n;
      host[i].max_unit_words = it.max_unit_words;
      host[i].out_bf16 = it.out_bf16;
      host[i].out_exp = nullptr;
      host[i].unit_list = nullptr;
      host[i].n_list = 0;
      host[i].gx = nullptr;
      host[i].partial = nullptr;
      host[i].in = host[i].seg = 0;
      host[i].flags = it.flags;
      host[i].tile_cols = 0;
      host[i].S = 0;
      host[i].grad = nullptr;
      host[i].exp_avg = host[i].exp_avg_sq = nullptr;
      host[i].norm = nullptr;
      host[i].norm_lg = 0;
      if (it.normalizers) {
        const uint32_t g = it.normalizer_group;
        if (g == 0 || g > 1024 || (g & (g - 1)) || it.operand_cols) {
          nz::set_error("nz_decompress_bf16_batch: item %u: the normaliser group must be a power "
                        "of two in [1, 1024] (got %u) and the tensor in stream order", base + i, g);
          return NZ_E_ARG;
        }
        host[i].norm = (const uint8_t *)it.normalizers;
        while ((1u << host[i].norm_lg) < g) ++host[i].norm_lg;
      }
      if (it.lane_symbols) {
        if (!nz::valid_lane_symbols(it.lane_symbols)) {
          nz::set_error("nz_decompress_bf16_batch: item %u: lane_symbols must be a multiple of 8 "
                        "in [8, %u] (got %u)", base + i, nz::kMaxLaneSymbols, it.lane_symbols);
          return NZ_E_ARG;
        }
        host[i].S = it.lane_symbols;
      }
      if (it.operand_cols) {
        const uint64_t c = it.operand_cols;
        const uint32_t item_s = it.lane_symbols ? it.lane_symbols : lane_symbols;
        if (c % 64 || it.n % (4 * c) || (c / 64) % (item_s / 8) || c >= (1ull << 31)) {
          nz::set_error("nz_decompress_bf16_batch: item %u: %llu elements in rows of %llu are not "
                        "in operand order for lane_symbols %u", base + i,
                        (unsigned long long)it.n, (unsigned long long)c, lane_symbols);
          return NZ_E_ARG;
        }
        host[i].tile_cols = (uint32_t)c;
      }
    }
    int rc = nz::decode_many(host, m, precision, lane_symbols, canonical_nan, true, status,
                             (cudaStream_t)stream);
    if (rc) return rc;
  }
  return NZ_OK;
}

extern "C" int nz_decompress_bf16_item(const nz_decompress_item *item, void *out_bf16, uint32_t flags,
                                       int precision, int canonical_nan, void *status,
                                       void *stream) {
  if (!item) {
    nz::set_error("nz_decompress_bf16_item: null item");
    return NZ_E_ARG;
  }
  nz_decompress_item it = *item;
  it.out_bf16 = out_bf16;
  it.flags = flags;
  return nz_decompress_bf16_batch(&it, 1, precision, it.lane_symbols, canonical_nan, status, stream);
}

static int decompress_units(const void *container, uint64_t container_bytes, const void *frac_in,
                            uint64_t n, int precision, uint32_t lane_symbols,
                            uint32_t max_unit_words, int canonical_nan, const void *unit_ids,
                            uint32_t n_ids, const void *normalizers, uint32_t group, void *out_bf16,
                            void *status, void *stream);

extern "C" int nz_decompress_bf16_units(const void *container, uint64_t container_bytes,
                                        const void *frac_in, uint64_t n, int precision,
                                        uint32_t lane_symbols, uint32_t max_unit_words,
                                        int canonical_nan, const void *unit_ids, uint32_t n_ids,
                                        void *out_bf16, void *status, void *stream) {
  return decompress_units(container, container_bytes, frac_in, n, precision, lane_symbols,
                          max_unit_words, canonical_nan, unit_ids, n_ids, nullptr, 0, out_bf16, status,
                          stream);
}

static int decompress_units(const void *container, uint64_t container_bytes, const void *frac_in,
                            uint64_t n, int precision, uint32_t lane_symbols,
                            uint32_t max_unit_words, int canonical_nan, const void *unit_ids,
                            uint32_t n_ids, const void *normalizers, uint32_t group, void *out_bf16,
                            void *status, void *stream) {
  if (!nz::valid_precision(precision)) {
    nz::set_error("nz_decompress_bf16_units: precision must be 0, 1, 3 or 7 (got %d)", precision);
    return NZ_E_ARG;
  }
  int rc = check_decode_args("nz_decompress_bf16_units", container, n, lane_symbols);
  if (rc) return rc;
  if (n_ids == 0) return NZ_OK;
  if (n == 0) {
    nz::set_error("nz_decompress_bf16_units: an empty tensor has no units");
    return NZ_E_ARG;
  }
  if (!unit_ids || ((uintptr_t)unit_ids & 3) || !out_bf16 || !frac_in ||
      ((uintptr_t)out_bf16 & 15) || ((uintptr_t)frac_in & 7)) {
    nz::set_error("nz_decompress_bf16_units: unit list must be a 4-byte aligned device pointer, "
                  "output 16-byte, fractions 8-byte aligned");
    return NZ_E_ARG;
  }
  nz::HostItem it;
  it.container = container;
  it.container_bytes = container_bytes;
  it.frac = frac_in;
  it.n = n;
  it.max_unit_words = max_unit_words;
  it.out_bf16 = out_bf16;
  it.out_exp = nullptr;
  it.unit_list = (const uint32_t *)unit_ids;
  it.n_list = n_ids;
  it.gx = nullptr;
  it.partial = nullptr;
  it.in = it.seg = 0;
  it.flags = 0;
  it.tile_cols = 0;
  it.S = 0;
  it.grad = nullptr;
  it.exp_avg = it.exp_avg_sq = nullptr;
  it.norm = nullptr;
  it.norm_lg = 0;
  if (normalizers) {
    if (group == 0 || group > 1024 || (group & (group - 1))) {
      nz::set_error("gather: the normaliser group must be a power of two in [1, 1024] (got %u)", group);
      return NZ_E_ARG;
    }
    it.norm = (const uint8_t *)normalizers;
    while ((1u << it.norm_lg) < group) ++it.norm_lg;
  }
  return nz::decode_many(&it, 1, precision, lane_symbols, canonical_nan, true, status,
                         (cudaStream_t)stream);
}

namespace nz {

// Row gather, step 1: the units that hold each requested row.  Row r of a
// table with rows of `row_len` elements starts at element r * row_len; it is
// decoded as `per_row` consecutive units from the one that holds its first
// element (numbers past the last unit are clamped: their output is not used).
// Rows outside the table get unit n_units, which the decoder reports.
__global__ void gather_plan_kernel(const int64_t *__restrict__ rows, uint32_t k, uint64_t row_len,
                                   uint64_t n_rows, uint64_t U, uint32_t n_units, uint32_t per_row,
                                   uint32_t *__restrict__ units) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint64_t)k * per_row) return;
  const int64_t r = rows[i / per_row];
  uint32_t u = n_units;
  if (r >= 0 && (uint64_t)r < n_rows) {
    const uint64_t v = (uint64_t)r * row_len / U + i % per_row;
    u = v < n_units ? (uint32_t)v : n_units - 1;
  }
  units[i] = u;
}

// Row gather, step 3: copy each row out of the units decoded for it.  VEC = 8
// moves 16 bytes per thread (row length and so every offset a multiple of 8).
template <int VEC>
__global__ void gather_copy_kernel(const int64_t *__restrict__ rows, uint32_t k, uint64_t row_len,
                                   uint64_t n_rows, uint64_t U, uint32_t per_row,
                                   const uint16_t *__restrict__ staging,
                                   uint16_t *__restrict__ out) {
  const uint64_t per = row_len / VEC;
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint64_t)k * per) return;
  const uint64_t row = i / per, j = (i % per) * VEC;
  const int64_t r = rows[row];
  if (r < 0 || (uint64_t)r >= n_rows) return;        // flagged by the decoder; left untouched
  const uint64_t src = row * per_row * U + ((uint64_t)r * row_len) % U + j;
  if (VEC == 8)
    *reinterpret_cast<uint4 *>(out + row * row_len + j) =
        *reinterpret_cast<const uint4 *>(staging + src);
  else
    out[row * row_len + j] = staging[src];
}

static inline uint32_t gather_units_per_row(uint64_t row_len, uint64_t U) {
  if (U % row_len == 0) return 1;                            // a unit holds whole rows
  if (row_len % U == 0) return (uint32_t)(row_len / U);      // a row is whole units
  return (uint32_t)((row_len + U - 1) / U + 1);              // rows straddle unit boundaries
}

}  // namespace nz

extern "C" uint64_t nz_gather_scratch_bytes(uint32_t n_rows_out, uint64_t row_len,
                                            uint32_t lane_symbols) {
  if (!nz::valid_lane_symbols(lane_symbols) || row_len == 0) return 0;
  const uint64_t U = 32ull * lane_symbols;
  const uint64_t per_row = nz::gather_units_per_row(row_len, U);
  // unit list (4 bytes each, rounded to 16) + the decoded units
  return nz::align16((uint64_t)n_rows_out * per_row * 4) + (uint64_t)n_rows_out * per_row * U * 2;
}

extern "C" int nz_gather_rows_bf16(const void *container, uint64_t container_bytes,
                                   const void *frac_in, uint64_t n, int precision,
                                   uint32_t lane_symbols, uint32_t max_unit_words,
                                   int canonical_nan, uint64_t row_len, const void *rows_i64,
                                   uint32_t n_rows_out, void *out_bf16, void *scratch,
                                   uint64_t scratch_bytes, void *status, void *stream) {
  return nz_gather_rows_normalized_bf16(container, container_bytes, frac_in, n, precision,
                                        lane_symbols, max_unit_words, canonical_nan, row_len,
                                        rows_i64, n_rows_out, nullptr, 0, out_bf16, scratch,
                                        scratch_bytes, status, stream);
}

extern "C" int nz_gather_rows_normalized_bf16(const void *container, uint64_t container_bytes,
                                              const void *frac_in, uint64_t n, int precision,
                                              uint32_t lane_symbols, uint32_t max_unit_words,
                                              int canonical_nan, uint64_t row_len,
                                              const void *rows_i64, uint32_t n_rows_out,
                                              const void *normalizers, uint32_t normalizer_group,
                                              void *out_bf16, void *scratch, uint64_t scratch_bytes,
                                              void *status, void *stream) {
  if (!nz::valid_precision(precision)) {
    nz::set_error("nz_gather_rows_bf16: precision must be 0, 1, 3 or 7 (got %d)", precision);
    return NZ_E_ARG;
  }
  int rc = check_decode_args("nz_gather_rows_bf16", container, n, lane_symbols);
  if (rc) return rc;
  if (row_len == 0 || n == 0 || n % row_len) {
    nz::set_error("nz_gather_rows_bf16: row length %llu does not divide the %llu elements",
                  (unsigned long long)row_len, (unsigned long long)n);
    return NZ_E_ARG;
  }
  if (n_rows_out == 0) return NZ_OK;
  if (!rows_i64 || ((uintptr_t)rows_i64 & 7) || !out_bf16 || !frac_in || !scratch ||
      ((uintptr_t)scratch & 15) || ((uintptr_t)frac_in & 7)) {
    nz::set_error("nz_gather_rows_bf16: null or misaligned pointer (rows and fractions 8-byte, "
                  "scratch 16-byte aligned)");
    return NZ_E_ARG;
  }
  const uint64_t need = nz_gather_scratch_bytes(n_rows_out, row_len, lane_symbols);
  if (scratch_bytes < need) {
    nz::set_error("nz_gather_rows_bf16: scratch of %llu bytes is smaller than the %llu required",
                  (unsigned long long)scratch_bytes, (unsigned long long)need);
    return NZ_E_CAPACITY;
  }
  const uint64_t U = 32ull * lane_symbols;
  const uint32_t per_row = nz::gather_units_per_row(row_len, U);
  const uint64_t n_list = (uint64_t)n_rows_out * per_row;
  if (n_list >= (1ull << 32)) {
    nz::set_error("nz_gather_rows_bf16: %u rows of %u units each are too many for one call",
                  n_rows_out, per_row);
    return NZ_E_ARG;
  }
  cudaStream_t st = (cudaStream_t)stream;
  uint32_t *units = (uint32_t *)scratch;
  uint16_t *staging = (uint16_t *)((uint8_t *)scratch + nz::align16(n_list * 4));
  const uint32_t n_units = (uint32_t)nz::unit_count(n, lane_symbols);
  const uint64_t table_rows = n / row_len;
  nz::gather_plan_kernel<<<(unsigned)((n_list + 255) / 256), 256, 0, st>>>(
      (const int64_t *)rows_i64, n_rows_out, row_len, table_rows, U, n_units, per_row, units);
  NZ_LAUNCH_CHECK("gather_plan_kernel");
  rc = decompress_units(container, container_bytes, frac_in, n, precision, lane_symbols,
                        max_unit_words, canonical_nan, units, (uint32_t)n_list, normalizers,
                        normalizer_group, staging, status, stream);
  if (rc) return rc;
  const bool vec = row_len % 8 == 0 && ((uintptr_t)out_bf16 & 15) == 0;
  const uint64_t threads = vec ? (uint64_t)n_rows_out * (row_len / 8) : (uint64_t)n_rows_out * row_len;
  const uint64_t blocks = (threads + 255) / 256;
  if (blocks >= (1ull << 31)) {
    nz::set_error("nz_gather_rows_bf16: output too large for one call");
    return NZ_E_ARG;
  }
  if (vec)
    nz::gather_copy_kernel<8><<<(unsigned)blocks, 256, 0, st>>>(
        (const int64_t *)rows_i64, n_rows_out, row_len, table_rows, U, per_row, staging,
        (uint16_t *)out_bf16);
  else
    nz::gather_copy_kernel<1><<<(unsigned)blocks, 256, 0, st>>>(
        (const int64_t *)rows_i64, n_rows_out, row_len, table_rows, U, per_row, staging,
        (uint16_t *)out_bf16);
  NZ_LAUNCH_CHECK("gather_copy_kernel");
  return NZ_OK;
}

namespace nz {
// Rows of an [out, in] matrix that one unit of U elements can touch.
static inline uint32_t dot_segments(uint64_t in_features, uint64_t U) {
  return (uint32_t)((U - 1) / in_features + 2);
}
}  // namespace nz

extern "C" uint64_t nz_linear_vec_scratch_bytes(uint64_t n, uint64_t in_features,
                                                uint32_t lane_symbols) {
  if (!nz::valid_lane_symbols(lane_symbols) || in_features == 0) return 0;
  const uint64_t U = 32ull * lane_symbols;
  return nz::align16(nz::unit_count(n, lane_symbols) * nz::dot_segments(in_features, U) * 4);
}

extern "C" int nz_linear_vec_bf16(const void *container, uint64_t container_bytes,
                                  const void *frac_in, uint64_t n, int precision,
                                  uint32_t lane_symbols, uint32_t max_unit_words,
                                  int canonical_nan, uint64_t in_features, const void *x_f32,
                                  const void *bias_bf16, void *y_bf16, void *scratch,
                                  uint64_t scratch_bytes, void *status, void *stream) {
  if (!nz::valid_precision(precision)) {
    nz::set_error("nz_linear_vec_bf16: precision must be 0, 1, 3 or 7 (got %d)", precision);
    return NZ_E_ARG;
  }
  int rc = check_decode_args("nz_linear_vec_bf16", container, n, lane_symbols);
  if (rc) return rc;
  if (n == 0 || in_features == 0 || in_features % 256 || n % in_features ||
      in_features >= (1ull << 31) || n / in_features >= (1ull << 31)) {
    nz::set_error("nz_linear_vec_bf16: the matrix must have rows of a multiple of 256 elements "
                  "(got %llu elements, rows of %llu)", (unsigned long long)n,
                  (unsigned long long)in_features);
    return NZ_E_ARG;
  }
  if (!x_f32 || ((uintptr_t)x_f32 & 15) || !y_bf16 || !frac_in || ((uintptr_t)frac_in & 7) ||
      !scratch || ((uintptr_t)scratch & 15)) {
    nz::set_error("nz_linear_vec_bf16: null or misaligned pointer (input vector and scratch "
                  "16-byte, fractions 8-byte aligned)");
    return NZ_E_ARG;
  }
  const uint64_t need = nz_linear_vec_scratch_bytes(n, in_features, lane_symbols);
  if (scratch_bytes < need) {
    nz::set_error("nz_linear_vec_bf16: scratch of %llu bytes is smaller than the %llu required",
                  (unsigned long long)scratch_bytes, (unsigned long long)need);
    return NZ_E_CAPACITY;
  }
  const uint64_t U = 32ull * lane_symbols;
  nz::HostItem it;
  it.container = container;
  it.container_bytes = container_bytes;
  it.frac = frac_in;
  it.n = n;
  it.max_unit_words = max_unit_words;
  it.out_bf16 = nullptr;
  it.out_exp = nullptr;
  it.unit_list = nullptr;
  it.n_list = 0;
  it.gx = (const float *)x_f32;
  it.partial = (float *)scratch;
  it.in = (uint32_t)in_features;
  it.seg = nz::dot_segments(in_features, U);
  it.flags = 0;
  it.tile_cols = 0;
  it.S = 0;
  it.grad = nullptr;
  it.exp_avg = it.exp_avg_sq = nullptr;
  it.norm = nullptr;
  it.norm_lg = 0;
  rc = nz::decode_many(&it, 1, precision, lane_symbols, canonical_nan, true, status,
                       (cudaStream_t)stream);
  if (rc) return rc;
  const uint32_t out_features = (uint32_t)(n / in_features);
  nz::dot_finish_kernel<<<(out_features + 255) / 256, 256, 0, (cudaStream_t)stream>>>(
      (const float *)scratch, it.seg, U, it.in, out_features, (const uint16_t *)bias_bf16,
      (uint16_t *)y_bf16);
  NZ_LAUNCH_CHECK("dot_finish_kernel");
  return NZ_OK;
}
