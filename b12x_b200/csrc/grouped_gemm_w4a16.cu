// Grouped expert GEMMs of the w4a16 recipe: BF16 activations x NVFP4 (or MXFP4) weights that are
// expanded to 16 bits on the fly, on tcgen05.mma.kind::f16 with FP32 accumulation in TMEM.
//
// The tensor core cannot read 4-bit operands next to 16-bit ones, so the main loop has a conversion
// step, and how often a weight is converted, and how much of a tile is padding, decides the time.
// Operand roles: the WEIGHTS are the 128 rows of the MMA (lanes of TMEM), an expert's tokens its N
// columns, any multiple of 16:
//   * an expert with 2 rows costs 16 columns and one with 270 costs 2 x 144: with the tokens as the
//     128 rows of a tile (what this kernel replaces) the first cost 128 and the second 384;
//   * a converter thread owns one weight row = one TMEM lane and stores its 16-bit values straight
//     into tensor memory (tcgen05.st), where the MMA takes its A operand from: no shared-memory
//     round trip, no proxy fence.
// FC1 with a gated activation interleaves the operand rows: lanes 0..15 of every warp hold 16 up
// rows, lanes 16..31 the gate rows of the same columns, so an epilogue lane finds the other half of
// its pair one shuffle away.
//
// Roles (20 warps): warp 0 fetches packed codes (TMA, 128-byte rows = four k-blocks of 64) and scale
// atoms, warp 2 the token rows, warp 1 issues the MMAs, warps 4..11 convert (two groups of four
// warps, one per TMEM sub-partition, that take the 256-value code stages in turn), warps 12..19 are
// the epilogue, on a double-buffered accumulator.  Every wait is bounded.
//
// Pairs: clusters of two share a tile of 256 weight rows (each CTA converts 128 into its own TMEM)
// and up to 160 token columns, of which each CTA loads half (cta_group::2).
//
// Conversion.  cvt.rn.f16x2.e2m1x2 turns a byte into two FP16 code values and a half2 multiply
// applies the E4M3 block scale, exactly: two instructions per pair.  Re-encoding the product as BF16
// takes three more (FP16 -> FP32 twice, pack), and that sequence tops out at 36 to 39 values per
// clock and SM against 70 to 77; so the MMA runs on FP16 x FP16 and the token rows come as FP16,
// scaled by a power of two per row (permute_rows_f16_kernel), which BF16 values survive unchanged.
// E8M0 scales exceed the FP16 range: with them both operands are BF16.  So they are for an expert one of
// whose rows spans more binades than FP16 carries exactly (permute_rows_f16_kernel marks it): the kernel
// takes the other experts first and then, if there are marks, the marked ones with the same roles on BF16 rows
// and re-encoded weights, at the lower rate.  (Of 50 million values of a SwiGLU some ten lie that close to zero.)
//
// What bounds it and what it took, on the Qwen3-235B shape (K 4096, I 1536, 128 experts, top-8),
// FC1 / FC2 in microseconds:
//   16 tokens, one CTA: 352 / 174 (128-token tiles) -> 121 / 63; the weights alone are 88 / 44 at the
//     copy rate, the rest is the MMA thread and 13.1 waves of 64-row tiles.
//   4096 tokens, pairs: 1046 / 570 (two launches each) -> 655 / 360 = 1260 / 1145 TFLOP/s of useful
//     work; the tensor pipe is busy 85 % of the time, 7 % of its columns are padding.
//   The MMA thread and the producers are `elect_one()` regions: behind `lane == 0` the compiler does
//     not know that one thread runs and every MMA, commit and TMA copy took 40 to 60 clocks to issue
//     (four MMAs and two commits 270 clocks against 40); that alone was 409 -> 269 us at 16 tokens.
//   Then, each: one barrier wait and commit per 128 or 256 values of K instead of 64 (269 -> 233),
//     one converter group per code stage instead of all warps looking at every stage (-> 144 with FP16),
//     factors of an epilogue's rows fetched ahead (prefill FC1 921 -> 650).
//
// Numerics follow the reference's W4A16 oracle (tests/_reference/w4a16_reference.py:266-359):
// weights de-quantised then held in BF16, x in BF16, FP32 accumulation, activation in FP32, BF16
// intermediate.
#include <stdlib.h>

#include <type_traits>

#include "cluster_pair.cuh"

namespace b200moe {

int make_tmap_bytes_2d(CUtensorMap* out, const void* base, uint64_t row_bytes, uint64_t rows,
                       uint32_t box_rows);
int num_sms_cached();

namespace w4a16 {
using namespace pair;

constexpr int kKPerBlock = 64;              // BF16 elements per 128-byte token row
constexpr int kKBlocksPerRaw = 4;           // k-blocks per 128-byte row of packed codes
constexpr int kConvGroups = 2;
constexpr int kConvWarps = 4 * kConvGroups;
constexpr int kTokStagesMax = 8;
constexpr int kEpiWarps = 8;               // two per TMEM sub-partition
constexpr int kThreads = (4 + kConvWarps + kEpiWarps) * 32;
constexpr int kSmemCodes = 128 * 128;       // packed codes of 128 weight rows, four k-blocks
constexpr int kSmemSf = 4 * 2048;           // scale atoms: two 64-row sub-tiles, each in at most two row groups
constexpr int kSmemRaw = kSmemCodes + kSmemSf;
constexpr int kMaxExperts = 1024;
constexpr int kTmemCols = 512;
constexpr int kMaxList = 256;               // work items a CTA decodes ahead of its main loop

// What the weights are expanded to: FP16 (E4M3 scales; the token rows then are FP16 too, scaled by a
// power of two per row), or BF16 (E8M0 scales, which exceed the FP16 range; E4M3 scales of marked experts).
enum { TO_F16 = 0, TO_BF16_E8M0 = 1, TO_BF16_E4M3 = 2 };

// A stage is what one wait and one commit of the MMA thread cover.
// ONE: one CTA, 2 x 64 accumulator columns + 3 converted stages of four k-blocks (128 columns each).
// PAIR_NARROW: the same on a CTA pair.  PAIR_WIDE: 2 x 160 + 3 stages of two k-blocks (64 columns).
enum { ONE = 0, PAIR_WIDE = 1, PAIR_NARROW = 2 };
template <int kForm>
struct Cfg {
  static constexpr bool kPair = kForm != ONE;
  static constexpr int kMaxTok = kForm == PAIR_WIDE ? 160 : 64;
  static constexpr int kColStep = kPair ? 32 : 16;   // granularity of the MMA's N (cta_group::2: 32)
  static constexpr int kStageKb = kForm == PAIR_WIDE ? 2 : 4;   // k-blocks per stage
  static constexpr int kStageCols = 32 * kStageKb;   // TMEM columns of a converted stage
  static constexpr int kRing = 3;
  static constexpr int kRingCol = 2 * kMaxTok;
  static constexpr int kRawStages = kForm == PAIR_WIDE ? 4 : 6;
  // token rows: two k-blocks per stage (four where a stage of A has four and no tile of the launch puts
  // more than 32 rows into a CTA), as many stages as the widest tile leaves room for
  static constexpr int kSmemTok = kForm == PAIR_WIDE ? 4 * 80 * 256 : 4 * 64 * 256;
  static_assert(kRingCol + kStageCols * kRing <= kTmemCols, "tensor memory");
};

struct Bars {
  uint64_t rfull[6];    // packed codes and scale atoms landed
  uint64_t rempty[6];   // ... read by the group that converts them
  uint64_t tfull[kTokStagesMax];             // token rows landed (pair: both halves, on the even CTA)
  uint64_t tempty[kTokStagesMax];
  uint64_t afull[4];             // converted stage in TMEM (the four warps of a group, of both CTAs)
  uint64_t aempty[4];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
};
struct __align__(16) SmemTail {
  Bars bars[2];                         // of the unmarked and of the marked experts' run
  uint32_t tmem_base;
  int abort_flag;
  int max_cols;                         // of all tiles of the run
  int any_wide;                         // some experts are marked
  int32_t tile_base[kMaxExperts + 1];   // token tiles before expert e (of the run's experts)
  uint8_t wide[kMaxExperts];
  int32_t offs[kMaxExperts + 1];        // first sorted row of expert e
  int4 list[kMaxList];                  // this CTA's first work items: {expert, weight tile, row0, nrows}
};
template <int kForm>
constexpr int smem_bytes() {
  return 1024 + Cfg<kForm>::kRawStages * kSmemRaw + Cfg<kForm>::kSmemTok + static_cast<int>(sizeof(SmemTail));
}
static_assert(smem_bytes<ONE>() <= 227 * 1024 && smem_bytes<PAIR_NARROW>() <= 227 * 1024 &&
                  smem_bytes<PAIR_WIDE>() <= 227 * 1024, "shared memory of the W4A16 kernel");

enum { EPI_FC1_GATED = 0, EPI_FC1_RELU2 = 1, EPI_FC2 = 2 };

struct Params {
  const uint8_t* sf;             // weight scale storage, 128x4-swizzled [E][sf_rowgroups][atoms_k][512]
  const int32_t* expert_offsets;
  int32_t* status;
  const float* alphas;
  __nv_bfloat16* out_bf16;       // FC1: intermediate [rows][out_cols]
  float* out_f32;                // FC2: routed rows [rows][out_cols]
  float* tap;
  const float* route_weights;    // FC1, optional: per flat route, multiplies the route's row with its alpha
  const int32_t* sorted_route_ids;
  int E, n_tiles, k_blocks, atoms_k, sf_rowgroups, w_rows;
  int sub0_base, sub1_base;      // first weight row of the two 64-row sub-tiles at weight tile 0
  int n_step;                    // weight rows a sub-tile advances per weight tile
  int out_cols;
  int n_row_tiles;               // weight tiles of 128 operand rows (n_tiles counts pairs of them if kPair)
  float limit, act_alpha, act_beta;
  int swigluoai;
  const float* row_inv;          // TO_F16: per sorted row, the power of two that undoes its scaling
  const int32_t* wide;           // TO_F16: per expert, nonzero = marked
};

// A work item: expert, weight tile, and the token rows [row0, row0 + nrows) of the expert.  An
// expert's rows are cut evenly into as few tiles as the column limit allows.
struct Work {
  int e, nt, row0, nrows, cols;
};
template <int kForm>
__device__ __forceinline__ Work decode_work(int w, const Params& p, const SmemTail* tail, int rank) {
  const int32_t* tb = tail->tile_base;
  const int q = w / p.n_tiles;
  int lo = 0, hi = p.E;  // e = number of i in [1,E] with tb[i] <= q
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (tb[mid + 1] <= q) lo = mid + 1; else hi = mid;
  }
  Work c;
  c.e = lo;
  const int me = tb[lo + 1] - tb[lo];
  const int local = w - tb[lo] * p.n_tiles;
  const int nt = local / me, mt = local - nt * me;
  c.nt = Cfg<kForm>::kPair ? 2 * nt + rank : nt;
  const int first = tail->offs[lo], cnt = tail->offs[lo + 1] - first;
  constexpr int kStep = Cfg<kForm>::kColStep;
  const int step = ((cnt + me - 1) / me + kStep - 1) & ~(kStep - 1);
  c.row0 = first + mt * step;
  c.nrows = min(step, cnt - mt * step);
  c.cols = (c.nrows + kStep - 1) & ~(kStep - 1);
  return c;
}
// the i-th item of this CTA, w = its number: out of the list the CTA made at its start where that reaches
template <int kForm>
__device__ __forceinline__ Work get_work(int i, int w, const Params& p, const SmemTail* tail, int rank) {
  if (i >= kMaxList) return decode_work<kForm>(w, p, tail, rank);
  const int4 v = tail->list[i];
  constexpr int kStep = Cfg<kForm>::kColStep;
  Work c;
  c.e = v.x;
  c.nt = v.y;
  c.row0 = v.z;
  c.nrows = v.w;
  c.cols = (c.nrows + kStep - 1) & ~(kStep - 1);
  return c;
}

__device__ __forceinline__ float act_gated(float gate, float up, const Params& p) {
  if (p.limit > 0.f) {
    gate = fminf(gate, p.limit);
    up = fminf(fmaxf(up, -p.limit), p.limit);
  }
  if (p.swigluoai) {
    const float s = __frcp_rn(1.0f + expf(-(p.act_alpha * gate)));
    return (gate * s) * (up + p.act_beta);
  }
  const float s = __frcp_rn(1.0f + expf(-gate));
  return (gate * s) * up;
}

// Four bytes of E2M1 codes (element 0 in the low nibble) -> four f16x2 words of code values: the
// hardware conversion takes a byte (two codes, low nibble -> low half).
__device__ __forceinline__ void cvt_e2m1x8_f16(uint32_t w, uint32_t (&v)[4]) {
  asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
      "mov.b32 {b0, b1, b2, b3}, %4;\n\t"
      "cvt.rn.f16x2.e2m1x2 %0, b0;\n\t"
      "cvt.rn.f16x2.e2m1x2 %1, b1;\n\t"
      "cvt.rn.f16x2.e2m1x2 %2, b2;\n\t"
      "cvt.rn.f16x2.e2m1x2 %3, b3;\n\t}\n"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
      : "r"(w));
}

// Eight E2M1 codes -> four bf16x2 words, each value multiplied in BF16 by the bf16 scale pair `sc`
// (power-of-two scales: the product is exact unless it leaves the BF16 range).
__device__ __forceinline__ void cvt_e2m1x8_bf16(uint32_t w, __nv_bfloat162 sc, uint32_t (&out)[4]) {
  uint32_t v[4];
  cvt_e2m1x8_f16(w, v);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&v[j]));
    const __nv_bfloat162 x = __hmul2(__floats2bfloat162_rn(f.x, f.y), sc);
    out[j] = *reinterpret_cast<const uint32_t*>(&x);
  }
}

// Eight E2M1 codes times an E4M3 block scale -> four f16x2 words; `sc` = the scale as an f16x2 pair.
// The product is exact in FP16 (2 + 4 significant bits, between 2^-10 and 2688).
__device__ __forceinline__ void cvt_e2m1x8_scaled_f16(uint32_t w, uint32_t sc, uint32_t (&out)[4]) {
  uint32_t v[4];
  cvt_e2m1x8_f16(w, v);
  const __half2 s2 = *reinterpret_cast<const __half2*>(&sc);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const __half2 r = __hmul2(*reinterpret_cast<const __half2*>(&v[j]), s2);
    out[j] = *reinterpret_cast<const uint32_t*>(&r);
  }
}
// (code x scale has at most six significant bits: exact)
__device__ __forceinline__ uint32_t f16x2_to_bf16x2(uint32_t w) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
  const __nv_bfloat162 b = __floats2bfloat162_rn(f.x, f.y);
  return *reinterpret_cast<const uint32_t*>(&b);
}
// Four E4M3 scale bytes -> two f16x2 words (bytes 0,1 and 2,3; low byte -> low half).
__device__ __forceinline__ void cvt_e4m3x4_f16(uint32_t w, uint32_t& s01, uint32_t& s23) {
  asm("{\n\t.reg .b16 lo, hi;\n\t"
      "mov.b32 {lo, hi}, %2;\n\t"
      "cvt.rn.f16x2.e4m3x2 %0, lo;\n\t"
      "cvt.rn.f16x2.e4m3x2 %1, hi;\n\t}\n"
      : "=r"(s01), "=r"(s23)
      : "r"(w));
}


// kind::f16 instruction descriptor, FP32 accumulation: both operands BF16 or both FP16
__device__ __forceinline__ uint32_t make_idesc_16bit(int m, int n, bool bf16) {
  return make_idesc_bf16(m, n) & (bf16 ? 0xffffffffu : ~((1u << 7) | (1u << 10)));
}

// D[tmem] (+)= A[tmem: 128 weight rows x 16] * B[smem: N token rows x 16]^T, kind::f16
__device__ __forceinline__ void mma_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
      ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_bf16_ts_pair(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                                 uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
      ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

template <int kForm>
__device__ __forceinline__ void init_bars(Bars* bars) {
  using C = Cfg<kForm>;
  for (int s = 0; s < C::kRawStages; ++s) {
    mbar_init(&bars->rfull[s], 1);
    mbar_init(&bars->rempty[s], 4);      // the group that converts the stage
  }
  for (int s = 0; s < kTokStagesMax; ++s) {
    mbar_init(&bars->tfull[s], 1);
    mbar_init(&bars->tempty[s], 1);
  }
  for (int s = 0; s < C::kRing; ++s) {
    mbar_init(&bars->afull[s], C::kPair ? 8 : 4);
    mbar_init(&bars->aempty[s], 1);
  }
  for (int b = 0; b < 2; ++b) {
    mbar_init(&bars->acc_full[b], 1);
    mbar_init(&bars->acc_empty[b], C::kPair ? 2 * kEpiWarps : kEpiWarps);
  }
  fence_mbar_init();
}

// The work of a run, by all threads of the CTA: token tiles of the experts whose mark is `wide`, and the
// CTA's first items.
template <int kForm>
__device__ __forceinline__ void build_work(const Params& p, SmemTail* tail, int wide, int rank, int w_first, int w_stride) {
  using C = Cfg<kForm>;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 32) {
    // token tiles per expert, exclusive prefix sums: every lane takes a contiguous span of experts
    const int per = (p.E + 31) >> 5;
    const int e0 = min(p.E, lane * per), e1 = min(p.E, e0 + per);
    auto tiles = [&](int e) {
      return tail->wide[e] == wide ? (tail->offs[e + 1] - tail->offs[e] + C::kMaxTok - 1) / C::kMaxTok : 0;
    };
    int n = 0, widest = 0, marked = 0;
    for (int e = e0; e < e1; ++e) {
      const int me = tiles(e);
      n += me;
      marked |= tail->wide[e];
      if (me > 0) widest = max(widest, (tail->offs[e + 1] - tail->offs[e] + me - 1) / me);
    }
    widest = __reduce_max_sync(0xffffffffu, widest);
    marked = __reduce_max_sync(0xffffffffu, marked);
    if (lane == 0) {
      tail->max_cols = max((widest + C::kColStep - 1) & ~(C::kColStep - 1), C::kColStep);
      tail->any_wide = marked;
    }
    int incl = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += v;
    }
    int at = incl - n;
    for (int e = e0; e < e1; ++e) {
      tail->tile_base[e] = at;
      at += tiles(e);
    }
    if (lane == 31) tail->tile_base[p.E] = incl;
  }
  __syncthreads();
  const int w = w_first + static_cast<int>(threadIdx.x) * w_stride;
  if (static_cast<int>(threadIdx.x) < kMaxList && w < tail->tile_base[p.E] * p.n_tiles) {
    const Work c = decode_work<kForm>(w, p, tail, rank);
    tail->list[threadIdx.x] = make_int4(c.e, c.nt, c.row0, c.nrows);
  }
  __syncthreads();
}

// All roles over the CTA's items of a run
template <int EPI, int kForm, int kTo>
__device__ __forceinline__ void run_items(const CUtensorMap& tmX64, const CUtensorMap& tmX32, const CUtensorMap& tmX16,
                                          const CUtensorMap& tmW, const Params& p, SmemTail* tail, Bars* bars,
                                          uint8_t* sTok, uint8_t* sRaw, int rank, int w_first, int w_stride) {
  using C = Cfg<kForm>;
  constexpr bool kPair = C::kPair;
  constexpr bool kGated = EPI == EPI_FC1_GATED;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int total_work = tail->tile_base[p.E] * p.n_tiles;
  const uint32_t tmem_base = tail->tmem_base;
  volatile int* abort_flag = &tail->abort_flag;
  // a k-block of the widest tile's token rows (of this CTA's share), k-blocks per stage, stages
  const int tok_kb_bytes = (kPair ? tail->max_cols >> 1 : tail->max_cols) * 128;
  const int tok_kbs = C::kStageKb == 4 && tok_kb_bytes <= 32 * 128 ? 4 : 2;
  const int tok_stages = min(kTokStagesMax, C::kSmemTok / (tok_kbs * tok_kb_bytes));

  if (warp == 0) {
    // ------------------------------ codes + scale atoms (of this CTA's 128 rows) -----------------
    // The packed codes of the two 64-row sub-tiles and the scale atoms of the row groups they lie in (a
    // second group only where a sub-tile straddles two).  One elected thread issues all copies: from
    // divergent lanes every TMA instruction costs tens of clocks more.
    if (elect_one()) {
      tma_prefetch_desc(&tmW);
      int rs = 0;
      uint32_t rphase = 0;
      bool ok = true;
      for (int w = w_first, it = 0; ok && w < total_work; w += w_stride, ++it) {
        const Work c = get_work<kForm>(it, w, p, tail, rank);
        const int nt = min(c.nt, p.n_row_tiles - 1);        // half-empty last pair: load the other half again
        const int r0 = p.sub0_base + nt * p.n_step;
        int r1 = p.sub1_base + nt * p.n_step;
        if (r1 >= p.w_rows) r1 = r0;                         // half-empty last tile
        const int last = p.sf_rowgroups - 1;
        const int g0 = r0 >> 7, g0b = min((r0 + 63) >> 7, last), g1 = r1 >> 7, g1b = min((r1 + 63) >> 7, last);
        const uint32_t n_atoms = 2u + (g0b != g0) + (g1b != g1);
        const uint8_t* sf_e = p.sf + static_cast<size_t>(c.e) * p.sf_rowgroups * p.atoms_k * 512;
        const size_t sf_group = static_cast<size_t>(p.atoms_k) * 512;
        const int y0 = c.e * p.w_rows + r0, y1 = c.e * p.w_rows + r1;
        for (int kb = 0; kb < p.k_blocks; kb += kKBlocksPerRaw) {
          if (!mbar_wait_bounded(&bars->rempty[rs], rphase ^ 1, abort_flag, p.status, WAIT_SMEM_EMPTY)) {
            ok = false;
            break;
          }
          const uint32_t atom_bytes = static_cast<uint32_t>(min(kKBlocksPerRaw, p.atoms_k - kb)) * 512u;
          uint8_t* dst = sRaw + rs * kSmemRaw;
          uint8_t* dst_sf = dst + kSmemCodes;
          const uint8_t* src_sf = sf_e + static_cast<size_t>(kb) * 512;
          uint64_t* bar = &bars->rfull[rs];
          mbar_expect_tx(bar, kSmemCodes + n_atoms * atom_bytes);
          tma_load_2d(dst, &tmW, bar, kb * 32, y0);
          tma_load_2d(dst + kSmemCodes / 2, &tmW, bar, kb * 32, y1);
          bulk_load(dst_sf, src_sf + g0 * sf_group, atom_bytes, bar);
          bulk_load(dst_sf + 2 * 2048, src_sf + g1 * sf_group, atom_bytes, bar);
          if (g0b != g0) bulk_load(dst_sf + 2048, src_sf + g0b * sf_group, atom_bytes, bar);
          if (g1b != g1) bulk_load(dst_sf + 3 * 2048, src_sf + g1b * sf_group, atom_bytes, bar);
          if (++rs == C::kRawStages) {
            rs = 0;
            rphase ^= 1;
          }
        }
      }
      if (!ok) {
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);   // let copies in flight land
      }
    }
  } else if (warp == 2) {
    // ------------------------------ token rows (pair: this CTA's half of the columns) ------------
    // a box of 64 or 32 rows and one of 16 (either may be missing) of each k-block of a stage
    if (elect_one()) {
      tma_prefetch_desc(&tmX64);
      tma_prefetch_desc(&tmX32);
      tma_prefetch_desc(&tmX16);
      int ts = 0;
      uint32_t tphase = 0;
      bool ok = true;
      for (int w = w_first, it = 0; ok && w < total_work; w += w_stride, ++it) {
        const Work c = get_work<kForm>(it, w, p, tail, rank);
        const int rows = kPair ? c.cols >> 1 : c.cols;       // 16, 32, 48, 64 or 80
        const int big = rows >= 64 ? 64 : (rows & 32);
        const CUtensorMap* tm = big == 64 ? &tmX64 : &tmX32;
        const int y = c.row0 + (kPair ? rank * rows : 0);
        for (int kb = 0; kb < p.k_blocks; kb += tok_kbs) {
          if (!mbar_wait_bounded(&bars->tempty[ts], tphase ^ 1, abort_flag, p.status, WAIT_SMEM_EMPTY)) {
            ok = false;
            break;
          }
          const int nk = min(tok_kbs, p.k_blocks - kb);
          if (rank == 0) mbar_expect_tx(&bars->tfull[ts], static_cast<uint32_t>(c.cols * 128 * nk));
          const uint32_t bar = kPair ? map_to_cta(smem_u32(&bars->tfull[ts]), 0) : 0u;
          for (int kq = 0; kq < nk; ++kq) {
            const int x = (kb + kq) * kKPerBlock;
            uint8_t* dst = sTok + (tok_kbs * ts + kq) * tok_kb_bytes;
            if (big != 0) {
              if (kPair) tma_load_2d_pair(dst, tm, bar, x, y);
              else tma_load_2d(dst, tm, &bars->tfull[ts], x, y);
            }
            if (rows != big) {
              if (kPair) tma_load_2d_pair(dst + big * 128, &tmX16, bar, x, y + big);
              else tma_load_2d(dst + big * 128, &tmX16, &bars->tfull[ts], x, y + big);
            }
          }
          if (++ts == tok_stages) {
            ts = 0;
            tphase ^= 1;
          }
        }
      }
      if (!ok) {
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (the even CTA's, in a pair) ------------------------
    if (rank == 0 && elect_one()) {
      int ts = 0, as = 0, buf = 0;
      uint32_t tphase = 0, aphase = 0;
      uint32_t acc_phase[2] = {0, 0};
      bool ok = true;
      const uint64_t bdesc0 = make_desc_sw128(smem_u32(sTok));
      for (int w = w_first, it = 0; ok && w < total_work; w += w_stride, ++it) {
        const Work c = get_work<kForm>(it, w, p, tail, rank);
        const uint32_t idesc = make_idesc_16bit(kPair ? 256 : 128, c.cols, kTo != TO_F16);
        if (!mbar_wait_bounded(&bars->acc_empty[buf], acc_phase[buf] ^ 1, abort_flag, p.status, WAIT_TMEM_EMPTY)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + buf * C::kMaxTok;
        // kU k-blocks per pass: one token stage, a whole converted stage or half of one
        auto main_loop = [&](auto units) {
          constexpr int kU = decltype(units)::value;
          for (int kb = 0; kb < p.k_blocks; kb += kU) {
            const bool first_of_a = kU == C::kStageKb || kb % C::kStageKb == 0;
            if ((first_of_a && !mbar_wait_bounded(&bars->afull[as], aphase, abort_flag, p.status, WAIT_CONVERT)) ||
                !mbar_wait_bounded(&bars->tfull[ts], tphase, abort_flag, p.status, WAIT_SMEM_FULL)) {
              ok = false;
              break;
            }
            tc_fence_after();
            uint64_t bdesc = bdesc0 + static_cast<uint32_t>(kU * ts * (tok_kb_bytes >> 4));
            const uint32_t a = tmem_base + C::kRingCol + as * C::kStageCols +
                               (kU == C::kStageKb ? 0 : (kb % C::kStageKb) * 32);
            const int nk = min(kU, p.k_blocks - kb);
            // 16 values of K = 8 TMEM columns of A, 32 bytes of B per MMA
#pragma unroll
            for (int kq = 0; kq < kU; ++kq) {
              if (kq < nk) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  const uint32_t accum = (kq > 0 || j > 0) ? 1u : (kb > 0 ? 1u : 0u);
                  if (kPair) mma_bf16_ts_pair(d_tmem, a + 32 * kq + 8 * j, bdesc + 2 * j, idesc, accum);
                  else mma_bf16_ts(d_tmem, a + 32 * kq + 8 * j, bdesc + 2 * j, idesc, accum);
                }
                bdesc += static_cast<uint32_t>(tok_kb_bytes >> 4);
              }
            }
            if (kPair) tc_commit_pair_both(&bars->tempty[ts]);
            else tc_commit(&bars->tempty[ts]);
            if (++ts == tok_stages) {
              ts = 0;
              tphase ^= 1;
            }
            if (kU == C::kStageKb || (kb + kU) % C::kStageKb == 0 || kb + kU >= p.k_blocks) {
              if (kPair) tc_commit_pair_both(&bars->aempty[as]);
              else tc_commit(&bars->aempty[as]);
              if (++as == C::kRing) {
                as = 0;
                aphase ^= 1;
              }
            }
          }
        };
        if (tok_kbs == 4) main_loop(std::integral_constant<int, C::kStageKb>{});
        else main_loop(std::integral_constant<int, 2>{});
        if (ok) {
          if (kPair) tc_commit_pair_both(&bars->acc_full[buf]);
          else tc_commit(&bars->acc_full[buf]);
        }
        acc_phase[buf] ^= 1;
        buf ^= 1;
      }
    }
  } else if (warp >= 4 && warp < 4 + kConvWarps) {
    // ------------------------------ converters (both CTAs of a pair) ------------------------------
    const int group = (warp - 4) >> 2, sub = warp & 3;
    // this lane's weight row inside the staged 128: sub-tile 0 = rows 0..63, sub-tile 1 = 64..127
    const int row = kGated ? 16 * sub + (lane & 15) + 64 * (lane >> 4) : 32 * sub + lane;
    const uint32_t a_lane = tmem_base + C::kRingCol + (static_cast<uint32_t>(sub * 32) << 16);
    const uint32_t afull0 = kPair ? map_to_cta(smem_u32(&bars->afull[0]), 0) : 0u;
    const uint32_t chunk_xor = static_cast<uint32_t>(row & 7) << 4;
    const int n_raw = (p.k_blocks + kKBlocksPerRaw - 1) / kKBlocksPerRaw, n_stages = (p.k_blocks + C::kStageKb - 1) / C::kStageKb;
    uint32_t raw0 = 0, stage0 = 0;   // raw stages and MMA stages before this tile
    bool ok = true;
    for (int w = w_first, it = 0; ok && w < total_work; w += w_stride, ++it) {
      const Work c = get_work<kForm>(it, w, p, tail, rank);
      const int nt = min(c.nt, p.n_row_tiles - 1);
      const int r0 = p.sub0_base + nt * p.n_step;
      int r1 = p.sub1_base + nt * p.n_step;
      if (r1 >= p.w_rows) r1 = r0;
      const int first = row < 64 ? r0 : r1;
      const int wrow = first + (row & 63);                 // weight row inside the expert
      const int slot = (row >> 6) * 2 + (wrow >> 7) - (first >> 7);
      const uint32_t sf_off = kSmemCodes + min(slot, 3) * 2048 + (wrow & 31) * 16 + ((wrow >> 5) & 3) * 4;
      // the two groups take the raw stages in turn
      for (int r = (group + raw0) & 1; r < n_raw; r += kConvGroups) {
        const uint32_t rs = (raw0 + r) % C::kRawStages, rphase = ((raw0 + r) / C::kRawStages) & 1u;
        if (!mbar_wait_bounded(&bars->rfull[rs], rphase, abort_flag, p.status, WAIT_CONVERT)) {
          ok = false;
          break;
        }
        const uint8_t* raw = sRaw + rs * kSmemRaw;
        const uint8_t* codes = raw + row * 128;
        const int nk = min(kKBlocksPerRaw, p.k_blocks - r * kKBlocksPerRaw);
#pragma unroll
        for (int q = 0; q < kKBlocksPerRaw / C::kStageKb; ++q) {   // the one or two MMA stages of the raw stage
          if (C::kStageKb * q >= nk) break;
          const uint32_t si = stage0 + (kKBlocksPerRaw / C::kStageKb) * r + q;
          const uint32_t as = si % C::kRing, aphase = (si / C::kRing) & 1u;
          if (!mbar_wait_bounded(&bars->aempty[as], aphase ^ 1, abort_flag, p.status, WAIT_CONVERT)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_t = a_lane + as * C::kStageCols;
          // the k-blocks of the stage (missing ones: unread values); the next one's codes are fetched
          // ahead of this one's stores
          const int k0 = C::kStageKb * q;
          uint4 nx0 = *reinterpret_cast<const uint4*>(codes + (static_cast<uint32_t>(2 * k0 << 4) ^ chunk_xor));
          uint4 nx1 = *reinterpret_cast<const uint4*>(codes + (static_cast<uint32_t>((2 * k0 + 1) << 4) ^ chunk_xor));
          uint32_t nsf = *reinterpret_cast<const uint32_t*>(raw + sf_off + k0 * 512);
#pragma unroll
          for (int hk = 0; hk < C::kStageKb; ++hk) {
            const uint4 cw[2] = {nx0, nx1};
            const uint32_t sfw = nsf;
            if (hk + 1 < C::kStageKb) {
              nx0 = *reinterpret_cast<const uint4*>(codes + (static_cast<uint32_t>(2 * (k0 + hk + 1) << 4) ^ chunk_xor));
              nx1 = *reinterpret_cast<const uint4*>(codes + (static_cast<uint32_t>((2 * (k0 + hk + 1) + 1) << 4) ^ chunk_xor));
              nsf = *reinterpret_cast<const uint32_t*>(raw + sf_off + (k0 + hk + 1) * 512);
            }
            uint32_t s01 = 0, s23 = 0;
            if (kTo != TO_BF16_E8M0) cvt_e4m3x4_f16(sfw, s01, s23);
#pragma unroll
            for (int h = 0; h < 2; ++h) {                    // 32 codes -> 16 TMEM columns
              const uint4 v = cw[h];
              const uint32_t words[4] = {v.x, v.y, v.z, v.w};
              uint32_t out[16];
#pragma unroll
              for (int b = 0; b < 2; ++b) {                  // 16 values per scale
                uint32_t o0[4], o1[4];
                if (kTo != TO_BF16_E8M0) {
                  const uint32_t sc = __byte_perm(h == 0 ? s01 : s23, 0u, b == 0 ? 0x1010u : 0x3232u);
                  cvt_e2m1x8_scaled_f16(words[2 * b], sc, o0);
                  cvt_e2m1x8_scaled_f16(words[2 * b + 1], sc, o1);
                } else {
                  const uint32_t sb = (sfw >> (16 * h + 8 * b)) & 0xffu;
                  // E8M0: 2^(b-127) is the f32 with exponent field b (b = 0: the subnormal 2^-127)
                  const __nv_bfloat16 s1 = __float2bfloat16_rn(__uint_as_float(sb != 0u ? sb << 23 : 0x00400000u));
                  const __nv_bfloat162 sc = __halves2bfloat162(s1, s1);
                  cvt_e2m1x8_bf16(words[2 * b], sc, o0);
                  cvt_e2m1x8_bf16(words[2 * b + 1], sc, o1);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  out[8 * b + i] = o0[i];
                  out[8 * b + 4 + i] = o1[i];
                }
              }
              if (kTo == TO_BF16_E4M3) {
#pragma unroll
                for (int i = 0; i < 16; ++i) out[i] = f16x2_to_bf16x2(out[i]);
              }
              tc_st_32x32b_x16(a_t + 32 * hk + 16 * h, out);
            }
          }
          tc_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            if (kPair) mbar_arrive_cluster(afull0 + as * static_cast<uint32_t>(sizeof(uint64_t)));
            else mbar_arrive(&bars->afull[as]);
          }
        }
        // this warp has read all it needs of the stage's codes and atoms
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->rempty[rs]);
      }
      raw0 += n_raw;
      stage0 += n_stages;
    }
  } else if (warp >= 4 + kConvWarps) {
    // ------------------------------ epilogue (both CTAs of a pair) --------------------------------
    // the two warps of a sub-partition take every other 32 token columns (FC1) / 16 (FC2)
    const int sub = warp & 3, half = (warp - 4 - kConvWarps) >> 2;
    const uint32_t release0 = kPair ? map_to_cta(smem_u32(&bars->acc_empty[0]), 0) : 0u;
    uint32_t acc_phase[2] = {0, 0};
    int buf = 0;
    for (int w = w_first, it = 0; w < total_work; w += w_stride, ++it) {
      const Work c = get_work<kForm>(it, w, p, tail, rank);
      const float alpha = p.alphas[c.e];
      // lane l holds the factors of token t + l of the warp's next 32 (FC2: 16) columns; the first are
      // fetched before the accumulator is waited for
      const int t_first = EPI == EPI_FC2 ? 16 * half : 32 * half;
      auto row_of = [&](int t) {
        return c.row0 + min(t + (EPI == EPI_FC2 ? (lane & 15) : lane), c.nrows - 1);
      };
            float inv_next = kTo == TO_F16 ? p.row_inv[row_of(t_first)] : 1.0f;
      if (!mbar_wait_idle(&bars->acc_full[buf], acc_phase[buf], abort_flag, p.status, WAIT_TMEM_FULL)) break;
      acc_phase[buf] ^= 1;
      tc_fence_after();
      const uint32_t t_lane = tmem_base + buf * C::kMaxTok + (static_cast<uint32_t>(sub * 32) << 16);
      // the output column of this lane
      const int col = kGated ? c.nt * 64 + 16 * sub + (lane & 15) : c.nt * 128 + 32 * sub + lane;
      const bool col_ok = c.nt < p.n_row_tiles && col < p.out_cols;
      if (EPI == EPI_FC2) {
        for (int ch = 16 * half; ch < c.cols; ch += 32) {
          uint32_t r[16];
          tc_ld_32x32b_x16(t_lane + ch, r);
          tc_wait_ld();
          const float inv_l = inv_next;
          if (kTo == TO_F16 && ch + 32 < c.cols) inv_next = p.row_inv[row_of(ch + 32)];
          float* o = p.out_f32 + static_cast<size_t>(c.row0 + ch) * p.out_cols + col;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float v = __uint_as_float(r[i]);
            if (kTo == TO_F16) v = __fmul_rn(v, __shfl_sync(0xffffffffu, inv_l, i));
            if (col_ok && ch + i < c.nrows) o[static_cast<size_t>(i) * p.out_cols] = __fmul_rn(v, alpha);
          }
        }
      } else {
        for (int t0 = 32 * half; t0 < c.cols; t0 += 64) {
          const float inv_l = inv_next;
          if (kTo == TO_F16 && t0 + 64 < c.cols) inv_next = p.row_inv[row_of(t0 + 64)];
          const float al_l = p.route_weights != nullptr
                                 ? __fmul_rn(alpha, p.route_weights[p.sorted_route_ids[row_of(t0)]]) : alpha;
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int ch = t0 + 16 * q;
            if (ch >= c.cols) break;
            uint32_t r[16];
            tc_ld_32x32b_x16(t_lane + ch, r);
            tc_wait_ld();
            if (EPI == EPI_FC1_RELU2) {
#pragma unroll
              for (int i = 0; i < 16; ++i) {
                const float inv = __shfl_sync(0xffffffffu, inv_l, 16 * q + i);
                const float al = __shfl_sync(0xffffffffu, al_l, 16 * q + i);
                if (col_ok && ch + i < c.nrows) {
                  const size_t pos = static_cast<size_t>(c.row0 + ch + i);
                  float v = __uint_as_float(r[i]);
                  if (kTo == TO_F16) v = __fmul_rn(v, inv);
                  v = __fmul_rn(v, al);
                  if (p.tap != nullptr) p.tap[pos * p.w_rows + col] = v;
                  const float z = fmaxf(v, 0.f);
                  p.out_bf16[pos * p.out_cols + col] = __float2bfloat16_rn(__fmul_rn(z, z));
                }
              }
            } else {
              // lanes 0..15 hold up values, lanes 16..31 the gate values of the same columns, of 16
              // tokens: the lower lanes finish tokens 0..7, the upper lanes tokens 8..15
              const bool upper = lane >= 16;
              const int tok0 = upper ? 8 : 0;
              uint32_t pk[4];
#pragma unroll
              for (int i2 = 0; i2 < 4; ++i2) {
                float h[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                  const int i = 2 * i2 + k;
                  const uint32_t got = __shfl_xor_sync(0xffffffffu, upper ? r[i] : r[8 + i], 16);
                  float up = __uint_as_float(upper ? got : r[i]), gate = __uint_as_float(upper ? r[8 + i] : got);
                  if (kTo == TO_F16) {
                    const float inv = __shfl_sync(0xffffffffu, inv_l, 16 * q + tok0 + i);
                    up = __fmul_rn(up, inv);
                    gate = __fmul_rn(gate, inv);
                  }
                  const float al = p.route_weights != nullptr ? __shfl_sync(0xffffffffu, al_l, 16 * q + tok0 + i) : alpha;
                  up = __fmul_rn(up, al);
                  gate = __fmul_rn(gate, al);
                  if (p.tap != nullptr && col_ok && ch + tok0 + i < c.nrows) {
                    float* trow = p.tap + static_cast<size_t>(c.row0 + ch + tok0 + i) * p.w_rows + col;
                    trow[p.sub0_base] = up;
                    trow[p.sub1_base] = gate;
                  }
                  h[k] = act_gated(gate, up, p);
                }
                const __nv_bfloat162 b2 = __floats2bfloat162_rn(h[0], h[1]);
                pk[i2] = *reinterpret_cast<const uint32_t*>(&b2);
              }
              // neighbouring lanes hold neighbouring columns: the even lane stores both columns of its
              // first four tokens, the odd lane of the last four (4 bytes instead of twice 2)
              const bool odd = lane & 1;
              const uint32_t g0 = __shfl_xor_sync(0xffffffffu, odd ? pk[0] : pk[2], 1);
              const uint32_t g1 = __shfl_xor_sync(0xffffffffu, odd ? pk[1] : pk[3], 1);
              const uint32_t a0 = odd ? g0 : pk[0], b0 = odd ? pk[2] : g0;     // tokens 0, 1 of the four; even / odd column
              const uint32_t a1 = odd ? g1 : pk[1], b1 = odd ? pk[3] : g1;     // tokens 2, 3
              const uint32_t out[4] = {__byte_perm(a0, b0, 0x5410), __byte_perm(a0, b0, 0x7632),
                                       __byte_perm(a1, b1, 0x5410), __byte_perm(a1, b1, 0x7632)};
              const int tok = ch + tok0 + (odd ? 4 : 0);
              if (col_ok) {
                __nv_bfloat16* o = p.out_bf16 + static_cast<size_t>(c.row0 + tok) * p.out_cols + (col & ~1);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                  if (tok + i < c.nrows) *reinterpret_cast<uint32_t*>(o + static_cast<size_t>(i) * p.out_cols) = out[i];
              }
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (kPair) mbar_arrive_cluster(release0 + static_cast<uint32_t>(buf * sizeof(uint64_t)));
        else mbar_arrive(&bars->acc_empty[buf]);
      }
      buf ^= 1;
    }
  }
}

// The run of the marked experts, on BF16 operands.  The other run has ended, here and in the other CTA of a pair; its
// barriers may still be signalled by commits that nobody waits for, so this one has a set of its own.
template <int EPI, int kForm>
__device__ __noinline__ void run_wide_items(const CUtensorMap& tmB64, const CUtensorMap& tmB32, const CUtensorMap& tmB16,
                                            const CUtensorMap& tmW, const Params& p, SmemTail* tail, uint8_t* sTok,
                                            uint8_t* sRaw, int rank, int w_first, int w_stride) {
  if (threadIdx.x == 0) init_bars<kForm>(&tail->bars[1]);
  tc_fence_before();
  __syncthreads();
  build_work<kForm>(p, tail, 1, rank, w_first, w_stride);
  if (Cfg<kForm>::kPair) cluster_sync_all();
  tc_fence_after();
  run_items<EPI, kForm, TO_BF16_E4M3>(tmB64, tmB32, tmB16, tmW, p, tail, &tail->bars[1], sTok, sRaw, rank, w_first, w_stride);
}

// tmX*: the token rows as kTo says, boxes of 64, 32 and 16 rows; tmB*: TO_F16: the same rows as BF16
template <int EPI, int kForm, int kTo>
__global__ void __launch_bounds__(kThreads, 1)
grouped_gemm_w4a16_kernel(const __grid_constant__ CUtensorMap tmX64, const __grid_constant__ CUtensorMap tmX32,
                          const __grid_constant__ CUtensorMap tmX16, const __grid_constant__ CUtensorMap tmB64,
                          const __grid_constant__ CUtensorMap tmB32, const __grid_constant__ CUtensorMap tmB16,
                          const __grid_constant__ CUtensorMap tmW, const __grid_constant__ Params p) {
  using C = Cfg<kForm>;
  constexpr bool kPair = C::kPair;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sTok = smem;
  uint8_t* sRaw = sTok + C::kSmemTok;
  SmemTail* tail = reinterpret_cast<SmemTail*>(sRaw + C::kRawStages * kSmemRaw);
  const int warp = threadIdx.x >> 5;
  const int rank = kPair ? static_cast<int>(cluster_ctarank()) : 0;

  if (threadIdx.x == 0) {
    tail->abort_flag = 0;
    init_bars<kForm>(&tail->bars[0]);
  }
  for (int i = threadIdx.x; i <= p.E; i += kThreads) {
    tail->offs[i] = p.expert_offsets[i];
    if (i < p.E) tail->wide[i] = kTo == TO_F16 && p.wide[i] != 0;
  }
  if (warp == 1) {
    if (kPair) {
      tmem_alloc_pair(&tail->tmem_base, kTmemCols);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(&tail->tmem_base, kTmemCols);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  const int w_first = kPair ? static_cast<int>(blockIdx.x) >> 1 : static_cast<int>(blockIdx.x);
  const int w_stride = kPair ? static_cast<int>(gridDim.x) >> 1 : static_cast<int>(gridDim.x);
  build_work<kForm>(p, tail, 0, rank, w_first, w_stride);
  if (kPair) cluster_sync_all();   // both CTAs' barriers are initialised before anyone signals them
  tc_fence_after();
  run_items<EPI, kForm, kTo>(tmX64, tmX32, tmX16, tmW, p, tail, &tail->bars[0], sTok, sRaw, rank, w_first, w_stride);

  if (kTo == TO_F16 && tail->any_wide != 0) {
    // the marked experts' items go round on from where the others ended: CTAs short of an item take one first
    const int first = (w_first + w_stride - tail->tile_base[p.E] * p.n_tiles % w_stride) % w_stride;
    tc_fence_before();
    __syncthreads();
    if (kPair) cluster_sync_all();
    run_wide_items<EPI, kForm>(tmB64, tmB32, tmB16, tmW, p, tail, sTok, sRaw, rank, first, w_stride);
  }

  // ------------------------------ teardown ------------------------------------
  tc_fence_before();
  __syncthreads();
  if (kPair) cluster_sync_all();   // nobody signals the other CTA's shared memory after this
  if (warp == 1) {
    const uint32_t tmem_base = tail->tmem_base;
    tc_fence_after();
    if (kPair) tmem_dealloc_pair(tmem_base, kTmemCols);
    else tmem_dealloc(tmem_base, kTmemCols);
  }
}

// Calibration side channel of the w4a16 recipe (reference W4A16FusedMoeKernel._collect_activation_amax_epilogue,
// b12x/moe/_shared/kernels/w4a16/kernel.py:7288-7365): amax[layer][expert][0] = max(old, max |x| over the
// rows routed to the expert), [..][1] the same over its activated BF16 intermediate rows.  One CTA per
// row tile and operand (blockIdx.y: 0 = FC1 input rows, 1 = FC2 input rows); non-negative floats
// order like their bit patterns, so the running maximum is an integer atomicMax.
__global__ void __launch_bounds__(256) activation_amax_kernel(
    const __nv_bfloat16* __restrict__ rows_fc1, const __nv_bfloat16* __restrict__ rows_fc2, int K, int I,
    const int32_t* __restrict__ tile_base, int E, const int32_t* __restrict__ mtile_expert,
    const int32_t* __restrict__ mtile_row0, const int32_t* __restrict__ mtile_rows, float* __restrict__ amax,
    int layer_idx) {
  const int mt = blockIdx.x;
  if (mt >= tile_base[E]) return;
  const int which = blockIdx.y;
  const int len = which == 0 ? K : I;
  const __nv_bfloat16* base = (which == 0 ? rows_fc1 : rows_fc2) + static_cast<size_t>(mtile_row0[mt]) * len;
  const int nvec = (mtile_rows[mt] * len) >> 3;                 // 8 values per 16-byte load; rows are contiguous
  float m = 0.f;
  for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
    const uint4 p = reinterpret_cast<const uint4*>(base)[i];
    const uint32_t w[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      m = fmaxf(m, fabsf(__uint_as_float(w[j] << 16)));
      m = fmaxf(m, fabsf(__uint_as_float(w[j] & 0xffff0000u)));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  __shared__ float part[8];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int wgt = 1; wgt < 8; ++wgt) m = fmaxf(m, part[wgt]);
    if (!(m != m)) {      // a NaN row leaves the record alone
      int* dst = reinterpret_cast<int*>(amax + (static_cast<size_t>(layer_idx) * E + mtile_expert[mt]) * 2 + which);
      atomicMax(dst, __float_as_int(m));
    }
  }
}

// x rows -> sorted-position order (the token operand of FC1), one warp per row
__global__ void __launch_bounds__(256) permute_rows_bf16_kernel(
    const __nv_bfloat16* __restrict__ x, int64_t x_row_stride, const int32_t* __restrict__ expert_offsets,
    int E, const int32_t* __restrict__ sorted_route_ids, int num_topk, int K,
    __nv_bfloat16* __restrict__ out) {
  const int total = expert_offsets[E];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int pos = blockIdx.x * 8 + warp; pos < total; pos += gridDim.x * 8) {
    const int tkn = sorted_route_ids[pos] / num_topk;
    const uint4* src = reinterpret_cast<const uint4*>(x + static_cast<int64_t>(tkn) * x_row_stride);
    uint4* dst = reinterpret_cast<uint4*>(out + static_cast<size_t>(pos) * K);
    for (int j = lane; j < (K >> 3); j += 32) dst[j] = __ldg(src + j);
  }
}

// The same, and the rows once more as FP16 (rows_bf16 and sorted_route_ids null: rows that lie in sorted order
// already, FC2's, as FP16 only), each multiplied by the power of two that puts its largest finite magnitude
// into [2^15, 2^16); row_inv[pos] takes the inverse.  BF16 has 8 significant bits: every value down to 2^-32
// of the row's largest binade is carried over exactly.  A row with smaller ones marks its expert `wide`
// (a mark too many is still right: such an expert's GEMMs run on the BF16 rows, at a lower rate; the sort clears
// the marks).  Infinities and NaNs stay what they are.
//
// Bound by its bytes for many rows (FC1, 32768 of 4096: 125 us for 268 MB read and 537 MB written, about 70 us
// without the BF16 copy), by the latency of one row's two passes for few: there the eight warps of a CTA share a
// row (512 rows of 14336: 34 -> 8 us).
template <int kWarps, bool kCopy>
__global__ void __launch_bounds__(256) permute_rows_f16_kernel(
    const __nv_bfloat16* __restrict__ x, int64_t x_row_stride, const int32_t* __restrict__ expert_offsets,
    int E, const int32_t* __restrict__ sorted_route_ids, int num_topk, int K,
    __nv_bfloat16* __restrict__ rows_bf16, __half* __restrict__ out, float* __restrict__ row_inv,
    int32_t* __restrict__ wide) {
  __shared__ uint32_t part_most[8];
  __shared__ int part_least[8];
  const int total = expert_offsets[E];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nvec = K >> 3, first = lane + 32 * (warp % kWarps);
  constexpr int kRows = 8 / kWarps, kStep = 32 * kWarps;
  // over the warps of the row (all threads of the CTA in step, if they share one)
  auto row_max = [&](uint32_t v) -> uint32_t {
    v = __reduce_max_sync(0xffffffffu, v);
    if (kWarps == 1) return v;
    __syncthreads();
    if (lane == 0) part_most[warp] = v;
    __syncthreads();
    for (int i = 0; i < kWarps; ++i) v = max(v, part_most[i]);
    return v;
  };
  auto row_min = [&](int v) -> int {
    v = __reduce_min_sync(0xffffffffu, v);
    if (kWarps == 1) return v;
    __syncthreads();
    if (lane == 0) part_least[warp] = v;
    __syncthreads();
    for (int i = 0; i < kWarps; ++i) v = min(v, part_least[i]);
    return v;
  };
  for (int pos = blockIdx.x * kRows + warp / kWarps; pos < total; pos += gridDim.x * kRows) {
    const int tkn = sorted_route_ids != nullptr ? sorted_route_ids[pos] / num_topk : pos;
    const uint4* src = reinterpret_cast<const uint4*>(x + static_cast<int64_t>(tkn) * x_row_stride);
    uint4* copy = kCopy ? reinterpret_cast<uint4*>(rows_bf16 + static_cast<size_t>(pos) * K) : nullptr;
    __nv_bfloat162 m2 = __float2bfloat162_rn(0.f);
    // smallest nonzero magnitude: + 0x7fff takes 0 to the largest signed 16-bit value and keeps the others in order
    uint32_t least2 = 0x7fff7fffu;
#pragma unroll 4
    for (int j = first; j < nvec; j += kStep) {
      const uint4 v = __ldg(src + j);
      if (kCopy) copy[j] = v;
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        m2 = __hmax2(m2, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[i])));
        least2 = __vmins2(least2, (w[i] & 0x7fff7fffu) + 0x7fff7fffu);
      }
    }
    // BF16 magnitudes order like their bits
    uint32_t m = row_max(static_cast<uint32_t>(max(__bfloat16_as_ushort(__low2bfloat16(m2)),
                                                   __bfloat16_as_ushort(__high2bfloat16(m2)))));
    if (m >= 0x7f80u) {            // an infinity: once more over the finite values
      m = 0;
      for (int j = first; j < nvec; j += kStep) {
        const uint4 v = __ldg(src + j);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t lo = w[i] & 0x7fffu, hi = (w[i] >> 16) & 0x7fffu;
          if (lo < 0x7f80u) m = max(m, lo);
          if (hi < 0x7f80u) m = max(m, hi);
        }
      }
      m = row_max(m);
    }
    // exponent field e of the largest: x 2^(142 - e), the factor kept a normal float either way
    const int sh = min(142 - max(static_cast<int>(m >> 7), 1), 126);
    const float scale = __uint_as_float(static_cast<uint32_t>(127 + sh) << 23);
    // the last bit of a value with exponent field f is 2^(f - 134 + sh) of the FP16 row, whose last is 2^-24
    const int least = row_min(min(static_cast<int>(static_cast<int16_t>(least2 & 0xffffu)),
                                  static_cast<int>(least2) >> 16)) + 0x8001;
    if (first == 0) {
      row_inv[pos] = __uint_as_float(static_cast<uint32_t>(127 - sh) << 23);
      if (max(least >> 7, 1) + sh < 110) {
        int lo = 0, hi = E - 1;      // the expert of the row: the last whose first row is not behind it
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (expert_offsets[mid] <= pos) lo = mid; else hi = mid - 1;
        }
        wide[lo] = 1;
      }
    }
    uint4* dst = reinterpret_cast<uint4*>(out + static_cast<size_t>(pos) * K);
#pragma unroll 4
    for (int j = first; j < nvec; j += kStep) {
      const uint4 v = __ldg(src + j);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
      uint32_t o[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const __half2 h = __floats2half2_rn(__fmul_rn(__uint_as_float(w[i] << 16), scale),
                                            __fmul_rn(__uint_as_float(w[i] & 0xffff0000u), scale));
        o[i] = *reinterpret_cast<const uint32_t*>(&h);
      }
      dst[j] = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

// copy: the rows as BF16 too (FC1; null for rows that lie in sorted order already)
static int launch_rows_f16(int rows, const __nv_bfloat16* x, int64_t x_row_stride, const int32_t* expert_offsets, int E,
                           const int32_t* sorted_route_ids, int num_topk, int K, __nv_bfloat16* copy, __half* out,
                           float* row_inv, int32_t* wide, cudaStream_t s) {
  constexpr int kFull = 148 * 8;                       // CTAs of 256 threads that run at once
  auto kern = rows <= kFull ? (copy != nullptr ? permute_rows_f16_kernel<8, true> : permute_rows_f16_kernel<8, false>)
                            : (copy != nullptr ? permute_rows_f16_kernel<1, true> : permute_rows_f16_kernel<1, false>);
  const int grid = rows <= kFull ? rows : ((rows + 7) / 8 < kFull ? (rows + 7) / 8 : kFull);
  kern<<<grid, 256, 0, s>>>(x, x_row_stride, expert_offsets, E, sorted_route_ids, num_topk, K, copy, out, row_inv, wide);
  return cudaGetLastError() == cudaSuccess ? B200MOE_OK : B200MOE_ECUDA;
}

// 2-D bf16 matrix [rows][cols], box = box_rows x 64 elements (128 bytes), 128-byte swizzle
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) ==
            cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}
static int make_tmap_bf16(CUtensorMap* out, const void* base, uint64_t cols, uint64_t rows,
                          uint32_t box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return B200MOE_ECUDA;
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || ((cols * 2) & 15) != 0) return B200MOE_EALIGN;
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {cols * 2};
  const cuuint32_t box[2] = {64, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims,
                        strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? B200MOE_OK : B200MOE_ECUDA;
}

template <int EPI, int kForm, int kTo>
static int launch(const CUtensorMap (&tmX)[6], const CUtensorMap& tmW, const Params& p, int ctas, cudaStream_t s) {
  constexpr bool kPair = Cfg<kForm>::kPair;
  auto kern = grouped_gemm_w4a16_kernel<EPI, kForm, kTo>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes<kForm>()) != cudaSuccess)
    return B200MOE_ECUDA;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = kPair ? 2 : 1;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.gridDim = dim3(static_cast<unsigned>(kPair ? ctas & ~1 : ctas));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem_bytes<kForm>();
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (kPair) {
    // persistent grid: as many CTA pairs as can be resident at once
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess || clusters < 1) return B200MOE_ECUDA;
    if (2 * clusters < static_cast<int>(cfg.gridDim.x)) cfg.gridDim = dim3(static_cast<unsigned>(2 * clusters));
  }
  return cudaLaunchKernelEx(&cfg, kern, tmX[0], tmX[1], tmX[2], tmX[3], tmX[4], tmX[5], tmW, p) == cudaSuccess ? B200MOE_OK : B200MOE_ECUDA;
}

// One CTA up to 18 rows per expert (finer tiles, no partner to wait for), narrow pairs to 58 (nearly every
// expert is one tile of at most 64 columns; one wait of the MMA thread covers 256 rows x 256 values), wide
// pairs beyond.  FC1 + FC2 of the Qwen3 shape, one CTA : narrow : wide, in us: 1 row per expert 185 : 200 :
// 249, 16 rows 283 : 290 : 366, 24 rows 360 : 296 : 368, 48 rows 397 : 323 : 387, 56 rows 447 : 361 : 401,
// 64 rows 564 : 444 : 421, 88 rows 759 : 583 : 454.  The lines lie in the same place elsewhere (layer, us): 128 experts
// of 2880 x 2880, 18 / 24 / 58 / 64 rows 423 / 535 / 701 / 840 : 461 / 473 / 623 / 734 : 543 / 551 / 637 / 674; 256 of
// 7168 x 256 282 / 351 / 576 / 636 : 288 / 318 / 531 / 584 : 317 / 343 / 520 / 538; 8 of 4096 x 3584 88 / 98 / 112 /
// 132 : 96 / 98 / 102 / 115 : 102 / 105 / 111 / 118.
// The rows are the call's, not the plan's capacity: the forms share one scratch layout, and a decode step
// through a workspace planned for a prompt batch (layer, 16 tokens of 4096) took 273 us on wide pairs, 211
// on one CTA.  B200MOE_W4A16_PAIR=1 / 0 forces wide pairs / one CTA (2: narrow pairs); a grid limited to one
// CTA has no pair.
static int form_for(const b200moe_gemm_args* a, int ctas) {
  static int mode = -2;
  if (mode == -2) {
    const char* e = getenv("B200MOE_W4A16_PAIR");
    mode = e == nullptr ? -1 : atoi(e);
  }
  if (ctas < 2) return ONE;
  if (mode >= 0) return mode == 0 ? ONE : (mode == 2 ? PAIR_NARROW : PAIR_WIDE);
  const int64_t rows = static_cast<int64_t>(a->num_tokens) * a->num_topk, experts = a->num_experts;
  return rows < 18 * experts ? ONE : (rows < 58 * experts ? PAIR_NARROW : PAIR_WIDE);
}

template <int EPI, int kTo>
static int launch_any(const b200moe_gemm_args* a, const void* tokens, const void* tokens_bf16, uint64_t cols,
                      const void* weights, Params& p, cudaStream_t s) {
  CUtensorMap tmX[6], tmW;      // the token rows as kTo says, then as BF16
  const uint32_t boxes[3] = {64, 32, 16};
  for (int i = 0; i < 3; ++i) {
    int rc = make_tmap_bf16(&tmX[i], tokens, cols, a->layout->rows, boxes[i]);
    if (rc == B200MOE_OK) rc = make_tmap_bf16(&tmX[3 + i], tokens_bf16, cols, a->layout->rows, boxes[i]);
    if (rc != B200MOE_OK) return rc;
  }
  const int rc = make_tmap_bytes_2d(&tmW, weights, cols / 2, static_cast<uint64_t>(a->num_experts) * p.w_rows, 64);
  if (rc != B200MOE_OK) return rc;
  const int ctas = a->num_sms > 0 ? a->num_sms : num_sms_cached();
  const int form = form_for(a, ctas);
  p.n_tiles = form == ONE ? p.n_row_tiles : ceil_div_i(p.n_row_tiles, 2);
  if (form == ONE) return launch<EPI, ONE, kTo>(tmX, tmW, p, ctas, s);
  if (form == PAIR_NARROW) return launch<EPI, PAIR_NARROW, kTo>(tmX, tmW, p, ctas, s);
  return launch<EPI, PAIR_WIDE, kTo>(tmX, tmW, p, ctas, s);
}

// one warp per row, eight per CTA
static int row_grid(int rows) {
  const int ctas = (rows + 7) / 8;
  return ctas < 148 * 8 ? ctas : 148 * 8;
}

// [2][E]: FC1's and FC2's marks, behind the expert counts
static int32_t* wide_marks(const b200moe_gemm_args* a, char* base) {
  return reinterpret_cast<int32_t*>(base + a->layout->expert_counts) + a->num_experts;
}

static void fill_common(Params& p, const b200moe_gemm_args* a, char* base) {
  const b200moe_scratch_layout& L = *a->layout;
  p.expert_offsets = reinterpret_cast<const int32_t*>(base + L.expert_offsets);
  p.status = reinterpret_cast<int32_t*>(base + L.status);
  p.E = a->num_experts;
  p.limit = a->swiglu_limit;
  p.act_alpha = a->swiglu_alpha;
  p.act_beta = a->swiglu_beta;
  p.swigluoai = a->activation == B200MOE_ACT_SWIGLUOAI;
}

}  // namespace w4a16

int w4a16_gemm1(const b200moe_gemm_args* a, cudaStream_t stream) {
  if (a->activation == B200MOE_ACT_SITU) return B200MOE_EUNSUPPORTED;   // no W4A16 oracle for it
  using namespace w4a16;
  const b200moe_scratch_layout& L = *a->layout;
  const int K = a->hidden_size, I = a->intermediate, E = a->num_experts;
  const bool gated = a->activation != B200MOE_ACT_RELU2;
  if (K % 64 != 0 || I % 16 != 0 || E > kMaxExperts || a->w13_sf == nullptr || a->x == nullptr)
    return B200MOE_EINVAL;
  if ((reinterpret_cast<uintptr_t>(a->x) & 15) != 0 || (a->x_row_stride % 8) != 0) return B200MOE_EALIGN;
  const int w_rows = gated ? 2 * I : I;
  char* base = static_cast<char*>(a->scratch);
  const int rows = a->num_tokens * a->num_topk;
  const int ggrid = row_grid(rows);
  const bool f16 = !a->sf_e8m0;
  const int32_t* offsets = reinterpret_cast<const int32_t*>(base + L.expert_offsets);
  const int32_t* routes = reinterpret_cast<const int32_t*>(base + L.sorted_route_ids);
  int32_t* wide = wide_marks(a, base);
  if (f16) {
    const int rc = launch_rows_f16(rows, static_cast<const __nv_bfloat16*>(a->x), a->x_row_stride, offsets, E, routes,
                                   a->num_topk, K, reinterpret_cast<__nv_bfloat16*>(base + L.act_q),
                                   reinterpret_cast<__half*>(base + L.mid_sf), reinterpret_cast<float*>(base + L.act_sf),
                                   wide, stream);
    if (rc != B200MOE_OK) return rc;
  } else {
    permute_rows_bf16_kernel<<<ggrid, 256, 0, stream>>>(
        static_cast<const __nv_bfloat16*>(a->x), a->x_row_stride, offsets, E, routes, a->num_topk, K,
        reinterpret_cast<__nv_bfloat16*>(base + L.act_q));
  }
  const void* tokens = base + (f16 ? L.mid_sf : L.act_q);
  Params p = {};
  fill_common(p, a, base);
  p.sf = a->w13_sf;
  p.alphas = a->w1_alphas;
  p.out_bf16 = reinterpret_cast<__nv_bfloat16*>(base + L.mid_q);
  p.row_inv = reinterpret_cast<const float*>(base + L.act_sf);
  p.wide = wide;
  p.tap = a->fc1_tap;
  p.route_weights = a->fc1_route_weights;
  p.sorted_route_ids = reinterpret_cast<const int32_t*>(base + L.sorted_route_ids);
  p.k_blocks = K / kKPerBlock;
  p.atoms_k = ceil_div_i(K, 64);
  p.sf_rowgroups = ceil_div_i(w_rows, 128);
  p.w_rows = w_rows;
  p.out_cols = I;
  if (gated) {
    p.n_row_tiles = ceil_div_i(I, 64);
    p.n_step = 64;
    p.sub0_base = a->gate_first ? I : 0;   // up rows
    p.sub1_base = a->gate_first ? 0 : I;   // gate rows
    return f16 ? launch_any<EPI_FC1_GATED, TO_F16>(a, tokens, base + L.act_q, K, a->w13, p, stream)
               : launch_any<EPI_FC1_GATED, TO_BF16_E8M0>(a, tokens, base + L.act_q, K, a->w13, p, stream);
  }
  p.n_row_tiles = ceil_div_i(I, 128);
  p.n_step = 128;
  p.sub0_base = 0;
  p.sub1_base = 64;
  return f16 ? launch_any<EPI_FC1_RELU2, TO_F16>(a, tokens, base + L.act_q, K, a->w13, p, stream)
             : launch_any<EPI_FC1_RELU2, TO_BF16_E8M0>(a, tokens, base + L.act_q, K, a->w13, p, stream);
}

int w4a16_gemm2(const b200moe_gemm_args* a, cudaStream_t stream) {
  using namespace w4a16;
  const b200moe_scratch_layout& L = *a->layout;
  const int K = a->hidden_size, I = a->intermediate, E = a->num_experts;
  if (I % 64 != 0 || K % 16 != 0 || E > kMaxExperts || a->w2_sf == nullptr) return B200MOE_EINVAL;
  char* base = static_cast<char*>(a->scratch);
  Params p = {};
  fill_common(p, a, base);
  p.sf = a->w2_sf;
  p.alphas = a->w2_alphas;
  p.out_f32 = reinterpret_cast<float*>(base + L.routed);
  p.k_blocks = I / kKPerBlock;
  p.atoms_k = ceil_div_i(I, 64);
  p.sf_rowgroups = ceil_div_i(K, 128);
  p.w_rows = K;
  p.out_cols = K;
  p.n_row_tiles = ceil_div_i(K, 128);
  p.n_step = 128;
  p.sub0_base = 0;
  p.sub1_base = 64;
  if (a->sf_e8m0) return launch_any<EPI_FC2, TO_BF16_E8M0>(a, base + L.mid_q, base + L.mid_q, I, a->w2, p, stream);
  // the intermediate rows as FP16, in the place of FC1's
  const int rows = a->num_tokens * a->num_topk;
  float* row_inv = reinterpret_cast<float*>(base + L.act_sf) + L.rows;
  int32_t* wide = wide_marks(a, base) + E;
  const int rc = launch_rows_f16(rows, reinterpret_cast<const __nv_bfloat16*>(base + L.mid_q), I, p.expert_offsets, E,
                                 nullptr, 1, I, nullptr, reinterpret_cast<__half*>(base + L.mid_sf), row_inv, wide, stream);
  if (rc != B200MOE_OK) return rc;
  p.row_inv = row_inv;
  p.wide = wide;
  return launch_any<EPI_FC2, TO_F16>(a, base + L.mid_sf, base + L.mid_q, I, a->w2, p, stream);
}

int w4a16_activation_amax(const b200moe_amax_args* a, cudaStream_t stream) {
  const b200moe_scratch_layout& L = *a->layout;
  char* base = static_cast<char*>(a->scratch);
  const int tr = L.tile_rows == 64 ? 64 : 128;
  const int rows = a->num_rows;
  const int mtiles = (rows + tr - 1) / tr + (a->num_experts < rows ? a->num_experts : rows);
  const int gx = mtiles < L.mtile_cap ? mtiles : L.mtile_cap;
  w4a16::activation_amax_kernel<<<dim3(gx, 2), 256, 0, stream>>>(
      reinterpret_cast<const __nv_bfloat16*>(base + L.act_q), reinterpret_cast<const __nv_bfloat16*>(base + L.mid_q),
      a->hidden_size, a->intermediate, reinterpret_cast<const int32_t*>(base + L.tile_base), a->num_experts,
      reinterpret_cast<const int32_t*>(base + L.mtile_expert), reinterpret_cast<const int32_t*>(base + L.mtile_row0),
      reinterpret_cast<const int32_t*>(base + L.mtile_rows), a->amax, a->layer_idx);
  return cudaGetLastError() == cudaSuccess ? B200MOE_OK : B200MOE_ECUDA;
}

}  // namespace b200moe
