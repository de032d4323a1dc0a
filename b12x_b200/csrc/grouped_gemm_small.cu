// Stages 4 and 5 for small batches (recipes nvfp4 and w4a8_mx): the grouped block-scaled expert GEMMs
// with the operand roles swapped, so that the expert WEIGHTS fill the 128 rows of the tcgen05 tile and
// the few tokens of an expert are its columns.
//
//   tile = two 128-row weight sub-tiles x NT token columns (NT = 16, 32 or 64, chosen per tile
//          from the number of rows the expert received; plans for this kernel cut experts into
//          64-row tiles; w4a8_mx: any multiple of 16 up to 80, see mx_tiles)
//   FC1 (gated):  sub-tile 0 = 128 up rows, sub-tile 1 = the 128 gate rows of the same columns
//                 acc0[i][t], acc1[i][t] -> x alpha1 -> activation -> bf16 -> NVFP4 re-quantise.
//                 A 16-value scale block runs along i, i.e. over 16 lanes: the block maximum is a
//                 warp shuffle reduction, two lanes share an output byte.  (w4a8_mx: 32 values, one
//                 redux.sync over the warp, a byte per lane.)
//   FC2:          sub-tiles = 256 consecutive output features; acc[h][t] x alpha2 -> float32 rows.
//
// Against the wide-tile kernel this reads the same weight bytes, but the accumulators take
// 2 x NT TMEM columns instead of 256 (double-buffered: the epilogue of a tile runs under the main
// loop of the next one), every epilogue warp has work when an expert holds two tokens, and the
// tensor pipe multiplies NT columns instead of 256 mostly empty rows.
//
// Warp roles: warp 0 TMA producer, warp 1 MMA issue, warps 2..9 epilogue, warp 10 (w4a8_mx: 10..13, see
// there) copies the scale atoms of every landed stage into TMEM (tcgen05.cp) and commits them to a
// barrier of their own.  An MMA that follows a tcgen05.cp in the SAME thread's
// instruction stream waits out the copy's latency in the tensor pipe (about 0.15 us per dependent
// MMA, measured); from a separate thread the copies run stages ahead.  Every wait is bounded.
#include <stdlib.h>

#include "gemm_shared.cuh"

namespace b200moe {
namespace small {

constexpr int kRowBytes = 128;                 // one swizzled operand row per stage = 256 values
constexpr int kSmemW = 128 * kRowBytes;        // one weight sub-tile per stage (16 KiB)
constexpr int kTmemCols = 512;
constexpr int kMaxStages = 5;

// nvfp4: 256 values per stage, four MMAs of 64, four scale atoms per operand.  w4a8_mx: 128 values (the
// weight codes expanded to one per byte by the TMA), four MMAs of 32, one scale atom per operand; the
// smaller scale ring makes room for a fifth stage, and 16 KiB of weights per stage need it.
template <int KIND>
struct Cfg {
  static constexpr bool kMx = KIND == KIND_MX;
  static constexpr int kStages = kMx ? 5 : 4;
  static constexpr int kPerStage = kMx ? 128 : 256;
  static constexpr int kPerMma = kMx ? 32 : 64;
  static constexpr int kAtoms = kMx ? 1 : 4;             // per operand and stage
  static constexpr int kSmemSf = kAtoms * 512;
  static constexpr int kMaxTok = kMx ? 80 : 64;          // token columns of a tile (MMA N)
  static constexpr int kSmemX = kMaxTok * kRowBytes;     // token rows per stage
  static constexpr int kAccCols = 2 * kMaxTok;           // one accumulator buffer: two sub-tiles
  static constexpr int kTmemSf = 2 * kAccCols;           // first scale column (two accumulator buffers)
  static constexpr int kSfCols = 12 * kAtoms;            // TMEM columns per stage: sub-tile 0, sub-tile 1, tokens
  // TMA, MMA, 8 epilogue warps, then one scale-copy warp (tcgen05.cp) or four (registers, tcgen05.st)
  static constexpr int kThreads = kMx ? 448 : 352;
};

struct __align__(8) SmemTail {
  uint64_t full[kMaxStages];
  uint64_t empty[kMaxStages];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint64_t sf_full[kMaxStages];  // nvfp4: scale atoms of the stage are in TMEM; w4a8_mx: in shared memory
  uint32_t tmem_base;
  int abort_flag;
  int32_t tile_base[kMaxExperts + 1];
};
template <int KIND>
constexpr int smem_bytes() {
  return 1024 + Cfg<KIND>::kStages * (2 * kSmemW + Cfg<KIND>::kSmemX + 3 * Cfg<KIND>::kSmemSf) + static_cast<int>(sizeof(SmemTail));
}
static_assert(smem_bytes<KIND_NVFP4>() <= 227 * 1024 && smem_bytes<KIND_MX>() <= 227 * 1024, "shared memory");

// MMA columns for a tile of nrows rows
template <int KIND>
__device__ __forceinline__ int token_cols(int nrows) {
  if (KIND == KIND_MX) return (nrows + 15) & ~15;
  return nrows <= 16 ? 16 : (nrows <= 32 ? 32 : 64);
}
// row tiles of a w4a8_mx expert: one up to 80 rows, tiles of 64 above (80 columns are what two accumulator
// buffers and the scale columns leave; 64 keeps a tile's scales aligned in the plan's 128-row atoms)
__device__ __forceinline__ int mx_tiles(int rows) { return rows <= kSmallTailRows ? (rows > 0) : (rows + 63) >> 6; }
// ... of a launch: all rows of the expert, or (TILES_TAIL) its left-over 128-row tile if that is small
__device__ __forceinline__ int mx_tiles_of(const GemmParams& p, int e) {
  const int rows = p.expert_offsets[e + 1] - p.expert_offsets[e];
  if (p.tile_mode != TILES_TAIL) return mx_tiles(rows);
  const int tiles = (rows + 127) >> 7;
  return (tiles & 1) && rows - 128 * (tiles - 1) <= kSmallTailRows ? 1 : 0;
}

// Maximum over the 16 lanes that hold one scale block.
__device__ __forceinline__ float block16_max(float a) {
  a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, 1));
  a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, 2));
  a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, 4));
  a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, 8));
  return a;
}

// NVFP4 re-quantisation of 16 token columns held by one lane (lane = intermediate column); the
// arithmetic per value is that of requant_block16.  codes[0] = tokens 0..7, codes[1] = 8..15 (one
// nibble per token), sfw[k] = the scale bytes of tokens 4k..4k+3.
__device__ __forceinline__ void requant_lane16(const float (&h)[16], float gs, float rgs,
                                               uint32_t (&codes)[2], uint32_t (&sfw)[4]) {
  float lo[16], hi[16], denom[16];
  sfw[0] = sfw[1] = sfw[2] = sfw[3] = 0u;
#pragma unroll
  for (int t = 0; t < 16; ++t) {
    const float amax = block16_max(fabsf(h[t]));
    const float raw =
        fminf(div_rn_normal(__fmul_rn(amax, gs), 6.0f, 0.16666667163372039794921875f), 448.0f);
    const uint8_t sfb = f32_to_e4m3_rn_sat(raw);
    sfw[t >> 2] |= static_cast<uint32_t>(sfb) << (8 * (t & 3));
    const float sf = e4m3_to_f32(sfb);
    denom[t] = fmaxf(div_rn_normal(sf, gs, rgs), 1e-30f);
    const float q = __fmul_rn(h[t], rcp_approx(denom[t]));
    lo[t] = __fmul_rn(q, 1.0f - 4.76837158e-7f);
    hi[t] = __fmul_rn(q, 1.0f + 4.76837158e-7f);
  }
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    float a[8], b[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      a[i] = lo[8 * w + i];
      b[i] = hi[8 * w + i];
    }
    codes[w] = pack_e2m1x8(a);
    if (codes[w] != pack_e2m1x8(b)) {
      // a quotient within 2^-21 of a rounding boundary: take the correctly rounded division
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = __fdiv_rn(h[8 * w + i], denom[8 * w + i]);
      codes[w] = pack_e2m1x8(a);
    }
  }
}

// A work item: expert, weight tile, row tile `mt` of the plan and the tile's rows.  nvfp4 plans for this
// kernel have 64-row tiles; w4a8_mx plans have 128-row tiles, of which an item takes the first 80 rows at
// most, or the upper or lower 64 (`half`).
struct Item {
  int e, nt, mt, half, row0, nrows;
};
template <int KIND>
__device__ __forceinline__ Item decode_item(int w, const GemmParams& p, const int32_t* tb) {
  const TileCoord c = decode_tile(w, p.n_tiles, tb, p.E);
  Item r;
  r.e = c.e;
  r.nt = c.nt;
  if (KIND == KIND_MX) {
    const int t = c.mt - tb[c.e], n = tb[c.e + 1] - tb[c.e];
    r.mt = p.tile_mode == TILES_TAIL ? p.tile_base[c.e + 1] - 1 : p.tile_base[c.e] + (t >> 1);
    r.half = t & 1;
    r.row0 = p.mtile_row0[r.mt] + 64 * r.half;
    r.nrows = p.mtile_rows[r.mt] - 64 * r.half;
    if (n > 1) r.nrows = min(64, r.nrows);
  } else {
    r.mt = c.mt;
    r.half = 0;
    r.row0 = p.mtile_row0[c.mt];
    r.nrows = p.mtile_rows[c.mt];
  }
  return r;
}

// MXFP8 re-quantisation of 16 token columns held by one lane (lane = intermediate column, the warp's 32
// lanes = one scale block); per value the arithmetic of quant_block32_mx.  codes[w] = tokens 4w..4w+3,
// sfw[w] = their scale bytes.
__device__ __forceinline__ void requant_lane32_mx(const float (&h)[16], uint32_t (&codes)[4], uint32_t (&sfw)[4]) {
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    codes[w] = 0u;
    sfw[w] = 0u;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      float q[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float v = h[4 * w + 2 * k + i];
        const uint32_t mag = v == v ? __float_as_uint(v) & 0x7fffffffu : 0u;    // a NaN does not count
        const float amax = __uint_as_float(__reduce_max_sync(0xffffffffu, mag));
        const uint8_t sfb = ue8m0_ceil_byte(__fmul_rn(amax, static_cast<float>(1.0 / 448.0)));
        sfw[w] |= static_cast<uint32_t>(sfb) << (8 * (2 * k + i));
        q[i] = fmaxf(__fmul_rn(v, ue8m0_inv_scale(sfb)), -448.f);
      }
      codes[w] |= static_cast<uint32_t>(__nv_cvt_float2_to_fp8x2(make_float2(q[0], q[1]), __NV_SATFINITE, __NV_E4M3))
                  << (16 * k);
    }
  }
}

template <int KIND, int EPI>
__global__ void __launch_bounds__(Cfg<KIND>::kThreads, 1)
grouped_gemm_small_kernel(const __grid_constant__ CUtensorMap tmW,
                          const __grid_constant__ CUtensorMap tmX16,
                          const __grid_constant__ CUtensorMap tmX32,
                          const __grid_constant__ CUtensorMap tmX64, const GemmParams p) {
  using C = Cfg<KIND>;
  constexpr bool kGated = epi_is_gated(EPI);
  constexpr bool kMx = C::kMx;
  constexpr int kStages = C::kStages, kSmemSf = C::kSmemSf, kSfCols = C::kSfCols;
  constexpr int kMaxTok = C::kMaxTok, kSmemX = C::kSmemX, kAccCols = C::kAccCols, kTmemSf = C::kTmemSf;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sW = smem;                              // [stage][sub-tile][16 KiB]
  uint8_t* sX = sW + kStages * 2 * kSmemW;         // [stage][8 KiB]
  uint8_t* sSf = sX + kStages * kSmemX;            // [stage][sub0, sub1, tokens][2 KiB]
  SmemTail* tail = reinterpret_cast<SmemTail*>(sSf + kStages * 3 * kSmemSf);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&tail->full[s], kMx ? 1 + 4 : 1);     // the producer's arrive (+ the four scale warps)
      mbar_init(&tail->empty[s], 1);
      mbar_init(&tail->sf_full[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tail->tmem_full[b], 1);
      mbar_init(&tail->tmem_empty[b], 8);
    }
    tail->abort_flag = 0;
    fence_mbar_init();
  }
  if (kMx) {
    if (warp == 0) prefix_experts(tail->tile_base, p.E, lane, [&](int e) { return mx_tiles_of(p, e); });
    if (p.tile_mode == TILES_TAIL) {
      __syncthreads();
      if (tail->tile_base[p.E] == 0) return;
    }
  } else {
    for (int i = threadIdx.x; i <= p.E; i += blockDim.x) tail->tile_base[i] = p.tile_base[i];
  }
  if (warp == 1) {
    tmem_alloc(&tail->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  const uint32_t tmem_base = tail->tmem_base;
  volatile int* abort_flag = &tail->abort_flag;
  const int total_work = tail->tile_base[p.E] * p.n_tiles;

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    // One elected thread issues all copies of a stage: token rows, the two weight sub-tiles, the
    // scale atoms of the tokens and of the sub-tiles.
    if (elect_one()) {
      tma_prefetch_desc(&tmW);
      tma_prefetch_desc(&tmX16);
      tma_prefetch_desc(&tmX32);
      tma_prefetch_desc(&tmX64);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int w = blockIdx.x; ok && w < total_work; w += gridDim.x) {
        const Item c = decode_item<KIND>(w, p, tail->tile_base);
        const int row0 = c.row0;
        const int ntok = token_cols<KIND>(c.nrows);
        // w4a8_mx: a box of 64 or 32 rows and one of 16 (either may be missing)
        const int big = ntok >= 64 ? 64 : (kMx ? ntok & 32 : ntok);
        const CUtensorMap* tmx = big == 64 ? &tmX64 : (big == 32 ? &tmX32 : &tmX16);
        // first weight rows (inside the expert) of the sub-tiles, and their scale atom chains
        const int wrow0 = p.sub0_base + c.nt * p.n_step;
        int wrow1 = p.sub1_base + c.nt * p.n_step;
        if (wrow1 >= p.w_rows) wrow1 = wrow0;                        // half-empty last tile
        const size_t chain = static_cast<size_t>(p.atoms_k) * 512;
        const uint8_t* sf_x = p.sfa + static_cast<size_t>(c.mt) * chain;
        const uint8_t* sf_e = p.sfb + static_cast<size_t>(c.e) * p.sfb_rowgroups * chain;
        // w4a8_mx FC1: the scale storage is pair atoms (64 up + 64 gate rows), of which a tile has two
        const int g0 = kMx && kGated ? 2 * c.nt : wrow0 >> 7;
        const int g1 = kMx && kGated ? min(2 * c.nt + 1, p.sfb_rowgroups - 1) : wrow1 >> 7;
        const uint8_t* sf_w0 = sf_e + static_cast<size_t>(g0) * chain;
        const uint8_t* sf_w1 = sf_e + static_cast<size_t>(g1) * chain;
        const int y0 = c.e * p.w_rows + wrow0, y1 = c.e * p.w_rows + wrow1;
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          if (!mbar_wait_bounded(&tail->empty[stage], phase ^ 1, abort_flag, p.status, WAIT_SMEM_EMPTY)) {
            ok = false;
            break;
          }
          const int ksteps = min(4, (p.kdim - kb * C::kPerStage) / C::kPerMma);
          const uint32_t sf_bytes = kMx ? 512u : static_cast<uint32_t>(ksteps) * 512u;
          const size_t sf_off = static_cast<size_t>(kb) * kSmemSf;
          uint64_t* bar = &tail->full[stage];
          uint64_t* sf_bar = kMx ? &tail->sf_full[stage] : bar;
          uint8_t* sf = sSf + stage * 3 * kSmemSf;
          // (the unpacking TMA type counts the packed bytes it reads, half of what it writes)
          const uint32_t row_bytes = static_cast<uint32_t>(ntok) * kRowBytes + (kMx ? kSmemW : 2u * kSmemW);
          if (kMx) mbar_expect_tx(sf_bar, 3u * sf_bytes);
          mbar_expect_tx(bar, kMx ? row_bytes : row_bytes + 3u * sf_bytes);
          tma_load_2d(sW + stage * 2 * kSmemW, &tmW, bar, kb * kRowBytes, y0);
          tma_load_2d(sW + (stage * 2 + 1) * kSmemW, &tmW, bar, kb * kRowBytes, y1);
          if (!kMx || big != 0) tma_load_2d(sX + stage * kSmemX, tmx, bar, kb * kRowBytes, row0);
          if (kMx && ntok != big)
            tma_load_2d(sX + stage * kSmemX + big * kRowBytes, &tmX16, bar, kb * kRowBytes, row0 + big);
          bulk_load(sf, sf_w0 + sf_off, sf_bytes, sf_bar);
          bulk_load(sf + kSmemSf, sf_w1 + sf_off, sf_bytes, sf_bar);
          bulk_load(sf + 2 * kSmemSf, sf_x + sf_off, sf_bytes, sf_bar);
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if (!ok) {
        // give copies that are still in flight time to land before the CTA leaves
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer --------------------------------
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      uint32_t acc_phase[2] = {0, 0};
      int buf = 0;
      bool ok = true;
      for (int w = blockIdx.x; ok && w < total_work; w += gridDim.x) {
        const Item c = decode_item<KIND>(w, p, tail->tile_base);
        const int ntok = token_cols<KIND>(c.nrows);
        const uint32_t idesc = kMx ? make_idesc_block_scaled(128, ntok, /*a e2m1*/ 5, /*b e4m3*/ 0, /*ue8m0*/ 1)
                                   : make_idesc_block_scaled(128, ntok, /*a*/ 1, /*b*/ 1, /*ue4m3*/ 0);
        if (!mbar_wait_bounded(&tail->tmem_empty[buf], acc_phase[buf] ^ 1, abort_flag, p.status,
                               WAIT_TMEM_EMPTY)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t d0 = tmem_base + buf * kAccCols;
        const uint32_t d1 = d0 + kMaxTok;
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          if (!mbar_wait_bounded(&tail->full[stage], phase, abort_flag, p.status, WAIT_SMEM_FULL)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const int ksteps = min(4, (p.kdim - kb * C::kPerStage) / C::kPerMma);
          const uint32_t sf_t = tmem_base + kTmemSf + stage * kSfCols;   // sub0 | sub1 | tokens
          const uint64_t w0 = make_desc_sw128(smem_u32(sW + (stage * 2) * kSmemW));
          const uint64_t w1 = make_desc_sw128(smem_u32(sW + (stage * 2 + 1) * kSmemW));
          const uint64_t xd = make_desc_sw128(smem_u32(sX + stage * kSmemX));
          if (kMx) {
            // the scale warps' arrivals are part of `full`; step j uses byte j of each scale word
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              if (j < ksteps) {
                const uint32_t accum = (kb > 0 || j > 0) ? 1u : 0u;
                const uint32_t ju = static_cast<uint32_t>(j);
                const uint32_t id = idesc | (ju << 29) | (ju << 4), byte = ju << 30;
                mma_mxf8f6f4(d0, w0 + 2 * j, xd + 2 * j, id, sf_t + byte, sf_t + 8 + byte, accum);
                mma_mxf8f6f4(d1, w1 + 2 * j, xd + 2 * j, id, sf_t + 4 + byte, sf_t + 8 + byte, accum);
              }
            }
            tc_commit(&tail->empty[stage]);
            if (++stage == kStages) {
              stage = 0;
              phase ^= 1;
            }
            continue;
          }
          // the scale-copy warp has put this stage's scale atoms into TMEM
          if (!mbar_wait_bounded(&tail->sf_full[stage], phase, abort_flag, p.status, WAIT_SF_FULL)) {
            ok = false;
            break;
          }
          tc_fence_after();
          for (int j = 0; j < ksteps; ++j) {
            // 64 FP4 values = 32 bytes further along the swizzled row -> +2 in 16-byte units
            const uint32_t accum = (kb > 0 || j > 0) ? 1u : 0u;
            mma_nvf4_4x(d0, w0 + 2 * j, xd + 2 * j, idesc, sf_t + 4 * j, sf_t + 32 + 4 * j, accum);
            mma_nvf4_4x(d1, w1 + 2 * j, xd + 2 * j, idesc, sf_t + 16 + 4 * j, sf_t + 32 + 4 * j, accum);
          }
          tc_commit(&tail->empty[stage]);
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (ok) tc_commit(&tail->tmem_full[buf]);
        acc_phase[buf] ^= 1;
        buf ^= 1;
      }
    }
  } else if (kMx && warp >= 10) {
    // ------------------------------ scale atoms -> TMEM (w4a8_mx) ---------------
    // Four warps, one per TMEM sub-partition: through registers, since the tile's scales are not the
    // atoms as they lie.  FC1: word j of lane i of sub-tile 0 is the scales of up row 32 j + i, which the
    // pair atoms hold as words 0, 1 (64 up rows each), and those of the gate rows as words 2, 3.  Tokens:
    // the words of this item's 64 of the row tile's 128 rows.
    const int sub = warp & 3;
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int w = blockIdx.x; ok && w < total_work; w += gridDim.x) {
      const Item c = decode_item<KIND>(w, p, tail->tile_base);
      for (int kb = 0; kb < p.k_blocks; ++kb) {
        if (!mbar_wait_bounded(&tail->sf_full[stage], phase, abort_flag, p.status, WAIT_SMEM_FULL)) {
          ok = false;
          break;
        }
        tc_fence_after();          // behind the MMAs that read these columns (the producer waited for them)
        const uint8_t* sf = sSf + stage * 3 * kSmemSf;
        const uint4 a = reinterpret_cast<const uint4*>(sf)[lane];
        const uint4 b = reinterpret_cast<const uint4*>(sf + kSmemSf)[lane];
        const uint4 t = reinterpret_cast<const uint4*>(sf + 2 * kSmemSf)[lane];
        const uint32_t r0[4] = {a.x, a.y, kGated ? b.x : a.z, kGated ? b.y : a.w};
        const uint32_t r1[4] = {kGated ? a.z : b.x, kGated ? a.w : b.y, b.z, b.w};
        const uint32_t rt[4] = {c.half ? t.z : t.x, c.half ? t.w : t.y, t.z, t.w};   // 80 rows: three words
        const uint32_t sf_t = tmem_base + kTmemSf + stage * kSfCols + (static_cast<uint32_t>(sub * 32) << 16);
        tc_st_32x32b_x4(sf_t, r0);
        tc_st_32x32b_x4(sf_t + 4, r1);
        tc_st_32x32b_x4(sf_t + 8, rt);
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tail->full[stage]);
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (!kMx && warp == 10) {
    // ------------------------------ scale copies -------------------------------
    // One thread moves the scale atoms of every landed stage from shared memory into TMEM and
    // signals their completion on a barrier of its own, so that the MMA issuer never has a
    // tensor-memory copy in front of a dependent MMA in its instruction stream.
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int w = blockIdx.x; ok && w < total_work; w += gridDim.x) {
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          if (!mbar_wait_bounded(&tail->full[stage], phase, abort_flag, p.status, WAIT_SMEM_FULL)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const int ksteps = min(4, (p.kdim - kb * 256) / 64);
          const uint32_t sf_t = tmem_base + kTmemSf + stage * kSfCols;
          const uint32_t sf_s = smem_u32(sSf + stage * 3 * kSmemSf);
          for (int j = 0; j < ksteps; ++j) {
            tc_cp_32x128b_warpx4(sf_t + 4 * j, make_desc_sf(sf_s + 512 * j));
            tc_cp_32x128b_warpx4(sf_t + 16 + 4 * j, make_desc_sf(sf_s + kSmemSf + 512 * j));
            tc_cp_32x128b_warpx4(sf_t + 32 + 4 * j, make_desc_sf(sf_s + 2 * kSmemSf + 512 * j));
          }
          tc_commit(&tail->sf_full[stage]);
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else {
    // ------------------------------ epilogue ----------------------------------
    // Warp w reads TMEM sub-partition (w & 3): weight rows 32*(w&3) .. +31 of a sub-tile.  The two
    // warps of a sub-partition split the token chunks (gated FC1: a lane needs the up and the gate
    // value of its column) or the two sub-tiles (FC2).
    const int sub = warp & 3;
    const int half = (warp - 2) >> 2;
    const int lrow = sub * 32 + lane;          // weight row inside the sub-tile = TMEM lane
    uint32_t acc_phase[2] = {0, 0};
    int buf = 0;
    for (int w = blockIdx.x; w < total_work; w += gridDim.x) {
      const Item c = decode_item<KIND>(w, p, tail->tile_base);
      const int row0 = c.row0;
      const int nrows = c.nrows;
      const int chunks = token_cols<KIND>(nrows) >> 4;
      const float alpha = p.alphas[c.e];
      if (!mbar_wait_bounded(&tail->tmem_full[buf], acc_phase[buf], abort_flag, p.status, WAIT_TMEM_FULL))
        break;
      acc_phase[buf] ^= 1;
      tc_fence_after();
      const uint32_t t_lane = tmem_base + buf * kAccCols + (static_cast<uint32_t>(sub * 32) << 16);

      if (kGated && kMx) {
        // chunk by chunk: the accumulator is double-buffered, so it need not be drained at once
        const int icol = c.nt * 128 + lrow;                    // intermediate column of this lane
        const bool col_ok = icol < p.out_cols;                 // a whole warp alike: out_cols is a multiple of 32
        uint8_t* sft = p.out_sf + static_cast<size_t>(c.mt) * p.out_atoms * 512;
        for (int ch = half; ch < chunks; ch += 2) {
          uint32_t ru[16], rg[16];
          tc_ld_32x32b_x16(t_lane + ch * 16, ru);
          tc_ld_32x32b_x16(t_lane + kMaxTok + ch * 16, rg);
          tc_wait_ld();
          if (p.tap != nullptr && col_ok) {
#pragma unroll
            for (int t = 0; t < 16; ++t) {
              if (ch * 16 + t < nrows) {
                float* trow = p.tap + static_cast<size_t>(row0 + ch * 16 + t) * p.w_rows + icol;
                trow[p.sub0_base] = __fmul_rn(__uint_as_float(ru[t]), alpha);
                trow[p.sub1_base] = __fmul_rn(__uint_as_float(rg[t]), alpha);
              }
            }
          }
          float h[16];
#pragma unroll
          for (int t = 0; t < 16; ++t)
            h[t] = act_gated<EPI>(__fmul_rn(__uint_as_float(rg[t]), alpha), __fmul_rn(__uint_as_float(ru[t]), alpha), p);
          uint32_t codes[4], sfw[4];
          requant_lane32_mx(h, codes, sfw);
          if (col_ok) {
            uint8_t* qcol = p.out_q + static_cast<size_t>(row0 + ch * 16) * p.out_cols + icol;
#pragma unroll
            for (int t = 0; t < 16; ++t)
              if (ch * 16 + t < nrows)
                qcol[static_cast<size_t>(t) * p.out_cols] = static_cast<uint8_t>(codes[t >> 2] >> (8 * (t & 3)));
            // scale bytes: lane j < 16 writes the byte of token j of the chunk
            const uint32_t word = lane < 8 ? (lane < 4 ? sfw[0] : sfw[1]) : (lane < 12 ? sfw[2] : sfw[3]);
            if (lane < 16 && ch * 16 + lane < nrows)
              sft[sf_atom_offset(static_cast<uint32_t>(64 * c.half + ch * 16 + lane), static_cast<uint32_t>(icol >> 5))] =
                  static_cast<uint8_t>(word >> (8 * (lane & 3)));
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tail->tmem_empty[buf]);
      } else if (kGated) {
        // this warp's token chunks: half, half + 2 (at most two)
        uint32_t ru[2][16], rg[2][16];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int ch = half + 2 * k;
          if (ch < chunks) {
            tc_ld_32x32b_x16(t_lane + ch * 16, ru[k]);
            tc_ld_32x32b_x16(t_lane + kMaxTok + ch * 16, rg[k]);
          }
        }
        tc_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tail->tmem_empty[buf]);

        const float gs2 = p.gscale2[p.gscale_len > 1 ? c.e : 0];
        const float rgs2 = __frcp_rn(gs2);
        const int icol = c.nt * 128 + lrow;                    // intermediate column of this lane
        uint8_t* sft = p.out_sf + static_cast<size_t>(c.mt) * p.out_atoms * 512;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int ch = half + 2 * k;
          if (ch < chunks) {
            if (p.tap != nullptr) {
#pragma unroll
              for (int t = 0; t < 16; ++t) {
                if (ch * 16 + t < nrows) {
                  float* trow = p.tap + static_cast<size_t>(row0 + ch * 16 + t) * p.w_rows + icol;
                  trow[p.sub0_base] = __fmul_rn(__uint_as_float(ru[k][t]), alpha);
                  trow[p.sub1_base] = __fmul_rn(__uint_as_float(rg[k][t]), alpha);
                }
              }
            }
            float h[16];
#pragma unroll
            for (int t = 0; t < 16; ++t) {
              const float up = __fmul_rn(__uint_as_float(ru[k][t]), alpha);
              const float gate = __fmul_rn(__uint_as_float(rg[k][t]), alpha);
              h[t] = round_bf16(act_gated<EPI>(gate, up, p));
            }
            uint32_t codes[2], sfw[4];
            requant_lane16(h, gs2, rgs2, codes, sfw);
            // Two lanes (columns 2j, 2j+1) share a byte: the even lane writes tokens 0..7 of the
            // chunk, the odd lane tokens 8..15.
            const bool odd = lane & 1;
            const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? codes[0] : codes[1], 1);
            const uint32_t even_nib = odd ? got : codes[0];      // column 2j   -> low nibble
            const uint32_t odd_nib = odd ? codes[1] : got;       // column 2j+1 -> high nibble
            const int tok0 = ch * 16 + (odd ? 8 : 0);
            uint8_t* qcol = p.out_q + (icol >> 1);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              if (tok0 + i < nrows) {
                const uint32_t byte = ((even_nib >> (4 * i)) & 0xfu) | (((odd_nib >> (4 * i)) & 0xfu) << 4);
                qcol[static_cast<size_t>(row0 + tok0 + i) * (p.out_cols >> 1)] = static_cast<uint8_t>(byte);
              }
            }
            // scale bytes: lane j of a 16-lane block writes the byte of token j of the chunk
            const int j = lane & 15;
            const uint32_t word = (j >> 2) == 0 ? sfw[0] : ((j >> 2) == 1 ? sfw[1] : ((j >> 2) == 2 ? sfw[2] : sfw[3]));
            if (ch * 16 + j < nrows)
              sft[sf_atom_offset(static_cast<uint32_t>(ch * 16 + j), static_cast<uint32_t>(icol >> 4))] =
                  static_cast<uint8_t>(word >> (8 * (j & 3)));
          }
        }
      } else {
        // FC2: this warp drains sub-tile `half`, all token chunks (at most four, w4a8_mx five)
        constexpr int kChunks = kMaxTok / 16;
        uint32_t rr[kChunks][16];
#pragma unroll
        for (int ch = 0; ch < kChunks; ++ch)
          if (ch < chunks) tc_ld_32x32b_x16(t_lane + half * kMaxTok + ch * 16, rr[ch]);
        tc_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tail->tmem_empty[buf]);
        const int f = c.nt * p.n_step + half * 128 + lrow;       // output feature of this lane
        if (f < p.out_cols) {
          float* ocol = p.out_f32 + f;
#pragma unroll
          for (int ch = 0; ch < kChunks; ++ch) {
            if (ch < chunks) {
#pragma unroll
              for (int t = 0; t < 16; ++t)
                if (ch * 16 + t < nrows)
                  ocol[static_cast<size_t>(row0 + ch * 16 + t) * p.out_cols] =
                      __fmul_rn(__uint_as_float(rr[ch][t]), alpha);
            }
          }
        }
      }
      buf ^= 1;
    }
  }

  // ------------------------------ teardown ------------------------------------
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

template <int KIND, int EPI>
static int launch(const CUtensorMap& tmW, const CUtensorMap (&tmX)[3], const GemmParams& p, int grid,
                  cudaStream_t s) {
  auto kern = grouped_gemm_small_kernel<KIND, EPI>;
  constexpr int smem = smem_bytes<KIND>();
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
    return B200MOE_ECUDA;
  kern<<<grid, Cfg<KIND>::kThreads, smem, s>>>(tmW, tmX[0], tmX[1], tmX[2], p);
  return cudaGetLastError() == cudaSuccess ? B200MOE_OK : B200MOE_ECUDA;
}

static int token_maps(CUtensorMap (&tmX)[3], const void* base, uint64_t row_bytes, uint64_t rows) {
  const uint32_t boxes[3] = {16, 32, 64};
  for (int i = 0; i < 3; ++i) {
    const int rc = make_tmap_bytes_2d(&tmX[i], base, row_bytes, rows, boxes[i]);
    if (rc != B200MOE_OK) return rc;
  }
  return B200MOE_OK;
}

}  // namespace small

// The small-batch kernels serve nvfp4 plans cut into 64-row tiles and small w4a8_mx calls (see below).
// B200MOE_SMALL_BATCH=0 keeps the wide-tile kernels on both (comparison runs).
static int small_batch_mode() {
  static int mode = -2;
  if (mode == -2) {
    const char* e = getenv("B200MOE_SMALL_BATCH");
    mode = e == nullptr ? -1 : (atoi(e) != 0 ? 1 : 0);
  }
  return mode;
}

bool nvfp4_small_batch_ok(const b200moe_gemm_args* a, bool fc1) {
  if (small_batch_mode() == 0 || a->layout->tile_rows != 64) return false;
  if (a->hidden_size % 64 != 0 || a->intermediate % 128 != 0 || a->num_experts > kMaxExperts) return false;
  if (fc1 && (a->activation == B200MOE_ACT_RELU2 || a->w13_sf_rows == nullptr)) return false;
  return true;
}

// w4a8_mx with a gated activation: calls that average up to 68 rows per expert (the call's rows, not the plan's
// capacity: all MX plans have the same 128-row tiles), where nearly every expert
// is one tile of at most 80 columns; beyond, tiles of 64 read the weights twice and the 128-row kernel is
// faster.  FC1 + FC2 of the GPT-OSS shape, 128-row kernel against this one: 32 tokens 243 : 203 us, 1024
// (32 rows per expert) 390 : 319, 2048 (64) 412 : 360, 2200 (69) 413 : 364, 2400 (75) 415 : 418, 2600 (81)
// 416 : 471.  On other shapes up to the limit this kernel takes 0.65 to 0.99 of the 128-row kernel's time (layer; 256
// experts of 7168 x 2048, 64 tokens 1264 : 852 us; 8 of 4096 x 14336, 256 tokens 200 : 171), 1.02 on a layer of 4 experts
// of 256 x 128.  Both wait for loads (some 2500 clocks from issue to landing); this kernel has five stages of
// 16 KiB of weights in flight against four, since its token rows take 10 KiB of a stage instead of 16.
// The left-over row tiles of the CTA-pair plans go here up to 80 rows (16384 tokens, FC1 + FC2 of the
// tails 219 -> 179 us) where the call averages 256 rows per expert, as such plans do; below that the two
// launches for left-over tiles would mostly find no work.  B200MOE_SMALL_BATCH=1 / 0 forces these kernels on / off.
static int64_t call_rows(const b200moe_gemm_args* a) { return static_cast<int64_t>(a->num_tokens) * a->num_topk; }
static bool mx_small_shape_ok(const b200moe_gemm_args* a) {
  if (small_batch_mode() == 0 || a->layout->tile_rows != 128 || a->activation == B200MOE_ACT_RELU2) return false;
  return a->hidden_size % 64 == 0 && a->intermediate % 64 == 0 && a->num_experts <= kMaxExperts;
}
bool mx_small_batch_ok(const b200moe_gemm_args* a) {
  const int mode = small_batch_mode();
  if (!mx_small_shape_ok(a)) return false;
  return mode == 1 || call_rows(a) <= 68ll * a->num_experts;
}
bool mx_small_tail_ok(const b200moe_gemm_args* a) {
  return mx_small_shape_ok(a) && call_rows(a) >= 256ll * a->num_experts;
}

int nvfp4_small_gemm1(const b200moe_gemm_args* a, cudaStream_t stream) {
  const b200moe_scratch_layout& L = *a->layout;
  const int K = a->hidden_size, I = a->intermediate, E = a->num_experts;
  if (a->a2_gscale == nullptr) return B200MOE_EINVAL;
  char* base = static_cast<char*>(a->scratch);
  CUtensorMap tmW, tmX[3];
  int rc = make_tmap_bytes_2d(&tmW, a->w13, K / 2, static_cast<uint64_t>(E) * 2 * I, 128);
  if (rc != B200MOE_OK) return rc;
  rc = small::token_maps(tmX, base + L.act_q, K / 2, L.rows);
  if (rc != B200MOE_OK) return rc;
  GemmParams p = {};
  fill_common(p, a, base);
  p.sfa = reinterpret_cast<const uint8_t*>(base + L.act_sf);
  p.sfb = a->w13_sf_rows;
  p.alphas = a->w1_alphas;
  p.gscale2 = a->a2_gscale;
  p.out_q = reinterpret_cast<uint8_t*>(base + L.mid_q);
  p.out_sf = reinterpret_cast<uint8_t*>(base + L.mid_sf);
  p.tap = a->fc1_tap;
  p.kdim = K;
  p.k_blocks = ceil_div_i(K, 256);
  p.atoms_k = K / 64;
  p.w_rows = 2 * I;
  p.sfb_rowgroups = 2 * I / 128;
  p.sub0_base = a->gate_first ? I : 0;   // up rows
  p.sub1_base = a->gate_first ? 0 : I;   // gate rows
  p.n_step = 128;
  p.n_tiles = I / 128;
  p.out_cols = I;
  p.out_atoms = I / 64;
  const int grid = a->num_sms > 0 ? a->num_sms : num_sms_cached();
  if (p.act_kind == 0 && !(p.limit > 0.f)) return small::launch<KIND_NVFP4, EPI_FC1_SILU>(tmW, tmX, p, grid, stream);
  if (p.act_kind == 2) return small::launch<KIND_NVFP4, EPI_FC1_SITU>(tmW, tmX, p, grid, stream);
  if (p.act_kind == 1 && p.limit > 0.f) return small::launch<KIND_NVFP4, EPI_FC1_OAI>(tmW, tmX, p, grid, stream);
  return small::launch<KIND_NVFP4, EPI_FC1_GATED>(tmW, tmX, p, grid, stream);
}

int nvfp4_small_gemm2(const b200moe_gemm_args* a, cudaStream_t stream) {
  const b200moe_scratch_layout& L = *a->layout;
  const int K = a->hidden_size, I = a->intermediate, E = a->num_experts;
  char* base = static_cast<char*>(a->scratch);
  CUtensorMap tmW, tmX[3];
  int rc = make_tmap_bytes_2d(&tmW, a->w2, I / 2, static_cast<uint64_t>(E) * K, 128);
  if (rc != B200MOE_OK) return rc;
  rc = small::token_maps(tmX, base + L.mid_q, I / 2, L.rows);
  if (rc != B200MOE_OK) return rc;
  GemmParams p = {};
  fill_common(p, a, base);
  p.sfa = reinterpret_cast<const uint8_t*>(base + L.mid_sf);
  p.sfb = a->w2_sf;
  p.alphas = a->w2_alphas;
  p.out_f32 = reinterpret_cast<float*>(base + L.routed);
  p.kdim = I;
  p.k_blocks = ceil_div_i(I, 256);
  p.atoms_k = I / 64;
  p.w_rows = K;
  p.sfb_rowgroups = ceil_div_i(K, 128);
  p.sub0_base = 0;
  p.sub1_base = 128;
  p.n_step = 256;
  p.n_tiles = ceil_div_i(K, 256);
  p.out_cols = K;
  const int grid = a->num_sms > 0 ? a->num_sms : num_sms_cached();
  return small::launch<KIND_NVFP4, EPI_FC2>(tmW, tmX, p, grid, stream);
}

int mx_small_gemm1(const b200moe_gemm_args* a, cudaStream_t stream, int tile_mode) {
  const b200moe_scratch_layout& L = *a->layout;
  const int K = a->hidden_size, I = a->intermediate, E = a->num_experts;
  if (a->w13_sf == nullptr) return B200MOE_EINVAL;
  char* base = static_cast<char*>(a->scratch);
  CUtensorMap tmW, tmX[3];
  int rc = make_tmap_fp4_unpack_2d(&tmW, a->w13, K, static_cast<uint64_t>(E) * 2 * I, 128);
  if (rc != B200MOE_OK) return rc;
  rc = small::token_maps(tmX, base + L.act_q, K, L.rows);
  if (rc != B200MOE_OK) return rc;
  GemmParams p = {};
  fill_common(p, a, base);
  p.tile_mode = tile_mode;
  p.sfa = reinterpret_cast<const uint8_t*>(base + L.act_sf);
  p.sfb = a->w13_sf;                     // pair atoms
  p.alphas = a->w1_alphas;
  p.out_q = reinterpret_cast<uint8_t*>(base + L.mid_q);
  p.out_sf = reinterpret_cast<uint8_t*>(base + L.mid_sf);
  p.tap = a->fc1_tap;
  p.kdim = K;
  p.k_blocks = ceil_div_i(K, 128);
  p.atoms_k = ceil_div_i(K, 128);
  p.w_rows = 2 * I;
  p.sfb_rowgroups = I / 64;
  p.sub0_base = a->gate_first ? I : 0;   // up rows
  p.sub1_base = a->gate_first ? 0 : I;   // gate rows
  p.n_step = 128;
  p.n_tiles = ceil_div_i(I, 128);
  p.out_cols = I;
  p.out_atoms = ceil_div_i(I, 128);
  const int grid = a->num_sms > 0 ? a->num_sms : num_sms_cached();
  if (p.act_kind == 0 && !(p.limit > 0.f)) return small::launch<KIND_MX, EPI_FC1_SILU>(tmW, tmX, p, grid, stream);
  if (p.act_kind == 2) return small::launch<KIND_MX, EPI_FC1_SITU>(tmW, tmX, p, grid, stream);
  if (p.act_kind == 1 && p.limit > 0.f) return small::launch<KIND_MX, EPI_FC1_OAI>(tmW, tmX, p, grid, stream);
  return small::launch<KIND_MX, EPI_FC1_GATED>(tmW, tmX, p, grid, stream);
}

int mx_small_gemm2(const b200moe_gemm_args* a, cudaStream_t stream, int tile_mode) {
  const b200moe_scratch_layout& L = *a->layout;
  const int K = a->hidden_size, I = a->intermediate, E = a->num_experts;
  if (a->w2_sf == nullptr) return B200MOE_EINVAL;
  char* base = static_cast<char*>(a->scratch);
  CUtensorMap tmW, tmX[3];
  int rc = make_tmap_fp4_unpack_2d(&tmW, a->w2, I, static_cast<uint64_t>(E) * K, 128);
  if (rc != B200MOE_OK) return rc;
  rc = small::token_maps(tmX, base + L.mid_q, I, L.rows);
  if (rc != B200MOE_OK) return rc;
  GemmParams p = {};
  fill_common(p, a, base);
  p.tile_mode = tile_mode;
  p.sfa = reinterpret_cast<const uint8_t*>(base + L.mid_sf);
  p.sfb = a->w2_sf;
  p.alphas = a->w2_alphas;
  p.out_f32 = reinterpret_cast<float*>(base + L.routed);
  p.kdim = I;
  p.k_blocks = ceil_div_i(I, 128);
  p.atoms_k = ceil_div_i(I, 128);
  p.w_rows = K;
  p.sfb_rowgroups = ceil_div_i(K, 128);
  p.sub0_base = 0;
  p.sub1_base = 128;
  p.n_step = 256;
  p.n_tiles = ceil_div_i(K, 256);
  p.out_cols = K;
  const int grid = a->num_sms > 0 ? a->num_sms : num_sms_cached();
  return small::launch<KIND_MX, EPI_FC2>(tmW, tmX, p, grid, stream);
}

}  // namespace b200moe
