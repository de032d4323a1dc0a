// The per-token router shared by the stand-alone top-k kernel and the fused gate kernels.
#pragma once

#include "common.cuh"

namespace b200moe {

// ------------------------------------------------------------------------------------------
// route_topk: one warp per token.  Lane l holds experts l, l+32, ... (E <= 1024: PER <= 32 values a
// lane).  Selection repeats "max, ties to the LARGEST expert index" k times, which is the tie rule
// of the reference router (b12x/moe/_shared/routing.py:38-46).
//
// What bounds it is the serial chain of k selections in one warp.  Every value becomes an unsigned
// key that orders as the float does, so a selection is two warp reductions (redux.sync: the largest
// key, then the largest index that holds it) instead of ten shuffles, a lane looks through its own
// values again only when it held the winner, and the tables are sized by E (PER), not by the
// maximum of 1024 experts.  One token of 256 experts, top-8, sigmoid: 11.2 -> 3.9 us; 16384 tokens of 128
// experts, top-4: 49.7 -> 10.7 us (8.4 MB of logits: 0.8 TB/s).
// ------------------------------------------------------------------------------------------
constexpr uint32_t kRouteKeyNone = 0u;             // NaN or no expert: never selected
constexpr uint32_t kRouteKeyNegInf = 0x007fffffu;  // -infinity, and every expert already taken

// unsigned order = float order, -0 with +0; NaN below everything
__device__ __forceinline__ uint32_t route_key(float v) {
  if (v != v) return kRouteKeyNone;
  const uint32_t u = __float_as_uint(__fadd_rn(v, 0.0f));
  return u ^ ((u >> 31) ? 0xffffffffu : 0x80000000u);
}

// One warp routes token `t`.  PAST_L1: the logits were written in this launch (read them with
// ld.global.cg).
template <int MODE, int PER, bool PAST_L1 = false>
__device__ __forceinline__ void route_topk_token(const b200moe_route_args& a, int t, int lane) {
  const int E = a.num_experts;
  const float NEG_INF = __int_as_float(0xff800000);

  auto logit = [&](int e) -> float {
    const int64_t o = static_cast<int64_t>(t) * a.logits_row_stride + e;
    if (a.logits_dtype == B200MOE_DT_BF16) {
      const unsigned short* p16 = reinterpret_cast<const unsigned short*>(a.logits) + o;
      return __bfloat162float(__ushort_as_bfloat16(PAST_L1 ? __ldcg(p16) : *p16));
    }
    const float* p32 = reinterpret_cast<const float*>(a.logits) + o;
    return PAST_L1 ? __ldcg(p32) : *p32;
  };
  // the value the weights are made from: the logit, or its sigmoid
  auto source = [&](float v) -> float { return MODE == B200MOE_ROUTE_SIGMOID ? 1.0f / (1.0f + expf(-v)) : v; };

  float v[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) v[i] = i * 32 + lane < E ? logit(i * 32 + lane) : 0.f;
  uint32_t key[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = i * 32 + lane;
    float sel = source(v[i]);
    if (MODE == B200MOE_ROUTE_SIGMOID && a.bias != nullptr && e < E) sel = sel + a.bias[e];
    key[i] = e < E ? route_key(sel) : kRouteKeyNone;
  }

  // this lane's best: the largest key, ties to the larger index
  uint32_t best = kRouteKeyNone;
  int best_i = 0;
  auto rescan = [&]() {
    best = kRouteKeyNone;
    best_i = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (key[i] >= best) {
        best = key[i];
        best_i = i;
      }
  };
  rescan();

  uint32_t taken = 0;            // bit i: this lane's value i has been selected
  int my_id = 0;                 // lane `slot` keeps the slot's expert (k <= 32) ...
  int my_kind = 0;               // ... 0: an expert, 1: nothing was left but NaNs, 2: taken before (-infinity)
  for (int slot = 0; slot < a.num_topk; ++slot) {
    const uint32_t top = __reduce_max_sync(0xffffffffu, best);
    int e = -1, kind = 1;
    if (top != kRouteKeyNone) {
      e = static_cast<int>(__reduce_max_sync(0xffffffffu, best == top ? static_cast<uint32_t>(best_i * 32 + lane) : 0u));
      kind = 0;
      const bool mine = (e & 31) == lane;
      // only experts at -infinity can come up twice (fewer finite values than slots)
      if (top == kRouteKeyNegInf && __ballot_sync(0xffffffffu, mine && ((taken >> (e >> 5)) & 1u)) != 0u) kind = 2;
      if (mine) {
        taken |= 1u << (e >> 5);
#pragma unroll
        for (int i = 0; i < PER; ++i)
          if (i == (e >> 5)) key[i] = kRouteKeyNegInf;
        rescan();
      }
      __syncwarp();
    }
    if (slot == lane) {
      my_id = e < 0 ? 0 : e;
      my_kind = kind;
    }
  }

  const bool active = lane < a.num_topk;
  float val = 0.f;
  if (active) val = my_kind == 0 ? source(logit(my_id)) : (my_kind == 1 ? 0.f : NEG_INF);
  const float out_logit = (MODE != B200MOE_ROUTE_SIGMOID && my_kind == 1) ? NEG_INF : val;
  float w = val;
  if (MODE == B200MOE_ROUTE_SOFTMAX_TOPK) {
    // softmax over the selected logits, max-shifted (slot 0 holds the maximum)
    const float mx = __shfl_sync(0xffffffffu, val, 0);
    float ex = active ? expf(val - mx) : 0.f;
    float sum = ex;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    w = ex / sum;
  } else if (MODE == B200MOE_ROUTE_SIGMOID) {
    float sum = active ? val : 0.f;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    if (a.renormalize) w = val / fmaxf(sum, 1e-20f);
    w = w * a.route_scale;
  }
  if (active) {
    const int64_t o = static_cast<int64_t>(t) * a.num_topk + lane;
    a.topk_ids[o] = my_id;
    a.topk_weights[o] = w;
    if (a.topk_logits) a.topk_logits[o] = out_logit;
  }
}

}  // namespace b200moe
