// Router selection shared by the standalone routing kernels and the one-launch decode step: one warp turns a
// token's E router scores into top-k expert ids and gate weights (softmax or sigmoid scoring, selection bias,
// group-limited routing, ties to the lowest id).  Contract of the reference router
// (native/shared/cuda/expert_router.cu:12-55,108-158): bias is used for selection only, weights come from the
// unbiased scores, normalised over the top-k with +1e-20, times the routed scale.  Scoring 2 is softmax over logits the bias is
// part of: it then shapes the weights too.
#pragma once

#include "common.cuh"

namespace cafd {

// Order-preserving key of a selection score, 0 for NaN (never selected; no number has it) and the same for both zeros.  One warp
// reduction of keys takes the place of five rounds of shuffled (value, id) pairs per pick (the router's launch behind the o projection,
// top-8 of 128 at one row: 9.8 -> 8.0 us together with the early request of its weights).
__device__ __forceinline__ uint32_t route_key(float v) {
  const uint32_t b = __float_as_uint(v + 0.0f);
  return v != v ? 0u : (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float route_value(uint32_t k) {
  return k == 0u ? -INFINITY : __uint_as_float((k & 0x80000000u) ? (k ^ 0x80000000u) : ~k);
}

// ---- router -------------------------------------------------------------------------------------
// One warp routes one token: `row` points at its E router logits in global memory, or (kShared) in the block's own shared memory.
template <int kPerLane, bool kShared = false>
__device__ __forceinline__ void route_row(const float* row, const float* __restrict__ bias, int* __restrict__ out_idx,
                                          float* __restrict__ out_w, int t, int E, int top_k, int scoring, int num_groups,
                                          int topk_groups, int normalize, float routed_scale, int group_max = 0) {
  const int lane = threadIdx.x & 31;
  float score[kPerLane], sel[kPerLane];
  float mx = -INFINITY;
#pragma unroll
  for (int j = 0; j < kPerLane; ++j) {
    const int e = j * 32 + lane;
    score[j] = e >= E ? -INFINITY : kShared ? row[e] : __ldcg(row + e);     // global: written by other blocks (or an earlier kernel), skip L1
    if (scoring == 2 && bias && e < E) score[j] += bias[e];
    mx = fmaxf(mx, score[j]);
  }
  if (scoring == 1) {
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
      const int e = j * 32 + lane;
      score[j] = e < E ? 1.0f / (1.0f + expf(-score[j])) : -INFINITY;
    }
  } else {
    mx = warp_max(mx);
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
      const int e = j * 32 + lane;
      score[j] = e < E ? expf(score[j] - mx) : 0.f;
      sum += score[j];
    }
    sum = warp_sum(sum);
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
      const int e = j * 32 + lane;
      score[j] = e < E ? score[j] / sum : -INFINITY;
    }
  }
#pragma unroll
  for (int j = 0; j < kPerLane; ++j) {
    const int e = j * 32 + lane;
    sel[j] = e < E ? score[j] + (bias && scoring != 2 ? bias[e] : 0.f) : -INFINITY;
  }
  if (num_groups > 1) {
    const int per_group = E / num_groups;
    // group of each of this lane's experts, computed once (the loops below would otherwise divide per element)
    int gid[kPerLane];
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
      const int e = j * 32 + lane;
      gid[j] = e < E ? e / per_group : -1;
    }
    unsigned keep = 0;   // bit g set = group g kept
    float gscore_mine = -INFINITY;   // lane g holds the score of group g
    for (int g = 0; g < num_groups; ++g) {
      // the group's two best selection scores (group_max: a group counts by its best alone): the best key of the warp, then the best of
      // what is left once the first lane that holds it has given up one
      uint32_t k1 = 0, k2 = 0;
#pragma unroll
      for (int j = 0; j < kPerLane; ++j) {
        if (gid[j] == g) {
          const uint32_t k = route_key(sel[j]);
          if (k > k1) { k2 = k1; k1 = k; }
          else if (k > k2) k2 = k;
        }
      }
      const uint32_t top1 = __reduce_max_sync(0xffffffffu, k1);
      const unsigned holders = __ballot_sync(0xffffffffu, k1 == top1);
      const uint32_t top2 = __reduce_max_sync(0xffffffffu, lane == __ffs(holders) - 1 ? k2 : k1);
      if (lane == g) gscore_mine = group_max ? route_value(top1) : route_value(top1) + route_value(top2);
    }
    for (int it = 0; it < topk_groups; ++it) {
      float v = (lane < num_groups && !((keep >> lane) & 1u)) ? gscore_mine : -INFINITY;
      int gi = lane;
      // groups with -inf scores can still be picked when fewer finite ones exist: mark via index
      if (!(lane < num_groups) || ((keep >> lane) & 1u)) gi = 0x7fffffff;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, gi, o);
        if (ov > v || (ov == v && oi < gi)) { v = ov; gi = oi; }
      }
      if (gi != 0x7fffffff) keep |= 1u << gi;
    }
#pragma unroll
    for (int j = 0; j < kPerLane; ++j)
      if (gid[j] >= 0 && !((keep >> gid[j]) & 1u)) sel[j] = -INFINITY;
  }
  float wsum = 0.f;
  float my_w = 0.f;
  int my_i = 0;
  unsigned taken = 0;   // bit j: this lane's element j was already selected
  for (int it = 0; it < top_k; ++it) {
    uint32_t bk = 0;
    int bi = 0x7fffffff;
    float bs = 0.f;
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
      const int e = j * 32 + lane;
      const uint32_t k = e < E && !((taken >> j) & 1u) ? route_key(sel[j]) : 0u;
      if (k > bk) { bk = k; bi = e; bs = score[j]; }             // ascending ids: an equal key keeps the lower one
    }
    const uint32_t best = __reduce_max_sync(0xffffffffu, bk);
    bi = static_cast<int>(__reduce_min_sync(0xffffffffu, best > 0 && bk == best ? static_cast<unsigned>(bi) : 0x7fffffffu));
    bs = __shfl_sync(0xffffffffu, bs, bi & 31);
    if (bi == 0x7fffffff) { bi = 0; bs = 0.f; }   // every candidate was NaN
#pragma unroll
    for (int j = 0; j < kPerLane; ++j)
      if (j * 32 + lane == bi) taken |= 1u << j;
    wsum += bs;
    if (lane == it) { my_w = bs; my_i = bi; }
  }
  if (lane < top_k) {
    float w = my_w;
    if (normalize) w = w / (wsum + 1e-20f);
    out_idx[static_cast<size_t>(t) * top_k + lane] = my_i;
    out_w[static_cast<size_t>(t) * top_k + lane] = w * routed_scale;
  }
}

}  // namespace cafd
