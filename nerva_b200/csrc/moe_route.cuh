// Softmax top-k routing of one token by one warp (moe.cu: the decode step, moe_block.cu: a block's rows).
#pragma once

#include "common.cuh"

namespace nb {

constexpr uint32_t kMoeMaxExperts = 256, kMoeMaxTopK = 16;

// weights = softmax(logits) with the reference's guards (divide only by a finite positive total); the k winners by
// (weight descending, index ascending) to ids_out / weights_out, written by lanes 0 .. top_k - 1.  All lanes call.
// Lane l holds experts l, l + 32, ..., in registers; a weight's bits order like the weight (it is not negative), so a
// rank is one maximum over the warp, one minimum over the indices that reach it and a shuffle.  (Comparing pairs of
// weight and index by ten shuffles a rank took 5.6 us for 8 of 64 experts, as long as the experts' weights.)
__device__ __forceinline__ void moe_route_warp(const float *logits, uint32_t num_experts, uint32_t top_k,
                                               uint32_t norm_topk_prob, uint32_t *ids_out, float *weights_out) {
  constexpr uint32_t kNone = 0xffffffffu, kPerLane = kMoeMaxExperts / 32u;
  const uint32_t lane = threadIdx.x & 31u;
  float w[kPerLane], m = -INFINITY, sum = 0.0f;
#pragma unroll
  for (uint32_t k = 0; k < kPerLane; ++k) {
    const uint32_t e = lane + 32u * k;
    w[k] = e < num_experts ? logits[e] : -INFINITY;
    m = fmaxf(m, w[k]);
  }
  m = warp_max(m);
#pragma unroll
  for (uint32_t k = 0; k < kPerLane; ++k) {
    w[k] = lane + 32u * k < num_experts ? expf(w[k] - m) : 0.0f;
    sum += w[k];
  }
  sum = warp_sum(sum);
  if (sum > 0.0f && isfinite(sum)) {
#pragma unroll
    for (uint32_t k = 0; k < kPerLane; ++k) w[k] /= sum;
  }
  uint32_t key[kPerLane];  // 0: taken or no expert
#pragma unroll
  for (uint32_t k = 0; k < kPerLane; ++k)
    key[k] = lane + 32u * k < num_experts ? (w[k] > 0.0f ? __float_as_uint(w[k]) : 0u) + 1u : 0u;  // not a number: as zero
  uint32_t my_id = 0;
  float chosen_sum = 0.0f, mine = 0.0f;
  for (uint32_t rank = 0; rank < top_k; ++rank) {
    uint32_t best = 0, at = 0;
    float best_w = 0.0f;
#pragma unroll
    for (uint32_t k = 0; k < kPerLane; ++k)
      if (key[k] > best) best = key[k], at = k, best_w = w[k];
    const uint32_t top = __reduce_max_sync(0xffffffffu, best);
    const uint32_t id = __reduce_min_sync(0xffffffffu, best == top ? lane + 32u * at : kNone);
    const float chosen = __shfl_sync(0xffffffffu, best_w, id & 31u);
#pragma unroll
    for (uint32_t k = 0; k < kPerLane; ++k)
      if (lane + 32u * k == id) key[k] = 0u;
    chosen_sum += chosen;
    if (lane == rank) mine = chosen, my_id = id;
  }
  if (norm_topk_prob != 0 && chosen_sum > 0.0f) mine /= chosen_sum;
  if (lane < top_k) {
    ids_out[lane] = my_id;
    weights_out[lane] = mine;
  }
}

}  // namespace nb
