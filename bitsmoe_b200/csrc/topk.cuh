// Softmax top-k of one token by one warp, the experts' probabilities in registers.
#pragma once

#include "common.cuh"

namespace bm {

__device__ __forceinline__ float round_route_weight(float w, int weight_round) {
  if (weight_round == BM_ROUND_F16) return __half2float(__float2half_rn(w));
  if (weight_round == BM_ROUND_BF16) return __bfloat162float(__float2bfloat16_rn(w));
  return w;
}

// Lane l holds experts l, l + 32, ... (REG of them: E <= 32 * REG).  Lane j < k returns the j-th choice and its final
// weight; ties go to the lower expert id.
template <int REG>
__device__ __forceinline__ void warp_topk(const void* __restrict__ logits, int dtype, int64_t t, int E, int k, int renorm,
                                          int weight_round, int* idx, float* weight) {
  const int lane = threadIdx.x & 31;
  float v[REG];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < REG; ++i) {
    const int e = lane + 32 * i;
    v[i] = e < E ? load_act(logits, dtype, t * E + e) : -INFINITY;
    mx = fmaxf(mx, v[i]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < REG; ++i) {
    v[i] = lane + 32 * i < E ? expf(v[i] - mx) : -1.f;   // padding can never win
    sum += fmaxf(v[i], 0.f);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  const float inv = 1.f / sum;
  // A lane keeps its best probability; only the lane whose probability was taken looks through its own again.
  float best;
  int bi;
  auto look = [&]() {
    best = v[0];
    bi = 0;
#pragma unroll
    for (int i = 1; i < REG; ++i) {
      bi = v[i] > best ? i : bi;                 // ascending e: the first hit wins ties
      best = fmaxf(v[i], best);
    }
  };
  look();
  float my_w = 0.f, wsum = 0.f;
  int my_i = 0;
  for (int j = 0; j < k; ++j) {
    // probabilities are non-negative, so their bit patterns order like unsigned integers: two warp reductions
    // (largest value, then the lowest expert id holding it) replace a ten-shuffle butterfly
    const unsigned bits = __float_as_uint(fmaxf(best, 0.f));
    const unsigned best_bits = __reduce_max_sync(0xffffffffu, bits);
    const int e = static_cast<int>(__reduce_min_sync(0xffffffffu, bits == best_bits && best >= 0.f ? static_cast<unsigned>(lane + 32 * bi) : 0x7fffffffu));
    const float w = __uint_as_float(best_bits) * inv;
    if (lane == j) { my_w = w; my_i = e; }
    wsum += w;
    if ((e & 31) == lane) {
#pragma unroll
      for (int i = 0; i < REG; ++i) v[i] = e == lane + 32 * i ? -2.f : v[i];
      look();
    }
  }
  *idx = my_i;
  *weight = round_route_weight(renorm ? my_w / wsum : my_w, weight_round);
}

}  // namespace bm
