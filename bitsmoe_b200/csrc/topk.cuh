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
  // A lane keeps the best two of its probabilities that come after the last one taken from it (largest first, equal ones by
  // ascending expert id) and looks through its own again only when both are gone: with the choices spread over 32 lanes
  // that is about k^2 / 64 times a token, where keeping one would look k times.
  float best, second, last = INFINITY;
  int bi, si, last_i = -1;
  auto look = [&]() {
    best = second = -1.f;
    bi = si = 0;
#pragma unroll
    for (int i = 0; i < REG; ++i) {
      const bool open = v[i] < last || (v[i] == last && i > last_i);
      const float c = open ? v[i] : -1.f;
      const bool first = c > best, next = c > second;      // ascending e: the earlier one wins ties
      si = first ? bi : next ? i : si;
      second = first ? best : next ? c : second;
      bi = first ? i : bi;
      best = first ? c : best;
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
    if (e == lane + 32 * bi && best >= 0.f) {
      last = best;
      last_i = bi;
      best = second;
      bi = si;
      second = -1.f;
      if (REG > 1 && best < 0.f) look();
    }
  }
  *idx = my_i;
  *weight = round_route_weight(renorm ? my_w / wsum : my_w, weight_round);
}

}  // namespace bm
