// Routing of a decode batch (up to 256 tokens): top-k, per-expert counts, offsets and the expert-contiguous permutation
// without a trip through global memory, by one thread-block cluster or, for a launch of its own with few tokens, one CTA.
//
// A token selects an expert at most once, so the assignments of an expert, in the order of the permutation (ascending
// token), are the set bits of a token mask.  Every warp takes a token, keeps its choices in registers and sets its bits
// in the masks of the cluster's first CTA (atomics on distributed shared memory); that CTA turns mask populations into
// offsets; a choice's place is its expert's offset plus the bits below its own.  Latency bound: a few barriers and one
// block scan.  Barriers across a cluster and atomics on another CTA's memory cost several times the local ones, so up to
// RS_ONE_TOKENS tokens, one for each of 32 warps, stay in one CTA (a whole block of one token 26.9 -> 25.4 us; at 64 tokens,
// two for a warp, the cluster is 0.9 us faster).
#pragma once

#include <cooperative_groups.h>

#include "skinny.cuh"
#include "topk.cuh"

namespace bm {

constexpr int RS_THREADS = 256, RS_CLUSTER = 8, RS_MAX_E = 512, RS_MAX_TOKENS = 256, RS_MASK_WORDS = RS_MAX_TOKENS / 32;
constexpr int RS_ONE_THREADS = 1024, RS_ONE_TOKENS = 32;

// Shared memory of the first CTA: masks [E][words], offsets [E + 1], scan scratch.
struct RouteSmallSmem {
  uint32_t mask[RS_MAX_E * RS_MASK_WORDS];
  int offset[RS_MAX_E + 1];
  int warp_tot[RS_ONE_THREADS / 32];
};

// CL CTAs of THREADS threads
template <int REG, int CL, int THREADS>
__device__ __forceinline__ void route_small_impl(const RouteSmallArgs& a, RouteSmallSmem* sm) {
  namespace cg = cooperative_groups;
  constexpr int WARPS = THREADS / 32, ROUNDS = CL == 1 ? 2 : RS_MAX_TOKENS / (CL * WARPS);    // tokens per warp at most
  static_assert(CL > 1 || ROUNDS * WARPS >= RS_ONE_TOKENS, "a round for every token");
  auto sync = [] { if constexpr (CL == 1) __syncthreads(); else cg::this_cluster().sync(); };
  const int rank = CL == 1 ? 0 : static_cast<int>(cg::this_cluster().block_rank());
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int words = (a.T + 31) >> 5;
  RouteSmallSmem* s0 = sm;
  if constexpr (CL > 1) s0 = cg::this_cluster().map_shared_rank(sm, 0);
  if (rank == 0)
    for (int i = threadIdx.x; i < a.E * words; i += THREADS) sm->mask[i] = 0u;
  cg::cluster_group::arrival_token cleared;
  if constexpr (CL > 1) cleared = cg::this_cluster().barrier_arrive();
  int idx[ROUNDS];
  float w[ROUNDS];
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) {
    const int t = (r * WARPS + warp) * CL + rank;     // neighbouring tokens go to different SMs
    idx[r] = -1;
    w[r] = 0.f;
    if (t < a.T) {
      warp_topk<REG>(a.logits, a.logits_dtype, t, a.E, a.k, a.renorm, a.weight_round, &idx[r], &w[r]);
      if (lane >= a.k || static_cast<unsigned>(idx[r]) >= static_cast<unsigned>(a.E)) idx[r] = -1;
    }
  }
  if constexpr (CL > 1) cg::this_cluster().barrier_wait(std::move(cleared));
  else __syncthreads();
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) {
    const int t = (r * WARPS + warp) * CL + rank;
    if (idx[r] >= 0) atomicOr(&s0->mask[idx[r] * words + (t >> 5)], 1u << (t & 31));
  }
  sync();
  if (rank == 0) {
    constexpr int PER = RS_MAX_E > THREADS ? RS_MAX_E / THREADS : 1;     // consecutive experts of a thread
    int cnt[PER], sum = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = threadIdx.x * PER + i;
      cnt[i] = 0;
      if (e < a.E)
        for (int q = 0; q < words; ++q) cnt[i] += __popc(sm->mask[e * words + q]);
      sum += cnt[i];
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += n;
    }
    if (lane == 31) sm->warp_tot[warp] = incl;
    __syncthreads();
    int run = incl - sum;
#pragma unroll
    for (int q = 0; q < RS_MAX_E / (32 * PER); ++q) run += q < warp ? sm->warp_tot[q] : 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = threadIdx.x * PER + i;
      if (e <= a.E) {
        sm->offset[e] = run;
        a.expert_offsets[e] = run;
      }
      run += cnt[i];
    }
    if (THREADS * PER == RS_MAX_E && a.E == RS_MAX_E && threadIdx.x == THREADS - 1) {
      sm->offset[RS_MAX_E] = run;
      a.expert_offsets[RS_MAX_E] = run;
    }
  }
  sync();
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) {
    const int t = (r * WARPS + warp) * CL + rank;
    if (idx[r] >= 0) {
      const uint32_t* m = &s0->mask[idx[r] * words];
      int pos = s0->offset[idx[r]] + __popc(m[t >> 5] & ((1u << (t & 31)) - 1u));
      for (int q = 0; q < (t >> 5); ++q) pos += __popc(m[q]);
      a.token_indices[pos] = t;
      a.route_flat[pos] = w[r];
    }
  }
  if constexpr (CL > 1) sync();      // the first CTA's shared memory is read until here
}

template <int CL = RS_CLUSTER, int THREADS = RS_THREADS>
__device__ __forceinline__ void route_small(const RouteSmallArgs& a, RouteSmallSmem* sm) {
  if (a.E <= 64) route_small_impl<2, CL, THREADS>(a, sm);
  else if (a.E <= 128) route_small_impl<4, CL, THREADS>(a, sm);
  else if (a.E <= 256) route_small_impl<8, CL, THREADS>(a, sm);
  else route_small_impl<16, CL, THREADS>(a, sm);
}

}  // namespace bm
