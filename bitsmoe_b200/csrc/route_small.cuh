// Routing of a decode batch (up to 256 tokens) by one thread-block cluster: top-k, per-expert counts, offsets and the
// expert-contiguous permutation without a trip through global memory.
//
// A token selects an expert at most once, so the assignments of an expert, in the order of the permutation (ascending
// token), are the set bits of a token mask.  Every warp takes a token, keeps its choices in registers and sets its bits
// in the masks of the cluster's first CTA (atomics on distributed shared memory); that CTA turns mask populations into
// offsets; a choice's place is its expert's offset plus the bits below its own.  Latency bound: a few cluster barriers and
// one block scan.
#pragma once

#include <cooperative_groups.h>

#include "skinny.cuh"
#include "topk.cuh"

namespace bm {

constexpr int RS_THREADS = 256, RS_CLUSTER = 8, RS_MAX_E = 512, RS_MAX_TOKENS = 256, RS_MASK_WORDS = RS_MAX_TOKENS / 32;
constexpr int RS_ROUNDS = RS_MAX_TOKENS / (RS_CLUSTER * RS_THREADS / 32);    // tokens per warp at most

// Shared memory of the first CTA: masks [E][words], offsets [E + 1], scan scratch.
struct RouteSmallSmem {
  uint32_t mask[RS_MAX_E * RS_MASK_WORDS];
  int offset[RS_MAX_E + 1];
  int warp_tot[RS_THREADS / 32];
};

template <int REG>
__device__ __forceinline__ void route_small_impl(const RouteSmallArgs& a, RouteSmallSmem* sm) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = static_cast<int>(cluster.block_rank());
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int words = (a.T + 31) >> 5;
  RouteSmallSmem* s0 = cluster.map_shared_rank(sm, 0);
  if (rank == 0)
    for (int i = threadIdx.x; i < a.E * words; i += RS_THREADS) sm->mask[i] = 0u;
  auto cleared = cluster.barrier_arrive();
  int idx[RS_ROUNDS];
  float w[RS_ROUNDS];
#pragma unroll
  for (int r = 0; r < RS_ROUNDS; ++r) {
    const int t = (r * (RS_THREADS / 32) + warp) * RS_CLUSTER + rank;     // neighbouring tokens go to different SMs
    idx[r] = -1;
    w[r] = 0.f;
    if (t < a.T) {
      warp_topk<REG>(a.logits, a.logits_dtype, t, a.E, a.k, a.renorm, a.weight_round, &idx[r], &w[r]);
      if (lane >= a.k) idx[r] = -1;
      else {
        if (a.topk_idx) a.topk_idx[t * a.k + lane] = idx[r];
        if (a.topk_w) a.topk_w[t * a.k + lane] = w[r];
        if (static_cast<unsigned>(idx[r]) >= static_cast<unsigned>(a.E)) idx[r] = -1;
      }
    }
  }
  cluster.barrier_wait(std::move(cleared));
#pragma unroll
  for (int r = 0; r < RS_ROUNDS; ++r) {
    const int t = (r * (RS_THREADS / 32) + warp) * RS_CLUSTER + rank;
    if (idx[r] >= 0) atomicOr(&s0->mask[idx[r] * words + (t >> 5)], 1u << (t & 31));
  }
  cluster.sync();
  if (rank == 0) {
    constexpr int PER = RS_MAX_E / RS_THREADS;     // consecutive experts of a thread
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
    for (int q = 0; q < warp; ++q) run += sm->warp_tot[q];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = threadIdx.x * PER + i;
      if (e <= a.E) {
        sm->offset[e] = run;
        a.expert_offsets[e] = run;
      }
      run += cnt[i];
    }
    if (a.E == RS_MAX_E && threadIdx.x == RS_THREADS - 1) {
      sm->offset[RS_MAX_E] = run;
      a.expert_offsets[RS_MAX_E] = run;
    }
  }
  cluster.sync();
#pragma unroll
  for (int r = 0; r < RS_ROUNDS; ++r) {
    const int t = (r * (RS_THREADS / 32) + warp) * RS_CLUSTER + rank;
    if (idx[r] >= 0) {
      const uint32_t* m = &s0->mask[idx[r] * words];
      int pos = s0->offset[idx[r]] + __popc(m[t >> 5] & ((1u << (t & 31)) - 1u));
      for (int q = 0; q < (t >> 5); ++q) pos += __popc(m[q]);
      a.token_indices[pos] = t;
      a.route_flat[pos] = w[r];
    }
  }
  cluster.sync();      // the first CTA's shared memory is read until here
}

__device__ __forceinline__ void route_small(const RouteSmallArgs& a, RouteSmallSmem* sm) {
  if (a.E <= 64) route_small_impl<2>(a, sm);
  else if (a.E <= 128) route_small_impl<4>(a, sm);
  else if (a.E <= 256) route_small_impl<8>(a, sm);
  else route_small_impl<16>(a, sm);
}

}  // namespace bm
