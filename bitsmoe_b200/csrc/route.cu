// Token routing: softmax -> top-k -> (renorm, rounding), then the expert-contiguous
// permutation with per-expert offsets and the padded tile table, all on the device
// with no host round trip.
//
// Semantics follow bitsmoe/models/qwen3moe/bitsmoe_block.py:47-51 (router tail) and
// bitsmoe/models/base_block.py:258-289 (_build_packed_routing).  Where the reference
// leaves the order open (torch.topk ties, an unstable argsort) this file fixes it:
// ties go to the lower expert id, and inside an expert assignments are ordered by
// ascending flat (token, slot) index.
//
// What bounds it is latency: dependent launches, two up to the sizes that one cluster places, four above.  Top-k and placement of 6216
// assignments of 128 experts 20 us (four launches one behind the other) -> 10.  16384 tokens of 512 experts, top 10: top-k 52 -> 24.5 us
// (topk.cuh), prefixes of the block histograms 16.5 -> 4 us (one block walked them; now a thread of a grid per expert, and the totals
// are scanned where they are used), counting 5, scatter 8.
#include <cooperative_groups.h>

#include "topk.cuh"

namespace bm {

constexpr int ROUTE_MAX_E = 1024;
constexpr int ROUTE_BLOCK = 1024;           // assignments per block of the permutation kernels
constexpr int ROUTE_WARPS = ROUTE_BLOCK / 32;

// ---------------------------------------------------------------- top-k
// One warp per token, the probabilities in registers.
template <int REG>
__global__ void __launch_bounds__(256) route_topk_kernel(const void* __restrict__ logits, int dtype, int T, int E, int k,
                                                        int renorm, int weight_round, int32_t* __restrict__ topk_idx,
                                                        float* __restrict__ topk_w) {
  const int lane = threadIdx.x & 31;
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  grid_launch_dependents();
  grid_wait();
  if (t >= T) return;
  int idx;
  float w;
  warp_topk<REG>(logits, dtype, t, E, k, renorm, weight_round, &idx, &w);
  if (lane < k) {
    topk_idx[static_cast<int64_t>(t) * k + lane] = idx;
    topk_w[static_cast<int64_t>(t) * k + lane] = w;
  }
}

// ---------------------------------------------------------------- permutation
// Exact per-warp exclusive bases (a block holds up to 1024 assignments of one expert, so
// bases need 16 bits while per-warp counts fit a byte).
__device__ __forceinline__ void block_warp_bases(int E, const uint8_t* warp_cnt, uint16_t* warp_base, int* block_count) {
  for (int x = threadIdx.x; x < E; x += blockDim.x) {
    int run = 0;
#pragma unroll 8
    for (int w = 0; w < ROUTE_WARPS; ++w) {
      warp_base[w * E + x] = static_cast<uint16_t>(run);
      run += warp_cnt[w * E + x];
    }
    block_count[x] = run;
  }
}

struct RouteSmem {
  // laid out by hand in dynamic shared memory: counts, bases, block_count, scan scratch
  uint8_t* warp_cnt;    // [ROUTE_WARPS][E]
  uint16_t* warp_base;  // [ROUTE_WARPS][E]
  int* block_count;     // [E]
  int* scan;            // [E + 1]
};

__device__ __forceinline__ RouteSmem carve_route_smem(unsigned char* base, int E) {
  RouteSmem s;
  size_t off = 0;
  s.block_count = reinterpret_cast<int*>(base + off); off += sizeof(int) * E;
  s.scan = reinterpret_cast<int*>(base + off); off += sizeof(int) * (E + 1);
  s.warp_base = reinterpret_cast<uint16_t*>(base + off); off += sizeof(uint16_t) * ROUTE_WARPS * E;
  s.warp_cnt = reinterpret_cast<uint8_t*>(base + off);
  return s;
}

__host__ __device__ inline size_t route_smem_bytes_dev(int E) {
  return (sizeof(int) * E + sizeof(int) * (E + 1) + sizeof(uint16_t) * ROUTE_WARPS * E + static_cast<size_t>(ROUTE_WARPS) * E + 15) / 16 * 16;
}
static size_t route_smem_bytes(int E) { return route_smem_bytes_dev(E); }

// Per-block counting shared by the fused and the multi-block paths.  Returns this
// thread's rank inside its warp; warp_base / block_count are valid after the call.
__device__ __forceinline__ int block_count_and_rank(int e, int E, RouteSmem& s) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < (ROUTE_WARPS * E + 3) / 4; i += blockDim.x) reinterpret_cast<uint32_t*>(s.warp_cnt)[i] = 0u;
  __syncthreads();
  const unsigned peers = __match_any_sync(0xffffffffu, e);
  const int rank_w = __popc(peers & ((1u << lane) - 1u));
  if (e >= 0 && rank_w == 0) s.warp_cnt[warp * E + e] = static_cast<uint8_t>(__popc(peers));
  __syncthreads();
  block_warp_bases(E, s.warp_cnt, s.warp_base, s.block_count);
  __syncthreads();
  return rank_w;
}

// Exclusive scan of block_count[0..E) into scan[0..E], single block, E <= ROUTE_MAX_E.
__device__ __forceinline__ void block_exclusive_scan(const int* in, int* out, int E) {
  __shared__ int warp_tot[32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int x = threadIdx.x;
  int v = (x < E) ? in[x] : 0;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int n = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += n;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int t = warp_tot[lane];
    int ti = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, ti, o);
      if (lane >= o) ti += n;
    }
    warp_tot[lane] = ti - t;
  }
  __syncthreads();
  const int excl = incl - v + warp_tot[warp];
  if (x < E) out[x] = excl;
  if (x == E - 1) out[E] = excl + v;
  __syncthreads();
}

__device__ __forceinline__ void write_tile_table(const int* offsets /*[E+1] shared*/, int E, int tile_rows,
                                                 int32_t* tile_table, int max_tiles, int32_t* counts, int* scratch /*[E+1]*/,
                                                 int* tiles_per /*[E]*/) {
  if (tile_table == nullptr && counts == nullptr) return;
  for (int x = threadIdx.x; x < E; x += blockDim.x) {
    const int n = offsets[x + 1] - offsets[x];
    tiles_per[x] = (n + tile_rows - 1) / tile_rows;
  }
  __syncthreads();
  block_exclusive_scan(tiles_per, scratch, E);
  const int total_tiles = scratch[E];
  if (tile_table) {
    for (int x = threadIdx.x; x < E; x += blockDim.x) {
      const int a0 = offsets[x], n = offsets[x + 1] - offsets[x];
      int slot = scratch[x];
      for (int r = 0; r < n; r += tile_rows, ++slot) {
        tile_table[slot * 3 + 0] = x;
        tile_table[slot * 3 + 1] = a0 + r;
        tile_table[slot * 3 + 2] = min(tile_rows, n - r);
      }
    }
    for (int s = total_tiles + threadIdx.x; s < max_tiles; s += blockDim.x) {
      tile_table[s * 3 + 0] = 0;
      tile_table[s * 3 + 1] = 0;
      tile_table[s * 3 + 2] = 0;
    }
  }
  if (counts && threadIdx.x == 0) {
    counts[0] = offsets[E];
    counts[1] = total_tiles;
  }
}

// Routed expert id of assignment i -> packed id, or -1 (dropped).  Ids outside [0, num_routed) -- a gate that is not
// this library's own can hand in anything -- and map entries outside [0, E) are dropped instead of indexing with them.
__device__ __forceinline__ int local_expert(const int32_t* __restrict__ topk_idx, const int32_t* __restrict__ g2l, int i,
                                            int num_routed, int E) {
  int e = topk_idx[i];
  if (static_cast<unsigned>(e) >= static_cast<unsigned>(num_routed)) return -1;
  if (g2l) e = g2l[e];
  return static_cast<unsigned>(e) < static_cast<unsigned>(E) ? e : -1;
}

// A <= ROUTE_BLOCK: everything in one block.
__global__ void __launch_bounds__(ROUTE_BLOCK) route_build_fused_kernel(
    const int32_t* __restrict__ topk_idx, const float* __restrict__ topk_w, const int32_t* __restrict__ g2l, int num_routed,
    int A, int k, int E, int tile_rows, int32_t* __restrict__ token_indices, int32_t* __restrict__ expert_offsets,
    float* __restrict__ route_flat, int32_t* __restrict__ tile_table, int max_tiles, int32_t* __restrict__ counts) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  RouteSmem s = carve_route_smem(sm_raw, E);
  grid_launch_dependents();
  grid_wait();
  const int i = threadIdx.x;
  int e = -1;
  if (i < A) e = local_expert(topk_idx, g2l, i, num_routed, E);
  const int rank_w = block_count_and_rank(e, E, s);
  block_exclusive_scan(s.block_count, s.scan, E);
  for (int x = threadIdx.x; x <= E; x += blockDim.x) expert_offsets[x] = s.scan[x];
  if (e >= 0) {
    const int pos = s.scan[e] + s.warp_base[(threadIdx.x >> 5) * E + e] + rank_w;
    token_indices[pos] = i / k;
    route_flat[pos] = topk_w[i];
  }
  __syncthreads();
  // reuse block_count / warp_base storage as scratch for the tile table
  write_tile_table(s.scan, E, tile_rows, tile_table, max_tiles, counts, reinterpret_cast<int*>(s.warp_base), s.block_count);
}

// Up to PLACE_CTAS x 1024 x PLACE_ROUNDS assignments by one cluster.  A CTA takes `rounds` x 1024 consecutive ones, a warp `rounds` x 32 of
// them, which it counts round by round into a table of its own; prefixes over the warps, over the CTAs (distributed shared memory) and
// over the experts give every assignment its place.
constexpr int PLACE_CTAS = 8, PLACE_ROUNDS = 8;
template <int ROUNDS>
__global__ void __launch_bounds__(ROUTE_BLOCK) route_place_kernel(
    const int32_t* __restrict__ topk_idx, const float* __restrict__ topk_w, const int32_t* __restrict__ g2l, int num_routed,
    int A, int k, int E, int tile_rows, int32_t* __restrict__ token_indices, int32_t* __restrict__ expert_offsets,
    float* __restrict__ route_flat, int32_t* __restrict__ tile_table, int max_tiles, int32_t* __restrict__ counts) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) unsigned char sm_raw[];
  const RouteSmem s = carve_route_smem(sm_raw, E);      // warp_base: counts, then prefixes over the warps; block_count: this CTA's counts
  int* const total = reinterpret_cast<int*>(sm_raw + route_smem_bytes_dev(E));
  const cg::cluster_group cluster = cg::this_cluster();
  const int rank = static_cast<int>(cluster.block_rank()), ctas = static_cast<int>(cluster.num_blocks());
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  grid_launch_dependents();
  for (int i = threadIdx.x; i < ROUTE_WARPS * E / 2; i += ROUTE_BLOCK) reinterpret_cast<uint32_t*>(s.warp_base)[i] = 0u;
  grid_wait();
  const int i0 = (rank * ROUTE_WARPS + warp) * (32 * ROUNDS) + lane;
  int e[ROUNDS], pos[ROUNDS];
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) e[r] = i0 + 32 * r < A ? local_expert(topk_idx, g2l, i0 + 32 * r, num_routed, E) : -1;
  __syncthreads();
  uint16_t* const mine = s.warp_base + warp * E;
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) {
    const unsigned peers = __match_any_sync(0xffffffffu, e[r]);
    const int below = __popc(peers & ((1u << lane) - 1u)), had = e[r] >= 0 ? mine[e[r]] : 0;
    __syncwarp();
    if (e[r] >= 0 && below == 0) mine[e[r]] = static_cast<uint16_t>(had + __popc(peers));
    __syncwarp();
    pos[r] = had + below;
  }
  __syncthreads();
  for (int x = threadIdx.x; x < E; x += ROUTE_BLOCK) {
    int run = 0;
#pragma unroll 8
    for (int w = 0; w < ROUTE_WARPS; ++w) {
      const int c = s.warp_base[w * E + x];
      s.warp_base[w * E + x] = static_cast<uint16_t>(run);      // a CTA holds at most PLACE_ROUNDS x 1024 of an expert
      run += c;
    }
    s.block_count[x] = run;
  }
  cluster.sync();
  int before = 0;
  const int x = threadIdx.x;
  if (x < E) {
    int all = 0;
#pragma unroll
    for (int c = 0; c < PLACE_CTAS; ++c) {
      const int n = c < ctas ? cluster.map_shared_rank(s.block_count, c)[x] : 0;
      before += c < rank ? n : 0;
      all += n;
    }
    total[x] = all;
  }
  const auto read = cluster.barrier_arrive();              // a CTA's counts may go once everybody has read them
  __syncthreads();
  block_exclusive_scan(total, s.scan, E);
  if (x < E) total[x] = s.scan[x] + before;                // where this CTA's assignments of the expert start
  __syncthreads();
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) {
    if (e[r] < 0) continue;
    const int at = total[e[r]] + mine[e[r]] + pos[r], i = i0 + 32 * r;
    token_indices[at] = i / k;
    route_flat[at] = topk_w[i];
  }
  cluster.barrier_wait(cg::cluster_group::arrival_token(read));
  if (rank == 0) {
    for (int j = threadIdx.x; j <= E; j += ROUTE_BLOCK) expert_offsets[j] = s.scan[j];
    __syncthreads();
    write_tile_table(s.scan, E, tile_rows, tile_table, max_tiles, counts, reinterpret_cast<int*>(s.warp_base), s.block_count);
  }
}

// More assignments: counts per block of assignments, prefixes across the blocks, scatter.
__global__ void __launch_bounds__(ROUTE_BLOCK) route_count_kernel(const int32_t* __restrict__ topk_idx,
                                                                 const int32_t* __restrict__ g2l, int num_routed, int A, int E,
                                                                 int32_t* __restrict__ block_hist /*[nblocks][E]*/) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  RouteSmem s = carve_route_smem(sm_raw, E);
  grid_launch_dependents();
  grid_wait();
  const int i = blockIdx.x * ROUTE_BLOCK + threadIdx.x;
  int e = -1;
  if (i < A) e = local_expert(topk_idx, g2l, i, num_routed, E);
  block_count_and_rank(e, E, s);
  for (int x = threadIdx.x; x < E; x += blockDim.x) block_hist[static_cast<int64_t>(blockIdx.x) * E + x] = s.block_count[x];
}

// block_hist -> exclusive prefixes over the blocks, and the experts' totals.  A CTA owns 32 experts (a lane each), its
// warps cut the blocks into runs: sums, a prefix over the runs in shared memory, prefixes.
__global__ void __launch_bounds__(ROUTE_BLOCK) route_scan_kernel(int32_t* __restrict__ block_hist, int nblocks, int E,
                                                                int32_t* __restrict__ total) {
  __shared__ int run_tot[ROUTE_WARPS][33];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, x = blockIdx.x * 32 + lane;
  grid_launch_dependents();
  grid_wait();
  const int len = (nblocks + ROUTE_WARPS - 1) / ROUTE_WARPS, b0 = warp * len, b1 = min(nblocks, b0 + len);
  int sum = 0;
  if (x < E)
#pragma unroll 8
    for (int b = b0; b < b1; ++b) sum += block_hist[static_cast<int64_t>(b) * E + x];
  run_tot[warp][lane] = sum;
  __syncthreads();
  int run = 0;
  for (int w = 0; w < warp; ++w) run += run_tot[w][lane];
  if (x >= E) return;
#pragma unroll 8
  for (int b = b0; b < b1; ++b) {
    const int v = block_hist[static_cast<int64_t>(b) * E + x];
    block_hist[static_cast<int64_t>(b) * E + x] = run;
    run += v;
  }
  if (warp == ROUTE_WARPS - 1) total[x] = run;
}

// Every block scans the totals for itself; the first one also writes the offsets and the tile table.
__global__ void __launch_bounds__(ROUTE_BLOCK) route_scatter_kernel(
    const int32_t* __restrict__ topk_idx, const float* __restrict__ topk_w, const int32_t* __restrict__ g2l, int num_routed,
    int A, int k, int E, const int32_t* __restrict__ block_hist, const int32_t* __restrict__ total, int tile_rows,
    int32_t* __restrict__ expert_offsets, int32_t* __restrict__ token_indices, float* __restrict__ route_flat, int32_t* __restrict__ tile_table,
    int max_tiles, int32_t* __restrict__ counts) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  RouteSmem s = carve_route_smem(sm_raw, E);
  grid_launch_dependents();
  grid_wait();
  block_exclusive_scan(total, s.scan, E);
  const int i = blockIdx.x * ROUTE_BLOCK + threadIdx.x;
  int e = -1;
  if (i < A) e = local_expert(topk_idx, g2l, i, num_routed, E);
  const int rank_w = block_count_and_rank(e, E, s);
  if (e >= 0) {
    const int pos = s.scan[e] + block_hist[static_cast<int64_t>(blockIdx.x) * E + e] + s.warp_base[(threadIdx.x >> 5) * E + e] + rank_w;
    token_indices[pos] = i / k;
    route_flat[pos] = topk_w[i];
  }
  if (blockIdx.x == 0) {
    for (int x = threadIdx.x; x <= E; x += blockDim.x) expert_offsets[x] = s.scan[x];
    __syncthreads();
    write_tile_table(s.scan, E, tile_rows, tile_table, max_tiles, counts, reinterpret_cast<int*>(s.warp_base), s.block_count);
  }
}

// f<REG>() for the register class of E experts (E <= ROUTE_MAX_E)
#define BM_TOPK_CLASS(E, CALL)                          \
  do {                                                  \
    if ((E) <= 64) { constexpr int REG = 2; CALL; }     \
    else if ((E) <= 128) { constexpr int REG = 4; CALL; }  \
    else if ((E) <= 256) { constexpr int REG = 8; CALL; }  \
    else if ((E) <= 512) { constexpr int REG = 16; CALL; } \
    else { constexpr int REG = 32; CALL; }              \
  } while (0)

static int set_route_attributes(int dev) {
  static PerDeviceOnce attr_once;
  if (attr_once.is_done(dev)) return BM_OK;
  const int big = static_cast<int>(route_smem_bytes(ROUTE_MAX_E));
  BM_CUDA(cudaFuncSetAttribute(route_build_fused_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
  BM_CUDA(cudaFuncSetAttribute(route_count_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
  BM_CUDA(cudaFuncSetAttribute(route_scatter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
  for (auto* kernel : {route_place_kernel<1>, route_place_kernel<2>, route_place_kernel<4>, route_place_kernel<8>})
    BM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, big + ROUTE_MAX_E * static_cast<int>(sizeof(int))));
  attr_once.mark(dev);
  return BM_OK;
}

}  // namespace bm

static int route_topk(const void* logits, int logits_dtype, int32_t T, int32_t E, int32_t k, int32_t renorm,
                             int32_t weight_round, int32_t* topk_idx, float* topk_w, bm::LaunchAfter after, cudaStream_t st) {
  using namespace bm;
  BM_REQUIRE(T >= 0 && E > 0 && k > 0, BM_ERR_INVALID_ARG, "route_topk: bad sizes T=%d E=%d k=%d", T, E, k);
  BM_REQUIRE(k <= 32 && k <= E, BM_ERR_UNSUPPORTED, "route_topk: top_k=%d must be <= min(32, E=%d)", k, E);
  BM_REQUIRE(E <= ROUTE_MAX_E, BM_ERR_UNSUPPORTED, "route_topk: E=%d exceeds %d", E, ROUTE_MAX_E);
  BM_REQUIRE(logits_dtype >= BM_F16 && logits_dtype <= BM_F32, BM_ERR_INVALID_ARG, "route_topk: bad logits dtype");
  if (T == 0) return BM_OK;
  BM_REQUIRE(logits && topk_idx && topk_w, BM_ERR_INVALID_ARG, "route_topk: null pointer");
  const int warps = 8;
  BM_TOPK_CLASS(E, BM_CUDA(launch_after(after, 1, route_topk_kernel<REG>, dim3((T + warps - 1) / warps), warps * 32, 0, st, logits, logits_dtype, T,
                                        E, k, renorm, weight_round, topk_idx, topk_w)));
  BM_LAUNCH_CHECK("route_topk_kernel");
  return BM_OK;
}

extern "C" int bm_route_topk(const void* logits, int logits_dtype, int32_t T, int32_t E, int32_t k, int32_t renorm,
                             int32_t weight_round, int32_t* topk_idx, float* topk_w, void* stream) {
  bm::NvtxRange nvtx_range("bm_route_topk");
  return route_topk(logits, logits_dtype, T, E, k, renorm, weight_round, topk_idx, topk_w, bm::AFTER_ALL, static_cast<cudaStream_t>(stream));
}

extern "C" int32_t bm_route_max_tiles(int32_t T, int32_t k, int32_t num_local, int32_t tile_rows) {
  if (tile_rows <= 0) return 0;
  const int64_t A = static_cast<int64_t>(T) * k;
  // every expert wastes at most one partial tile
  const int64_t bound = A / tile_rows + num_local;
  const int64_t m = bound < A ? bound : A;  // a tile holds at least one row
  return static_cast<int32_t>(m > 0 ? m : 1);
}

extern "C" size_t bm_route_build_workspace_bytes(int32_t T, int32_t k, int32_t num_local) {
  const int64_t A = static_cast<int64_t>(T) * k;
  if (A <= bm::ROUTE_BLOCK) return 0;
  return bm::align_up(static_cast<size_t>((A + bm::ROUTE_BLOCK - 1) / bm::ROUTE_BLOCK + 1) * num_local * sizeof(int32_t), 256);     // histograms, totals
}

static int route_build(const int32_t* topk_idx, const float* topk_w, const int32_t* global_to_local,
                              int32_t num_routed, int32_t T,
                              int32_t k, int32_t num_local, int32_t tile_rows, int32_t* token_indices,
                              int32_t* expert_offsets, float* route_flat, int32_t* tile_table, int32_t* counts,
                              void* workspace, size_t workspace_bytes, bm::LaunchAfter after, bool beside_follows, cudaStream_t st) {
  using namespace bm;
  BM_REQUIRE(T >= 0 && k > 0 && num_local > 0 && num_routed > 0, BM_ERR_INVALID_ARG, "route_build: bad sizes");
  BM_REQUIRE(global_to_local != nullptr || num_routed == num_local, BM_ERR_INVALID_ARG,
             "route_build: %d routed experts but %d packed and no id map", num_routed, num_local);
  BM_REQUIRE(num_local <= ROUTE_MAX_E, BM_ERR_UNSUPPORTED, "route_build: %d experts exceed %d", num_local, ROUTE_MAX_E);
  BM_REQUIRE(tile_rows > 0, BM_ERR_INVALID_ARG, "route_build: tile_rows must be positive");
  BM_REQUIRE(expert_offsets, BM_ERR_INVALID_ARG, "route_build: null expert_offsets");
  const int64_t A64 = static_cast<int64_t>(T) * k;
  BM_REQUIRE(A64 < (1ll << 30), BM_ERR_UNSUPPORTED, "route_build: too many assignments");
  const int A = static_cast<int>(A64);
  BM_REQUIRE(A == 0 || (topk_idx && topk_w && token_indices && route_flat), BM_ERR_INVALID_ARG, "route_build: null pointer");
  const int max_tiles = bm_route_max_tiles(T, k, num_local, tile_rows);
  const size_t smem = route_smem_bytes(num_local);
  int dev = -1;
  BM_CUDA(cudaGetDevice(&dev));
  const int rc = set_route_attributes(dev);
  if (rc) return rc;
  if (A <= ROUTE_BLOCK) {
    BM_CUDA(launch_after(after, 1, route_build_fused_kernel, dim3(1), ROUTE_BLOCK, smem, st, topk_idx, topk_w, global_to_local, num_routed, A, k,
                         num_local, tile_rows, token_indices, expert_offsets, route_flat, tile_table, max_tiles, counts));
    BM_LAUNCH_CHECK("route_build_fused_kernel");
    return BM_OK;
  }
  const int nblocks = (A + ROUTE_BLOCK - 1) / ROUTE_BLOCK;
  const size_t need = bm_route_build_workspace_bytes(T, k, num_local);
  BM_REQUIRE(workspace && workspace_bytes >= need, BM_ERR_WORKSPACE, "route_build: workspace of %zu bytes needed, %zu given",
             need, workspace_bytes);
  // One launch of a cluster against three over all SMs, us on 128 experts: 8192 assignments 6.6 / 10.8, 16384 9.0 / 11.3, 32768 13.6 / 11.4,
  // 65536 23.4 / 12.5 (eight SMs scatter 4-byte words).  With a launch beside it the cluster's time does not show up to the largest.
  if (A <= PLACE_CTAS * ROUTE_BLOCK * (beside_follows ? PLACE_ROUNDS : 2)) {
    int rounds = 1, ctas = 2;
    while (rounds * PLACE_CTAS * ROUTE_BLOCK < A) rounds *= 2;
    while (ctas * rounds * ROUTE_BLOCK < A) ctas *= 2;
    auto* kernel = rounds == 1 ? route_place_kernel<1> : rounds == 2 ? route_place_kernel<2> : rounds == 4 ? route_place_kernel<4> : route_place_kernel<8>;
    BM_CUDA(launch_after(after, ctas, kernel, dim3(ctas), ROUTE_BLOCK, smem + num_local * sizeof(int), st, topk_idx, topk_w, global_to_local, num_routed,
                         A, k, num_local, tile_rows, token_indices, expert_offsets, route_flat, tile_table, max_tiles, counts));
    BM_LAUNCH_CHECK("route_place_kernel");
    return BM_OK;
  }
  int32_t* total = static_cast<int32_t*>(workspace);
  int32_t* block_hist = total + num_local;
  BM_CUDA(launch_after(after, 1, route_count_kernel, dim3(nblocks), ROUTE_BLOCK, smem, st, topk_idx, global_to_local, num_routed, A, num_local, block_hist));
  BM_LAUNCH_CHECK("route_count_kernel");
  BM_CUDA(launch_after(AFTER_READS, 1, route_scan_kernel, dim3((num_local + 31) / 32), ROUTE_BLOCK, 0, st, block_hist, nblocks, num_local, total));
  BM_LAUNCH_CHECK("route_scan_kernel");
  BM_CUDA(launch_after(AFTER_READS, 1, route_scatter_kernel, dim3(nblocks), ROUTE_BLOCK, smem, st, topk_idx, topk_w, global_to_local, num_routed, A, k,
                       num_local, block_hist, total, tile_rows, expert_offsets, token_indices, route_flat, tile_table, max_tiles, counts));
  BM_LAUNCH_CHECK("route_scatter_kernel");
  return BM_OK;
}

extern "C" int bm_route_build(const int32_t* topk_idx, const float* topk_w, const int32_t* global_to_local,
                              int32_t num_routed, int32_t T,
                              int32_t k, int32_t num_local, int32_t tile_rows, int32_t* token_indices,
                              int32_t* expert_offsets, float* route_flat, int32_t* tile_table, int32_t* counts,
                              void* workspace, size_t workspace_bytes, void* stream) {
  bm::NvtxRange nvtx_range("bm_route_build");
  return route_build(topk_idx, topk_w, global_to_local, num_routed, T, k, num_local, tile_rows, token_indices, expert_offsets, route_flat,
                     tile_table, counts, workspace, workspace_bytes, bm::AFTER_ALL, false, static_cast<cudaStream_t>(stream));
}

int bm::route_tokens(const void* logits, int logits_dtype, int32_t T, int32_t E_routed, int32_t k, int32_t renorm, int32_t weight_round,
                     const int32_t* global_to_local, int32_t num_local, int32_t tile_rows, int32_t* topk_idx, float* topk_w,
                     int32_t* token_indices, int32_t* expert_offsets, float* route_flat, int32_t* tile_table, int32_t* counts, void* workspace,
                     size_t workspace_bytes, LaunchAfter after, bool beside_follows, cudaStream_t st) {
  const int rc = route_topk(logits, logits_dtype, T, E_routed, k, renorm, weight_round, topk_idx, topk_w, after, st);
  if (rc) return rc;
  return route_build(topk_idx, topk_w, global_to_local, E_routed, T, k, num_local, tile_rows, token_indices, expert_offsets, route_flat, tile_table,
                     counts, workspace, workspace_bytes, T > 0 ? AFTER_READS : after, beside_follows, st);
}

extern "C" int bm_route(const void* logits, int logits_dtype, int32_t T, int32_t E_routed, int32_t k, int32_t renorm,
                        int32_t weight_round, const int32_t* global_to_local, int32_t num_local, int32_t tile_rows,
                        int32_t* topk_idx, float* topk_w, int32_t* token_indices, int32_t* expert_offsets,
                        float* route_flat, int32_t* tile_table, int32_t* counts, void* workspace, size_t workspace_bytes,
                        void* stream) {
  bm::NvtxRange nvtx_range("bm_route");
  return bm::route_tokens(logits, logits_dtype, T, E_routed, k, renorm, weight_round, global_to_local, num_local, tile_rows, topk_idx, topk_w,
                          token_indices, expert_offsets, route_flat, tile_table, counts, workspace, workspace_bytes, bm::AFTER_ALL, false,
                          static_cast<cudaStream_t>(stream));
}
