// Shared declarations of the bitsmoe_b200 library (host + device).
#pragma once

#include <nvtx3/nvToolsExt.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <vector>

#include "../../include/bitsmoe_b200.h"

namespace bm {

constexpr int K_SLAB = 64;     // rows per slab at most
constexpr int N_TILE = 128;    // columns per scale group
constexpr int K_STAGE = 16;    // rows per payload stage
constexpr int N_MICRO = 32;    // columns per bit-plane word
constexpr int MICROS = N_TILE / N_MICRO;

int set_error(int status, const char* fmt, ...);
void count_launch();   // every kernel launch of the library is counted (bm_launch_count)

#define BM_REQUIRE(cond, status, ...)                       \
  do {                                                      \
    if (!(cond)) return ::bm::set_error((status), __VA_ARGS__); \
  } while (0)

#define BM_CUDA(expr)                                                                   \
  do {                                                                                  \
    cudaError_t _e = (expr);                                                            \
    if (_e != cudaSuccess)                                                              \
      return ::bm::set_error(BM_ERR_CUDA, "%s failed: %s", #expr, cudaGetErrorString(_e)); \
  } while (0)

#define BM_LAUNCH_CHECK(name)                                                              \
  do {                                                                                     \
    ::bm::count_launch();                                                                  \
    cudaError_t _e = cudaGetLastError();                                                   \
    if (_e != cudaSuccess)                                                                 \
      return ::bm::set_error(BM_ERR_CUDA, "launch of %s failed: %s", name, cudaGetErrorString(_e)); \
  } while (0)

// Set-up that belongs to a (kernel, device) pair -- cudaFuncSetAttribute, occupancy queries -- runs once per device
// ordinal, not once per process: a second GPU driven from the same process needs its own.  Two host threads may both
// run the set-up for a device (it is idempotent); the flag only publishes that it has been done.
constexpr int MAX_DEVICES = 64;
struct PerDeviceOnce {
  std::atomic<unsigned char> done[MAX_DEVICES] = {};
  bool is_done(int dev) const { return dev >= 0 && dev < MAX_DEVICES && done[dev].load(std::memory_order_acquire) != 0; }
  void mark(int dev) { if (dev >= 0 && dev < MAX_DEVICES) done[dev].store(1, std::memory_order_release); }
};

// What a kernel's launch may overlap of the launches before it on the same stream (programmatic serialisation).
enum LaunchAfter {
  AFTER_ALL = 0,       // an ordinary launch
  AFTER_READS = 1,     // starts while they drain, waits for them before it touches memory
  AFTER_BESIDE = 2     // reads nothing that they write and writes nothing that they read: waits for them before it ends, so that
                       // whoever waits for it has waited for them
};
template <typename... P, typename... A>
inline cudaError_t launch_after(LaunchAfter after, int cluster, void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  if (after != AFTER_ALL) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = cluster;
    attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs++].val.clusterDim.z = 1;
  }
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
// The next launch may be set up / what the launches before wrote is there (both without effect on ordinary launches).
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// One packed matrix as the device sees it (pointers into the caller's buffers).
struct MatDev {
  const uint32_t* payload;
  const int32_t* rank_idx;
  const int32_t* tile_meta;
  const int32_t* slab_meta;
  const __half* scale;
  const __half* s;
  int32_t n_slabs;
  int32_t n_tile_rows;
  int32_t n_rows;
  int32_t pad_;
};

struct ExpertDev {
  MatDev m[3];
};

// Host mirror of one slab (validated at plan time).
struct SlabHost {
  int32_t bits, k_slab, rank_off, tile_off, tile_end;
};

struct MatHost {
  std::vector<SlabHost> slabs;
  std::vector<int32_t> tile_meta;  // [n_tile_rows * 3]
  std::vector<int32_t> rank_idx;   // [n_rows]
  int64_t bytes = 0;               // as stored by the reference
  int32_t n_rows = 0;
};

constexpr int DEFAULT_WAIT_LIMIT_US = 2000000;
constexpr int FAST_MAX_TOK = 8;    // assignments per pass of the decode kernel (one MMA N-block)

struct FastMat {
  int32_t nblk[2];      // 16-slot blocks in the nibble group (3/4-bit rows), in the dense 2-bit group (1/2-bit rows)
  int32_t nslots;       // 16 * (nblk[0] + nblk[1])
  int32_t words;        // uint32 words per tile = 256 nblk[0] + 128 nblk[1]
  int32_t tab_off;      // byte offset (from arena base) of [int16 rank[nslots] | fp16 s[nslots] | int16 row[nslots]]
  int32_t pad_[3];
};

struct FastExpert {
  FastMat m[3];
  int64_t unit_base;    // byte offset of tile 0's unit block from arena base
  int32_t unit_bytes;   // bytes per unit block (multiple of 128)
  int32_t sec_off[6];   // byte offsets inside a unit: [0..2] scales of g,u,d, [3..5] words of g,u,d; sec_off[3+m] == sec_off[m] + 2 * nslots(m)
  int32_t pad_;
};

// Token-side table of one expert, built at load time: what a kernel needs to put token rows into an expert's operand order
// and its sums back into rank order, as one contiguous copy.  All experts of a layer share the offsets.
struct TokTabHead {
  FastExpert fe;
  int32_t loose;            // gate or up has slots that no rank's position names: without a row, or with a rank that another slot has too
  uint32_t broken[2][4];    // gate, up: octets of ranks that are not one 16-byte piece of the operand row (bit per octet)
};
constexpr int TOKTAB_MAX_RANK = 1024;
struct TokTab {
  int s_r, pos_r, oct_r;    // [gate, up][rank] factor s (fp16), contraction position or -1 (int16); per octet: its piece or -1 (int16)
  int s_d, rank_d, oct_d;   // per down slot: factor (fp32), rank or -1 (int16); per eight slots: first rank of an aligned octet or -1
  int bytes;
  __host__ __device__ TokTab(int rank_in, int max_slots) {
    auto up = [](int v) { return (v + 15) & ~15; };
    s_r = up(static_cast<int>(sizeof(TokTabHead)));
    pos_r = s_r + 4 * rank_in;
    oct_r = pos_r + 4 * rank_in;
    s_d = up(oct_r + rank_in / 2);
    rank_d = s_d + 4 * max_slots;
    oct_d = rank_d + 2 * max_slots;
    bytes = up(oct_d + max_slots / 4);
  }
};

struct FastPlan {
  bool ok = false;
  std::vector<FastExpert> experts;
  std::vector<int16_t> slot_row;      // concatenated per (expert, matrix): slot -> local row or -1
  std::vector<int32_t> slot_row_off;  // [E*3] element offset into slot_row
  size_t table_off = 0;               // FastExpert table
  size_t toktab_off = 0;              // token-side tables (rank_in <= TOKTAB_MAX_RANK), 0 = none
  size_t total = 0;
  int max_unit_bytes = 0, max_slots = 0, max_words = 0;
};

__host__ __device__ inline int words_per_row(int bits) { return bits == 16 ? 16 : bits; }

inline bool supported_bits(int b) { return b == 1 || b == 2 || b == 3 || b == 4 || b == 6 || b == 8 || b == 16; }

__device__ __forceinline__ float load_act(const void* p, int dtype, int64_t i) {
  if (dtype == BM_F16) return __half2float(reinterpret_cast<const __half*>(p)[i]);
  if (dtype == BM_BF16) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]);
  return reinterpret_cast<const float*>(p)[i];
}

__device__ __forceinline__ void store_act(void* p, int dtype, int64_t i, float v) {
  if (dtype == BM_F16) reinterpret_cast<__half*>(p)[i] = __float2half_rn(v);
  else if (dtype == BM_BF16) reinterpret_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(v);
  else reinterpret_cast<float*>(p)[i] = v;
}

// Accumulation into rank_accum: fp32 atomics (as bitsmoe/algorithms/cpp/mlp_forward.cu:2062 does), or -- the
// deterministic mode -- 64-bit fixed-point atomics: integer addition is associative, so the sum does not depend on the
// order in which CTAs arrive and two runs are bit-identical.  2^40 leaves 2^23 of range and 1e-12 of resolution.
constexpr float ACC_FIXED_SCALE = 1099511627776.f;
__device__ __forceinline__ void acc_add(float* __restrict__ acc32, long long* __restrict__ acc64, int64_t idx, float v) {
  if (acc64) atomicAdd(reinterpret_cast<unsigned long long*>(acc64) + idx, static_cast<unsigned long long>(__float2ll_rn(v * ACC_FIXED_SCALE)));
  else atomicAdd(acc32 + idx, v);
}

// C[M,N] = A[M,K] . B[N,K]^T ; up to two problems sharing A's shape in one launch.
struct GemmArgs {
  const void* A[2];
  const __half* B[2];
  void* C[2];
  const void* residual;  // same dtype / shape as C, problem 0 only
  int a_dtype, c_dtype;
  int round_a_f16;       // round an fp32 A through fp16 first (rank_accum.half())
  int M, N, K;
  int vec_a, vec_b;      // every A / B starts on a 16-byte boundary (filled in by the launcher)
};

// What 16-byte loads and tiled copies need of a base address (null counts as aligned).
template <typename... P>
inline bool aligned16(const P*... p) {
  return ((reinterpret_cast<uintptr_t>(p) | ...) & 15u) == 0;
}

inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }
__host__ __device__ inline size_t align_up_c(size_t v, size_t a) { return (v + a - 1) / a * a; }

// Arguments of the tensor-core basis products (gemm_tma.cu, gemm_tc.cu): C[z] = X . W[z]^T (+ residual for z = 0).
struct GemmTcArgs {
  const void* X;          // [M, K]
  const __half* W[2];     // [N, K] each
  void* C[2];             // [M, N] each
  const void* residual;   // [M, N] (W[0] only) or null
  int M, N, K;
  int x_dtype, c_dtype;
  int* status;
  LaunchAfter after;
  float4* zero;           // optional buffer cleared on the way (the expert stage's accumulator), 16-byte units
  int64_t zero_n;
};
int launch_gemm_tc(const GemmTcArgs& a, int problems, cudaStream_t st);
// The tiled-copy kernel (gemm_tma.cu): several stacks of weight rows sharing X in one launch.  C[m][n] = X[m] . W[n], or
// with W_up the gated pair silu(X[m] . W[n]) * (X[m] . W_up[n]).
constexpr int GEMM_MAX_SEG = 4;
struct GemmSeg {
  const __half* W;          // [rows, K]
  const __half* W_up;
  void* C;                  // [M, rows]
  int rows, c_dtype;
};
struct GemmTmaArgs {
  const void* X;            // [M, K]
  int x_dtype, M, K;
  GemmSeg seg[GEMM_MAX_SEG];
  int n_seg;
  // second contraction of a lone stack: += X2 [M, K2] fp16 . W2 [rows, K2]^T
  const __half* X2;
  const __half* W2;
  int K2;
  const void* residual;     // added to stack 0, of its type
  const float* row_gate;    // [M] factor of the gated pair's rows, or null
  int* status;
  LaunchAfter after;
  float4* zero;             // optional buffer cleared on the way, 16-byte units
  int64_t zero_n;
};
// BM_ERR_UNSUPPORTED, with nothing launched, when a shape or pointer does not suit tiled copies.
int launch_gemm_tma(const GemmTmaArgs& a, cudaStream_t st);
// One or two products sharing X: the tiled-copy kernel, else launch_gemm_tc.
int launch_gemm_basis(const GemmTcArgs& a, int problems, cudaStream_t st);

// bm_route with its first launch placed as `after` says; `beside_follows`: the next launch on the stream is an AFTER_BESIDE one.
int route_tokens(const void* logits, int logits_dtype, int32_t T, int32_t E_routed, int32_t k, int32_t renorm, int32_t weight_round,
                 const int32_t* global_to_local, int32_t num_local, int32_t tile_rows, int32_t* topk_idx, float* topk_w,
                 int32_t* token_indices, int32_t* expert_offsets, float* route_flat, int32_t* tile_table, int32_t* counts, void* workspace,
                 size_t workspace_bytes, LaunchAfter after, bool beside_follows, cudaStream_t st);

// NVTX range around a public entry point (route / projection / experts / combine / exchange show up as named ranges
// in a timeline tool; without a tool attached a push or pop is one null-pointer test).
struct NvtxRange {
  explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
  NvtxRange(const NvtxRange&) = delete;
  NvtxRange& operator=(const NvtxRange&) = delete;
};

}  // namespace bm

struct bm_layer {
  int32_t num_experts = 0, hidden = 0, intermediate = 0, rank_in = 0, rank_out = 0, n_tiles = 0;
  int32_t max_rows = 0;            // largest n_rows over all matrices
  int device = 0;
  const __half* vh_gate = nullptr;
  const __half* vh_up = nullptr;
  const __half* u_down = nullptr;
  std::vector<bm::MatHost> host[3];   // [which][expert]
  std::vector<bm_matrix_t> src[3];    // caller's descriptors (pointers kept)
  bm::ExpertDev* experts_dev = nullptr;  // in the arena
  void* arena = nullptr;
  size_t arena_bytes = 0;
  bool fast_ok = false;            // every slab is 1/2/3/4-bit and shapes fit the decode / tensor paths
  const bm::FastExpert* fast_dev = nullptr;   // in the arena
  std::vector<bm::FastExpert> fast_host;
  const unsigned char* toktab_dev = nullptr;  // in the arena
  int max_unit_bytes = 0, max_slots = 0, max_words = 0;
  // launch geometry of the decode kernel on this layer's device (plan_experts_decode)
  bool dec_ok = false;
  bool deterministic = false;      // rank_accum through 64-bit fixed-point atomics (bm_layer_set_option)
  int dec_ring = 0, dec_sec_bytes = 0, dec_grid = 0, dec_act_bufs = 2, dec_ctas = 0, dec_force_ctas = 0;
  size_t dec_smem = 0;
  int sms = 148;                   // of the device that the layer was created on
  int bat_ring = 0, bat_sec_bytes = 0, bat_smem = 0, bat_grid = 0;      // of experts_batch_kernel (bat_ring 0: not for this layer)
  int wait_limit_us = bm::DEFAULT_WAIT_LIMIT_US;   // of the packed-expert kernels' waits (bm_layer_set_option)
  int* status_dev = nullptr;       // device flag set by a kernel whose bounded wait gave up
};
