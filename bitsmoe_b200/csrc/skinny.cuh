// Launch interface of the small-batch products (skinny_nt.cu) and of the routing cluster (route_small.cuh).
#pragma once

#include "common.cuh"

namespace bm {

constexpr int SKINNY_MAX_TOKENS = 256;   // callers hand over to the tcgen05 GEMM at their own, lower counts where it takes the shape
constexpr int SK_MAX_SEG = 6;

// One stack of output rows: C[n][m] = sum_k W[m][k] X[n][k] for m < rows, stored at C[n * rows + m].  With W_up set the
// stack is a gated pair: C[n][m] = silu(W[m] . X[n]) * (W_up[m] . X[n]).
struct SkSeg {
  const __half* W;
  const __half* W_up;
  void* C;
  int rows, c_dtype;
  int w_bf16;              // W, W_up are bf16 and are rounded to fp16 on the way to shared memory
  int tile0;               // first row tile of this stack (filled in by the launcher)
};

// Routing of up to 256 tokens by one thread-block cluster (route_small.cuh).
struct RouteSmallArgs {
  const void* logits;
  int logits_dtype;
  int T, E, k, renorm, weight_round;
  int32_t* token_indices;
  int32_t* expert_offsets;
  float* route_flat;
};

struct SkinnyArgs {
  SkSeg seg[SK_MAX_SEG];
  int n_seg;
  const void* X;           // [N, K]
  int N, K, x_dtype;
  const float* x_gate;     // [N] or null (fp32 X): X[n] is scaled by sigmoid(x_gate[n])
  // second contraction of stack 0 (unsplit launches only): += sum_k W2[m][k] X2[n][k] * sigmoid(x2_gate[n])
  const __half* W2;        // [rows, K2] or null
  const float* X2;         // [N, K2]
  const float* x2_gate;    // [N] logits or null
  int K2, w2_bf16;
  const void* residual;    // [N, rows] of stack 0, c_dtype of stack 0, or null
  int splits;              // cluster size along K: 1, 2, 4 or 8
  float4* zero;            // optional buffer the grid clears on its way (the next kernel's accumulator), 16-byte units
  int zero_n;
  RouteSmallArgs route;    // route.T > 0: one more cluster routes these tokens (splits must be 8)
  // The launch may start while the kernel before it drains.  Weights are read before that kernel is complete, so only for
  // a launch that follows another one of the same entry point: whatever wrote the weights came before that one.
  int overlap;
  int row_tiles, clusters; // filled in by the launcher
};

// BM_ERR_UNSUPPORTED (nothing launched) when the shape does not tile; the caller then takes a general GEMM.
int launch_skinny_nt(SkinnyArgs a, cudaStream_t st);
bool skinny_fits(int K, int K2, int splits);
// Whether the product's grid is more than one wave of the device (three CTAs an SM).
bool skinny_many_waves(int row_tiles, int splits, int T);
// Cluster size along K for a product of `rows` output rows.
int skinny_splits(int rows, int K);

// gate[t] = sigmoid(x[t] . w) (dense.cu)
int launch_row_gate(const void* x, int x_dtype, const uint16_t* w, int w_dtype, int T, int H, float* gate, LaunchAfter after, cudaStream_t st);

bool route_small_fits(int T, int E, int k);
int launch_route_small(const RouteSmallArgs& a, cudaStream_t st);

}  // namespace bm
