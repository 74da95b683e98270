// Dense products around the packed experts, so that a whole MoE block runs inside the library:
//   router logits   logits = x . W_gate^T          (bitsmoe/models/qwen3moe/bitsmoe_block.py:45)
//   shared expert   y = (silu(x . Wg^T) * (x . Wu^T)) . Wd^T, optionally scaled per token by sigmoid(x . w)
//                   (bitsmoe/models/deepseekv2/bitsmoe_block.py:123-124, bitsmoe/models/qwen3next/bitsmoe_block.py:144-147)
// The products run on the same kernels as the shared-basis projections: the cluster split-K kernel for decode-sized
// batches, the tcgen05 GEMM above that, a CUDA-core GEMM for shapes neither takes.
#include "skinny.cuh"

namespace bm {

int launch_gemm_nt(const GemmArgs& g, int problems, cudaStream_t st);

// C_i [T, N] = X [T, K] . W_i [N, K]^T for `problems` (1 or 2) weight matrices sharing X; residual (problem 0 only) may
// be null.  Chooses the kernel by shape: where both suit, the skinny one up to `skinny_tokens`.
int dense_xwT(const void* X, int x_dtype, const __half* W0, const __half* W1, void* C0, void* C1, int c_dtype,
              const void* residual, int T, int N, int K, int problems, int* status, LaunchAfter after, int skinny_tokens, cudaStream_t st) {
  if (T == 0) return BM_OK;
  const bool aligned = aligned16(X, W0, W1), tiled = aligned && K % 64 == 0 && N % 8 == 0;
  if (T <= (tiled ? skinny_tokens : SKINNY_MAX_TOKENS) && aligned && K % 8 == 0) {
    SkinnyArgs a{};
    a.n_seg = problems;
    a.seg[0] = SkSeg{W0, nullptr, C0, N, c_dtype, 0, 0};
    a.seg[1] = SkSeg{W1, nullptr, C1, N, c_dtype, 0, 0};
    a.X = X; a.N = T; a.K = K; a.x_dtype = x_dtype; a.residual = residual;
    a.splits = skinny_splits(N * problems, K);
    a.overlap = after != AFTER_ALL;
    const int rc = launch_skinny_nt(a, st);
    if (rc != BM_ERR_UNSUPPORTED) return rc;
  }
  if (tiled) {
    GemmTcArgs t{};
    t.X = X; t.W[0] = W0; t.W[1] = problems > 1 ? W1 : W0; t.C[0] = C0; t.C[1] = problems > 1 ? C1 : C0;
    t.residual = residual; t.M = T; t.N = N; t.K = K; t.x_dtype = x_dtype; t.c_dtype = c_dtype; t.status = status;
    t.after = after;
    return launch_gemm_basis(t, problems, st);
  }
  GemmArgs g{};
  g.A[0] = g.A[1] = X;
  g.B[0] = W0; g.B[1] = problems > 1 ? W1 : W0;
  g.C[0] = C0; g.C[1] = problems > 1 ? C1 : C0;
  g.residual = residual;
  g.a_dtype = x_dtype; g.c_dtype = c_dtype; g.round_a_f16 = x_dtype == BM_F32 ? 1 : 0;
  g.M = T; g.N = N; g.K = K;
  return launch_gemm_nt(g, problems, st);
}

// The whole MLP of a decode batch in two launches: gate and up rows paired in the same CTA (z = silu(g) * u leaves in
// fp32) with the per-token gate's logit beside them, then the down product, which scales z by the gate as it rounds it.
static int dense_mlp_small(const void* x, int x_dtype, const __half* wg, const __half* wu, const __half* wd, const __half* token_gate_w,
                           int T, int H, int I, const void* residual, void* y, int y_dtype, float* z, float* gate, cudaStream_t st) {
  if (token_gate_w && x_dtype == BM_F32) return BM_ERR_UNSUPPORTED;     // the gate's logit is taken from the unrounded fp32 row
  // From 17 tokens on a pair whose row tiles are more than a wave of CTAs goes to the tiled product (us, two shared experts of 1408, bf16:
  // 8 tokens 24.2 / 29.8, 16 29.1 / 29.4, 24 32.0 / 27.4, 64 68 / 23.6, 256 244 / 27.5; intermediate size 512: 64 tokens 13.9 / 15.9, 80 21.3 / 15.9).
  if (T > 16 && H % 64 == 0 && I % 64 == 0 && skinny_many_waves((I + 15) / 16, 8, T)) return BM_ERR_UNSUPPORTED;
  if (T > SKINNY_MAX_TOKENS || H % 8 != 0 || I % 8 != 0 || !skinny_fits(H, 0, 8) || !skinny_fits(I, 0, skinny_splits(H, I)))
    return BM_ERR_UNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(wg) | reinterpret_cast<uintptr_t>(wu) | reinterpret_cast<uintptr_t>(wd) |
       reinterpret_cast<uintptr_t>(token_gate_w)) & 15u)
    return BM_ERR_UNSUPPORTED;
  SkinnyArgs a{};
  a.seg[0] = SkSeg{wg, wu, z, I, BM_F32, 0, 0};
  a.seg[1] = SkSeg{token_gate_w, nullptr, gate, 1, BM_F32, 0, 0};
  a.n_seg = token_gate_w ? 2 : 1;
  a.X = x; a.N = T; a.K = H; a.x_dtype = x_dtype;
  a.splits = 8;
  int rc = launch_skinny_nt(a, st);
  if (rc) return rc;
  SkinnyArgs d{};
  d.seg[0] = SkSeg{wd, nullptr, y, H, y_dtype, 0, 0};
  d.n_seg = 1;
  d.X = z; d.N = T; d.K = I; d.x_dtype = BM_F32; d.x_gate = token_gate_w ? gate : nullptr; d.residual = residual; d.overlap = 1;
  d.splits = skinny_splits(H, I);
  return launch_skinny_nt(d, st);
}

// gate[t] = sigmoid(x[t] . w), w fp16 or bf16 rounded to it.  A warp takes two tokens, whose loads share those of w: a pass over x at
// memory speed.  It runs beside the rounding of a block's weights, which it does not read (16384 x 2048 bf16 and 4.2 M weights: 25 -> 20 us, 3 of them from types
// that the compiler knows, so that a lane's loads are in flight together).
template <int DTYPE>
__device__ __forceinline__ float2 row_gate_pair(uint32_t v) {
  if (DTYPE == BM_F16) return __half22float2(*reinterpret_cast<const __half2*>(&v));
  return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}
constexpr int RG_TOKENS = 2;
template <int XD, int WD>
__global__ void __launch_bounds__(256) row_gate_kernel(const void* __restrict__ x, const uint16_t* __restrict__ w, int T, int H, float* __restrict__ gate,
                                                       int beside) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t0 = (blockIdx.x * (blockDim.x >> 5) + warp) * RG_TOKENS;
  grid_launch_dependents();
  if (!beside) grid_wait();
  auto weight = [&](uint32_t v) {
    const float2 f = row_gate_pair<WD>(v);
    return WD == BM_F16 ? f : __half22float2(__floats2half2_rn(f.x, f.y));
  };
  if (XD != BM_F32 && H % 8 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15u) == 0) {
    float acc[RG_TOKENS] = {};
    const uint4* xr[RG_TOKENS];
#pragma unroll
    for (int u = 0; u < RG_TOKENS; ++u) xr[u] = reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(x) + static_cast<int64_t>(min(t0 + u, T - 1)) * H);
    const uint4* wr = reinterpret_cast<const uint4*>(w);
#pragma unroll 4
    for (int i = lane; i < H / 8; i += 32) {
      uint4 xv[RG_TOKENS];
#pragma unroll
      for (int u = 0; u < RG_TOKENS; ++u) xv[u] = __ldg(xr[u] + i);
      const uint4 wv = __ldg(wr + i);
      const uint32_t* wp = reinterpret_cast<const uint32_t*>(&wv);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 wf = weight(wp[j]);
#pragma unroll
        for (int u = 0; u < RG_TOKENS; ++u) {
          const float2 xf = row_gate_pair<XD>(reinterpret_cast<const uint32_t*>(&xv[u])[j]);
          acc[u] = fmaf(xf.x, wf.x, fmaf(xf.y, wf.y, acc[u]));
        }
      }
    }
#pragma unroll
    for (int u = 0; u < RG_TOKENS; ++u) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], o);
      if (lane == 0 && t0 + u < T) gate[t0 + u] = 1.f / (1.f + __expf(-acc[u]));
    }
  } else {
    for (int t = t0; t < min(t0 + RG_TOKENS, T); ++t) {
      float acc = 0.f;
      for (int i = lane; i < H; i += 32) {
        const float wf = WD == BM_F16 ? load_act(w, BM_F16, i) : __half2float(__float2half_rn(load_act(w, BM_BF16, i)));
        acc += load_act(x, XD, static_cast<int64_t>(t) * H + i) * wf;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane == 0) gate[t] = 1.f / (1.f + __expf(-acc));
    }
  }
  if (beside) grid_wait();
}

int launch_row_gate(const void* x, int x_dtype, const uint16_t* w, int w_dtype, int T, int H, float* gate, LaunchAfter after, cudaStream_t st) {
  const int per = 8 * RG_TOKENS;
  const bool wh = w_dtype == BM_F16;
  auto* kernel = x_dtype == BM_F32 ? (wh ? row_gate_kernel<BM_F32, BM_F16> : row_gate_kernel<BM_F32, BM_BF16>)
                 : x_dtype == BM_F16 ? (wh ? row_gate_kernel<BM_F16, BM_F16> : row_gate_kernel<BM_F16, BM_BF16>)
                                     : (wh ? row_gate_kernel<BM_BF16, BM_F16> : row_gate_kernel<BM_BF16, BM_BF16>);
  BM_CUDA(launch_after(after, 1, kernel, dim3((T + per - 1) / per), 256, 0, st, x, w, T, H, gate, after == AFTER_BESIDE));
  BM_LAUNCH_CHECK("row_gate_kernel");
  return BM_OK;
}

// z[t, c] = fp16(silu(g) * u * gate[t]); g, u fp16 [T, I].
__global__ void __launch_bounds__(256) silu_mul_kernel(const __half2* __restrict__ g, const __half2* __restrict__ u,
                                                       const float* __restrict__ gate, int64_t n_pairs, int pairs_per_row,
                                                       __half2* __restrict__ z) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n_pairs; i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const float2 gv = __half22float2(g[i]), uv = __half22float2(u[i]);
    const float s = gate ? gate[i / pairs_per_row] : 1.f;
    z[i] = __floats2half2_rn(__fdividef(gv.x, 1.f + __expf(-gv.x)) * uv.x * s, __fdividef(gv.y, 1.f + __expf(-gv.y)) * uv.y * s);
  }
}

}  // namespace bm

using namespace bm;

extern "C" int bm_gate_logits(const void* x, int x_dtype, const uint16_t* gate_w, int32_t T, int32_t num_routed, int32_t hidden,
                              void* logits, int logits_dtype, void* stream) {
  bm::NvtxRange nvtx_range("bm_gate_logits");
  BM_REQUIRE(T >= 0 && num_routed > 0 && hidden > 0, BM_ERR_INVALID_ARG, "gate_logits: bad sizes");
  BM_REQUIRE(x_dtype >= BM_F16 && x_dtype <= BM_F32 && logits_dtype >= BM_F16 && logits_dtype <= BM_F32, BM_ERR_INVALID_ARG,
             "gate_logits: bad dtype");
  if (T == 0) return BM_OK;
  BM_REQUIRE(x && gate_w && logits, BM_ERR_INVALID_ARG, "gate_logits: null pointer");
  return dense_xwT(x, x_dtype, reinterpret_cast<const __half*>(gate_w), nullptr, logits, nullptr, logits_dtype, nullptr, T, num_routed,
                   hidden, 1, nullptr, AFTER_ALL, SKINNY_MAX_TOKENS, static_cast<cudaStream_t>(stream));
}

extern "C" size_t bm_dense_mlp_workspace_bytes(int32_t T, int32_t intermediate) {
  if (T < 0 || intermediate <= 0) return 0;
  // g, u, z fp16 [T, I] and the per-token gate
  return align_up(static_cast<size_t>(T) * intermediate * 2, 256) * 3 + align_up(static_cast<size_t>(T) * 4, 256);
}

extern "C" int bm_dense_mlp_forward(const void* x, int x_dtype, const uint16_t* w_gate, const uint16_t* w_up, const uint16_t* w_down,
                                    const uint16_t* token_gate_w, int32_t T, int32_t hidden, int32_t intermediate,
                                    const void* residual, void* y, int y_dtype, void* workspace, size_t workspace_bytes, void* stream) {
  bm::NvtxRange nvtx_range("bm_dense_mlp_forward");
  BM_REQUIRE(T >= 0 && hidden > 0 && intermediate > 0 && intermediate % 2 == 0, BM_ERR_INVALID_ARG, "dense_mlp: bad sizes");
  BM_REQUIRE(x_dtype >= BM_F16 && x_dtype <= BM_F32 && y_dtype >= BM_F16 && y_dtype <= BM_F32, BM_ERR_INVALID_ARG, "dense_mlp: bad dtype");
  if (T == 0) return BM_OK;
  BM_REQUIRE(x && w_gate && w_up && w_down && y, BM_ERR_INVALID_ARG, "dense_mlp: null pointer");
  const size_t need = bm_dense_mlp_workspace_bytes(T, intermediate);
  BM_REQUIRE(workspace && workspace_bytes >= need && (reinterpret_cast<uintptr_t>(workspace) & 255u) == 0, BM_ERR_WORKSPACE,
             "dense_mlp: workspace must be 256-byte aligned and hold %zu bytes (%zu given)", need, workspace_bytes);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  const size_t mat = align_up(static_cast<size_t>(T) * intermediate * 2, 256);
  __half* g = reinterpret_cast<__half*>(ws);
  __half* u = reinterpret_cast<__half*>(ws + mat);
  __half* z = reinterpret_cast<__half*>(ws + 2 * mat);
  float* gate = reinterpret_cast<float*>(ws + 3 * mat);
  int rc = dense_mlp_small(x, x_dtype, reinterpret_cast<const __half*>(w_gate), reinterpret_cast<const __half*>(w_up),
                           reinterpret_cast<const __half*>(w_down), reinterpret_cast<const __half*>(token_gate_w), T, hidden, intermediate,
                           residual, y, y_dtype, reinterpret_cast<float*>(ws), gate, st);
  if (rc != BM_ERR_UNSUPPORTED) return rc;
  if (token_gate_w && (rc = launch_row_gate(x, x_dtype, token_gate_w, BM_F16, T, hidden, gate, AFTER_ALL, st))) return rc;
  // gated pair in the epilogue of one launch where tiled copies take the shape
  GemmTmaArgs a{};
  a.X = x; a.x_dtype = x_dtype; a.M = T; a.K = hidden;
  a.seg[0] = GemmSeg{reinterpret_cast<const __half*>(w_gate), reinterpret_cast<const __half*>(w_up), z, intermediate, BM_F16};
  a.n_seg = 1;
  a.row_gate = token_gate_w ? gate : nullptr;
  a.after = token_gate_w ? AFTER_READS : AFTER_ALL;
  rc = launch_gemm_tma(a, st);
  if (rc == BM_OK)      // (behind a tiled pair the tiled product of z is the faster one as well: 33 tokens 26.0 -> 23.4 us a call)
    return dense_xwT(z, BM_F16, reinterpret_cast<const __half*>(w_down), nullptr, y, nullptr, y_dtype, residual, T, hidden, intermediate, 1,
                     nullptr, AFTER_READS, /*skinny_tokens=*/0, st);
  if (rc != BM_ERR_UNSUPPORTED) return rc;
  rc = dense_xwT(x, x_dtype, reinterpret_cast<const __half*>(w_gate), reinterpret_cast<const __half*>(w_up), g, u, BM_F16, nullptr,
                 T, intermediate, hidden, 2, nullptr, AFTER_ALL, SKINNY_MAX_TOKENS, st);
  if (rc) return rc;
  const int64_t pairs = static_cast<int64_t>(T) * intermediate / 2;
  const int blocks = static_cast<int>((pairs + 255) / 256 < 148 * 8 ? (pairs + 255) / 256 : 148 * 8);
  silu_mul_kernel<<<blocks, 256, 0, st>>>(reinterpret_cast<const __half2*>(g), reinterpret_cast<const __half2*>(u),
                                          token_gate_w ? gate : nullptr, pairs, intermediate / 2, reinterpret_cast<__half2*>(z));
  BM_LAUNCH_CHECK("silu_mul_kernel");
  return dense_xwT(z, BM_F16, reinterpret_cast<const __half*>(w_down), nullptr, y, nullptr, y_dtype, residual, T, hidden, intermediate, 1,
                   nullptr, AFTER_ALL, SKINNY_MAX_TOKENS, st);
}
