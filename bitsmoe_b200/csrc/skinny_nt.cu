// Products of a decode batch with streamed weights:  C[n][m] = sum_k W[m][k] * X[n][k], up to 256 tokens.
//   logits / h_gate / h_up / shared-expert gate and up = x . W^T   (stacks of output rows sharing x, K = hidden)
//   y = fp16(rank_accum) . U_down^T (+ shared down product) (+ residual)
// These are weight-streaming GEMVs: a CTA reads a [rows x k-slice] block of W once, keeps it in shared memory and
// multiplies it with 64 token rows on the tensor cores (mma.sync m16n8k16, W rows as the A operand, tokens as N).
// A long contraction is split over the CTAs of a thread-block cluster whose partial sums meet through distributed shared
// memory: no atomics, no second pass.  More tokens than 64 are more CTAs (grid y), not a loop: the weights come from L2
// then, and the chunks run side by side.
//
// What bounds a launch is latency: weights -> shared memory -> MMA -> cluster exchange.  Three things shorten the chain:
// everything that multiplies the same x is one launch (SkSeg stacks; the gated pair of a shared expert leaves as
// silu(g) * u), the routing of given logits is one more cluster of the same grid, and a launch behind
// another one of the same call is programmatically serialised: its weights are on their way to shared memory while the
// previous kernel still runs.  A whole block of one token went from 60.6 us a call (seven launches and the host work between
// them) to 25.5, 24 tokens of a 512-expert block with a gated shared expert from 130 to 53.
#include <algorithm>

#include "route_small.cuh"

namespace cg = cooperative_groups;

namespace bm {

constexpr int SK_THREADS = 256;
constexpr int SK_NTOK = 64;          // tokens per CTA
constexpr int SK_RECV = 72;          // floats per received row: four neighbouring rows start eight banks apart

__host__ __device__ constexpr int sk_mrows(int splits) { return splits == 1 ? 16 : 32; }

__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void ldsm_x4(const __half* p, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))));
}

__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// Columns [k0, k0 + width) of the rows n0 .. n0 + nn of a row-major [*, ld] matrix -> fp16 at dst (row stride `stride`),
// rows up to `rows` zero; the loads of eight 8-element vectors are issued before the first conversion.
template <int XD>
__device__ __forceinline__ void stage_rows(const void* X, int64_t ld, int k0, int width, int n0, int nn, int rows, const float* gate,
                                           __half* dst, int stride) {
  const int vpr = width >> 3, nvec = rows * vpr;
  constexpr int U = XD == BM_F32 ? 4 : 8;
  for (int v0 = threadIdx.x; v0 < nvec; v0 += U * SK_THREADS) {
    uint4 raw[U][XD == BM_F32 ? 2 : 1];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int v = v0 + u * SK_THREADS;
      const int r = v / vpr, c = (v - r * vpr) * 8;
      raw[u][0] = make_uint4(0u, 0u, 0u, 0u);
      if (XD == BM_F32) raw[u][XD == BM_F32 ? 1 : 0] = make_uint4(0u, 0u, 0u, 0u);
      if (v < nvec && r < nn) {
        const int64_t idx = static_cast<int64_t>(n0 + r) * ld + k0 + c;
        if (XD == BM_F32) {
          const uint4* src = reinterpret_cast<const uint4*>(static_cast<const float*>(X) + idx);
          raw[u][0] = src[0];
          raw[u][XD == BM_F32 ? 1 : 0] = src[1];
        } else {
          raw[u][0] = *reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(X) + idx);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int v = v0 + u * SK_THREADS;
      if (v >= nvec) break;
      const int r = v / vpr, c = (v - r * vpr) * 8;
      uint4 out = raw[u][0];
      if (XD == BM_BF16) {
        uint32_t* o = reinterpret_cast<uint32_t*>(&out);
#pragma unroll
        for (int i = 0; i < 4; ++i) o[i] = pack_half2(__uint_as_float(o[i] << 16), __uint_as_float(o[i] & 0xffff0000u));
      } else if (XD == BM_F32) {
        const float* f0 = reinterpret_cast<const float*>(&raw[u][0]);
        const float* f1 = reinterpret_cast<const float*>(&raw[u][XD == BM_F32 ? 1 : 0]);
        const float s = gate && r < nn ? 1.f / (1.f + __expf(-gate[n0 + r])) : 1.f;
        out = make_uint4(pack_half2(f0[0] * s, f0[1] * s), pack_half2(f0[2] * s, f0[3] * s), pack_half2(f1[0] * s, f1[1] * s),
                         pack_half2(f1[2] * s, f1[3] * s));
      }
      *reinterpret_cast<uint4*>(dst + static_cast<size_t>(r) * stride + c) = out;
    }
  }
}

// smem: Ws [bufs][mrows][kw + 8] half | Xs [xrows][kw + 8] half | recv [bufs][splits][mrows / splits][72] float (only when
// splits > 1), kw = K / splits + K2, bufs = 2 when a CTA takes more than one row tile
__host__ __device__ inline int sk_xrows(int N) { return N >= SK_NTOK ? SK_NTOK : (N + 7) & ~7; }
__host__ __device__ inline size_t sk_smem_bytes(int K, int K2, int splits, int N, int bufs) {
  const int mrows = sk_mrows(splits);
  size_t s = static_cast<size_t>(bufs * mrows + sk_xrows(N)) * (K / splits + K2 + 8) * 2;
  if (splits > 1) s += static_cast<size_t>(bufs) * mrows * SK_RECV * 4;
  return s;
}
constexpr size_t SK_SMEM_LIMIT = 160 * 1024;
// CTAs per SM that the registers of a thread allow: the fourth costs a few instructions (one token: 1 us a block), so it is
// taken where it saves a second wave (24 tokens of a 512-expert block: 59 -> 53 us) or a loop wants the warps.
constexpr int SK_FEW = 3, SK_MANY = 4;

template <bool LOOP, int CTAS>
__global__ void __launch_bounds__(SK_THREADS, CTAS) skinny_nt_kernel(const __grid_constant__ SkinnyArgs a) {
  extern __shared__ __align__(16) unsigned char sk_smem[];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int split = blockIdx.x % a.splits, cluster_id = blockIdx.x / a.splits;
  if (cluster_id >= a.clusters) {      // the routing cluster
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (blockIdx.y == 0) route_small(a.route, reinterpret_cast<RouteSmallSmem*>(sk_smem));
    return;
  }
  const int ks = a.K / a.splits, kw = ks + a.K2;
  const int stride = kw + 8;
  const int mrows = sk_mrows(a.splits);
  constexpr int bufs = LOOP ? 2 : 1;      // more row tiles than clusters
  __half* const Ws0 = reinterpret_cast<__half*>(sk_smem);
  __half* const Xs = Ws0 + static_cast<size_t>(bufs * mrows) * stride;
  float* const recv0 = reinterpret_cast<float*>(Xs + static_cast<size_t>(sk_xrows(a.N)) * stride);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;

  // peers' shared memory may be written only once every CTA of the cluster runs: arrive now, wait before the first push
  cg::cluster_group::arrival_token started;
  if (a.splits > 1) started = cg::this_cluster().barrier_arrive();
  const int n0 = blockIdx.y * SK_NTOK;
  const int nn = min(SK_NTOK, a.N - n0);
  const int nblocks = (nn + 7) >> 3;
  // (mblock, nblock) items round-robin over the warps, two at a time: items `it` and `it + 8` share the W rows when
  // mblocks divides the warp count, so one A fragment feeds two MMAs; a lone item splits its contraction over two
  // accumulators instead.  Fragments come from ldmatrix (rows are 16-byte aligned and 16 bytes apart modulo 128).
  const int mblocks = mrows / 16;
  const int n_items = mblocks * nblocks;
  const int a_row = (lane & 7) + 8 * ((lane >> 3) & 1), a_kofs = 8 * (lane >> 4);   // ldmatrix.x4 address roles, A operand
  const int b_row = lane & 7, b_sel = lane >> 3;                                     // B operand: matrix b_sel of four
  // A cluster takes row tiles `a.clusters` apart; the next tile's weights travel while this one is multiplied.  One cluster
  // barrier per tile: when it opens, everybody has summed the tile before, whose receive buffer the next one uses again.
#pragma unroll(LOOP ? 1 : 2)
  for (int turn = 0; LOOP || turn < 2; ++turn) {
    // ---- W block of tile `turn` -> smem.  A gated pair alternates gate and up rows, so that one CTA of the cluster owns
    // both sums of an output.
    const int load_tile = cluster_id + turn * a.clusters;
    if (LOOP ? load_tile < a.row_tiles : turn == 0) {
      __half* Ws = Ws0 + static_cast<size_t>(turn & (bufs - 1)) * mrows * stride;
      int si = 0;
      while (si + 1 < a.n_seg && load_tile >= a.seg[si + 1].tile0) ++si;
      const SkSeg& sg = a.seg[si];
      const bool glu = sg.W_up != nullptr;
      const int m0 = (load_tile - sg.tile0) * (glu ? mrows / 2 : mrows);
      const int vpr = kw >> 3;
      for (int v = threadIdx.x; v < mrows * vpr; v += SK_THREADS) {
        const int r = v / vpr, c = (v - r * vpr) * 8;
        const int m = m0 + (glu ? r >> 1 : r);
        __half* dst = Ws + static_cast<size_t>(r) * stride + c;
        const bool live = m < sg.rows;
        const __half* src = c < ks ? (glu && (r & 1) ? sg.W_up : sg.W) + static_cast<size_t>(live ? m : 0) * a.K + split * ks + c
                                   : a.W2 + static_cast<size_t>(live ? m : 0) * a.K2 + (c - ks);
        if (c < ks ? sg.w_bf16 : a.w2_bf16) {
          uint4 raw = live ? __ldg(reinterpret_cast<const uint4*>(src)) : make_uint4(0u, 0u, 0u, 0u);
          uint32_t* o = reinterpret_cast<uint32_t*>(&raw);
#pragma unroll
          for (int i = 0; i < 4; ++i) o[i] = pack_half2(__uint_as_float(o[i] << 16), __uint_as_float(o[i] & 0xffff0000u));
          *reinterpret_cast<uint4*>(dst) = raw;
        } else {
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src),
                       "r"(live ? 16 : 0)
                       : "memory");
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (turn == 0) {
      asm volatile("griddepcontrol.wait;" ::: "memory");
      if (a.zero != nullptr) {
        const int ctas = a.clusters * a.splits;      // without the routing cluster's
        for (int i = (blockIdx.y * ctas + blockIdx.x) * SK_THREADS + threadIdx.x; i < a.zero_n; i += ctas * gridDim.y * SK_THREADS)
          a.zero[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
      if (a.x_dtype == BM_F32) stage_rows<BM_F32>(a.X, a.K, split * ks, ks, n0, nn, nblocks * 8, a.x_gate, Xs, stride);
      else if (a.x_dtype == BM_BF16) stage_rows<BM_BF16>(a.X, a.K, split * ks, ks, n0, nn, nblocks * 8, nullptr, Xs, stride);
      else stage_rows<BM_F16>(a.X, a.K, split * ks, ks, n0, nn, nblocks * 8, nullptr, Xs, stride);
      if (a.K2) stage_rows<BM_F32>(a.X2, a.K2, 0, a.K2, n0, nn, nblocks * 8, a.x2_gate, Xs + ks, stride);
      if (a.splits > 1) cg::this_cluster().barrier_wait(std::move(started));
      continue;
    }
    // ---- products of tile turn - 1
    asm volatile("cp.async.wait_group %0;" ::"n"(LOOP ? 1 : 0) : "memory");
    __syncthreads();
    const int row_tile = load_tile - a.clusters;
    const __half* Ws = Ws0 + static_cast<size_t>((turn - 1) & (bufs - 1)) * mrows * stride;
    float* recv = recv0 + static_cast<size_t>((turn - 1) & (bufs - 1)) * mrows * SK_RECV;
    int si = 0;
    while (si + 1 < a.n_seg && row_tile >= a.seg[si + 1].tile0) ++si;
    const SkSeg& sg = a.seg[si];
    const bool glu = sg.W_up != nullptr;
    const int m0 = (row_tile - sg.tile0) * (glu ? mrows / 2 : mrows);      // first output row of the stack in this CTA
    for (int it = warp; it < n_items; it += 2 * (SK_THREADS / 32)) {
      const int it2 = it + SK_THREADS / 32;
      const int mb = it % mblocks, nb = it / mblocks;
      const bool pair = it2 < n_items && (it2 % mblocks) == mb;
      const int nb2 = pair ? it2 / mblocks : nb;
      float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
      const __half* wa = Ws + static_cast<size_t>(mb * 16 + a_row) * stride + a_kofs;
      if (pair) {
        // B matrices: (nb, k 0-7) (nb, k 8-15) (nb2, k 0-7) (nb2, k 8-15)
        const __half* xb = Xs + static_cast<size_t>((b_sel < 2 ? nb : nb2) * 8 + b_row) * stride + 8 * (b_sel & 1);
#pragma unroll 4
        for (int k = 0; k < kw; k += 16) {
          uint32_t a0, a1, a2, a3, b0, b1, c0, c1;
          ldsm_x4(wa + k, a0, a1, a2, a3);
          ldsm_x4(xb + k, b0, b1, c0, c1);
          mma16816(acc[0], a0, a1, a2, a3, b0, b1);
          mma16816(acc[1], a0, a1, a2, a3, c0, c1);
        }
      } else {
        // B matrices: (nb, k 0-7) (nb, k 8-15) (nb, k 16-23) (nb, k 24-31); even / odd 16-steps in separate accumulators
        const __half* xb = Xs + static_cast<size_t>(nb * 8 + b_row) * stride + 8 * b_sel;
        int k = 0;
#pragma unroll 4
        for (; k + 32 <= kw; k += 32) {
          uint32_t a0, a1, a2, a3, e0, e1, e2, e3, b0, b1, c0, c1;
          ldsm_x4(wa + k, a0, a1, a2, a3);
          ldsm_x4(wa + k + 16, e0, e1, e2, e3);
          ldsm_x4(xb + k, b0, b1, c0, c1);
          mma16816(acc[0], a0, a1, a2, a3, b0, b1);
          mma16816(acc[1], e0, e1, e2, e3, c0, c1);
        }
        if (k < kw) {   // one 16-step left: the upper two B matrices repeat the lower ones instead of reading past the row
          uint32_t a0, a1, a2, a3, b0, b1, c0, c1;
          ldsm_x4(wa + k, a0, a1, a2, a3);
          ldsm_x4(Xs + static_cast<size_t>(nb * 8 + b_row) * stride + 8 * (b_sel & 1) + k, b0, b1, c0, c1);
          mma16816(acc[0], a0, a1, a2, a3, b0, b1);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) { acc[0][j] += acc[1][j]; acc[1][j] = 0.f; }
      }
      // D: rows m = mb*16 + g (+8), cols n = nb*8 + 2t (+1)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        if (q == 1 && !pair) break;
        const int nbq = q ? nb2 : nb;
        if (a.splits == 1) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int m = m0 + mb * 16 + g + (j >= 2 ? 8 : 0), n = nbq * 8 + 2 * t + (j & 1);
            if (n < nn && m < sg.rows) {
              const int64_t idx = static_cast<int64_t>(n0 + n) * sg.rows + m;
              float v = acc[q][j];
              if (a.residual && si == 0) v += load_act(a.residual, sg.c_dtype, idx);
              store_act(sg.C, sg.c_dtype, idx, v);
            }
          }
        } else {
          // push the partial sums into the shared memory of the CTA that owns these output rows
          const int rows_per_owner = mrows / a.splits;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int m = mb * 16 + g + 8 * h;
            float* dst = cg::this_cluster().map_shared_rank(recv, m / rows_per_owner) +
                         (static_cast<size_t>(split) * rows_per_owner + m % rows_per_owner) * SK_RECV + nbq * 8 + 2 * t;
            *reinterpret_cast<float2*>(dst) = make_float2(acc[q][2 * h], acc[q][2 * h + 1]);
          }
        }
      }
    }
    if (a.splits > 1) {
      cg::this_cluster().sync();   // every CTA's partial sums have landed in their owners
      // this CTA owns rows [split * rows_per_owner, +rows_per_owner) of the mrows x nn tile: sum the `splits` copies
      const int rows_per_owner = mrows / a.splits, outs = glu ? rows_per_owner / 2 : rows_per_owner;
      auto total = [&](int r, int n) {
        float pv[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) pv[c] = c < a.splits ? recv[(static_cast<size_t>(c) * rows_per_owner + r) * SK_RECV + n] : 0.f;
        return ((pv[0] + pv[1]) + (pv[2] + pv[3])) + ((pv[4] + pv[5]) + (pv[6] + pv[7]));
      };
      // consecutive threads take consecutive rows of a token: an owner's rows are one short piece of the output row
      for (int o = threadIdx.x; o < outs * nn; o += SK_THREADS) {
        const int n = o / outs, r = o - n * outs;
        const int m = m0 + split * outs + r;
        if (m >= sg.rows) continue;
        float v;
        if (glu) {
          const float gv = total(2 * r, n), uv = total(2 * r + 1, n);
          v = __fdividef(gv, 1.f + __expf(-gv)) * uv;
        } else {
          v = total(r, n);
        }
        const int64_t idx = static_cast<int64_t>(n0 + n) * sg.rows + m;
        if (a.residual && si == 0) v += load_act(a.residual, sg.c_dtype, idx);
        store_act(sg.C, sg.c_dtype, idx, v);
      }
    }
    if (!LOOP || load_tile >= a.row_tiles) break;
    if (a.splits == 1) __syncthreads();      // (a cluster's barrier stands between the products and the next copy)
  }
}

bool skinny_fits(int K, int K2, int splits) {
  return K % (16 * splits) == 0 && K2 % 16 == 0 && (K2 == 0 || splits == 1) && sk_smem_bytes(K, K2, splits, SKINNY_MAX_TOKENS, 1) <= SK_SMEM_LIMIT;
}

// The fewest splits whose k-slice fits shared memory and whose grid reaches most SMs.
int skinny_splits(int rows, int K) {
  for (int s = 1; s < 8; s *= 2)
    if (skinny_fits(K, 0, s) && ((rows + sk_mrows(s) - 1) / sk_mrows(s) * s >= 96 || K / s <= 256)) return s;
  return 8;
}

bool skinny_many_waves(int row_tiles, int splits, int T) {
  int dev = -1, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return false;
  return row_tiles * splits * ((T + SK_NTOK - 1) / SK_NTOK) > SK_FEW * sms;
}

int launch_skinny_nt(SkinnyArgs a, cudaStream_t st) {
  BM_REQUIRE(a.N >= 1 && a.N <= SKINNY_MAX_TOKENS && a.n_seg >= 1 && a.n_seg <= SK_MAX_SEG && a.splits >= 1 && a.splits <= 8 &&
                 (a.splits & (a.splits - 1)) == 0 && skinny_fits(a.K, a.K2, a.splits) && aligned16(a.X, a.W2, a.X2),
             BM_ERR_UNSUPPORTED, "skinny_nt: shape does not tile");
  const int mrows = sk_mrows(a.splits);
  a.row_tiles = 0;
  for (int i = 0; i < a.n_seg; ++i) {
    const bool glu = a.seg[i].W_up != nullptr;
    BM_REQUIRE(((reinterpret_cast<uintptr_t>(a.seg[i].W) | reinterpret_cast<uintptr_t>(a.seg[i].W_up)) & 15u) == 0 && (!glu || a.splits > 1) &&
                   (!glu || mrows / a.splits % 2 == 0),
               BM_ERR_UNSUPPORTED, "skinny_nt: weights are not aligned");
    a.seg[i].tile0 = a.row_tiles;
    const int per = glu ? mrows / 2 : mrows;
    a.row_tiles += (a.seg[i].rows + per - 1) / per;
  }
  static PerDeviceOnce attr_once;
  static int sm_counts[MAX_DEVICES];
  int dev = -1;
  BM_CUDA(cudaGetDevice(&dev));
  BM_REQUIRE(dev >= 0 && dev < MAX_DEVICES, BM_ERR_UNSUPPORTED, "skinny_nt: device ordinal %d out of range", dev);
  if (!attr_once.is_done(dev)) {
    for (auto* kernel : {skinny_nt_kernel<false, SK_FEW>, skinny_nt_kernel<false, SK_MANY>, skinny_nt_kernel<true, SK_MANY>})
      BM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(SK_SMEM_LIMIT)));
    BM_CUDA(cudaDeviceGetAttribute(&sm_counts[dev], cudaDevAttrMultiProcessorCount, dev));
    attr_once.mark(dev);
  }
  const bool route = a.route.T > 0;
  // One cluster per row tile while the device holds them all at once; more row tiles than that are a loop, which has the
  // next tile's weights in flight where a second wave would start from nothing (5 tokens, two shared experts of 1408: 59 -> 52
  // us a call).
  const int chunks = (a.N + SK_NTOK - 1) / SK_NTOK;
  const int sms = sm_counts[dev];
  auto resident = [sms](size_t bytes, int most) { return sms * std::min(static_cast<int>(227 * 1024 / (bytes + 1024)), most); };
  size_t smem = sk_smem_bytes(a.K, a.K2, a.splits, a.N, 1);
  a.clusters = a.row_tiles;
  const int total = (a.row_tiles + (route ? 1 : 0)) * a.splits * chunks;
  const bool few = total <= resident(smem, SK_FEW);
  if (total > resident(smem, SK_MANY)) {
    const size_t two = sk_smem_bytes(a.K, a.K2, a.splits, a.N, 2);
    const int fit = two <= SK_SMEM_LIMIT ? resident(two, SK_MANY) / (a.splits * chunks) : 0;
    if (fit >= 1 && fit < a.row_tiles) {
      const int turns = (a.row_tiles + fit - 1) / fit;
      a.clusters = (a.row_tiles + turns - 1) / turns;      // the same number of turns for everybody
      smem = two;
    }
  }
  if (a.clusters == a.row_tiles) {
    // small CTAs are placed several to an SM while other SMs stay empty: ask for the memory that spreads them evenly, with
    // a tenth to spare for clusters that do not fill their group of SMs (64 tokens: 47.2 -> 44.3 us a block)
    int per_sm = (total * 11 + 10 * sms - 1) / (10 * sms);
    // one CTA an SM leaves clusters without a whole group of SMs, and the last ones wait for a second wave (basis pair of 64 tokens, 16
    // clusters of eight: 11.4 -> 7.5 us, of one token 8.3 -> 5.1)
    if (a.splits > 1 && per_sm == 1 && total * 5 > sms * 4) per_sm = 2;
    const size_t room = (227 * 1024 / std::min(per_sm, 8) - 1024) / 128 * 128;
    smem = std::max(smem, std::min(room, SK_SMEM_LIMIT));
  }
  BM_REQUIRE(!route || a.splits == RS_CLUSTER, BM_ERR_UNSUPPORTED, "skinny_nt: routing needs clusters of %d", RS_CLUSTER);
  if (route && smem < sizeof(RouteSmallSmem)) smem = sizeof(RouteSmallSmem);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((a.clusters + (route ? 1 : 0)) * a.splits, chunks);
  cfg.blockDim = dim3(SK_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  if (a.overlap) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (a.splits > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = a.splits;
    attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs++].val.clusterDim.z = 1;
  }
  count_launch();
  BM_CUDA(cudaLaunchKernelEx(&cfg, a.clusters < a.row_tiles ? skinny_nt_kernel<true, SK_MANY> : few ? skinny_nt_kernel<false, SK_FEW> : skinny_nt_kernel<false, SK_MANY>, a));
  return BM_OK;
}

// ---- routing on its own, behind the launch that computes the logits
template <int CL, int THREADS>
__global__ void __launch_bounds__(THREADS) route_small_kernel(const __grid_constant__ RouteSmallArgs a) {
  __shared__ RouteSmallSmem sm;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  route_small<CL, THREADS>(a, &sm);
}

bool route_small_fits(int T, int E, int k) { return T >= 1 && T <= RS_MAX_TOKENS && E >= 1 && E <= RS_MAX_E && k >= 1 && k <= 32 && k <= E; }

int launch_route_small(const RouteSmallArgs& a, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  const bool one = a.T <= RS_ONE_TOKENS;
  cfg.gridDim = dim3(one ? 1 : RS_CLUSTER);
  cfg.blockDim = dim3(one ? RS_ONE_THREADS : RS_THREADS);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = RS_CLUSTER;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = one ? 1 : 2;
  count_launch();
  BM_CUDA(cudaLaunchKernelEx(&cfg, one ? route_small_kernel<1, RS_ONE_THREADS> : route_small_kernel<RS_CLUSTER, RS_THREADS>, a));
  return BM_OK;
}

}  // namespace bm
