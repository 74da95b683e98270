// Dense products for large token counts, warp-specialised: tiled TMA loads, tcgen05.mma, persistent CTAs.
//   C_i[m][n] = sum_k X[m][k] * W_i[n][k],  X = activations (rows = tokens), W_i = fp16 matrices ("stacks") sharing X
//   router logits, h_gate / h_up = x . Vh^T, z = silu(x . Wg^T) * (x . Wu^T) of a shared expert: one launch
//   (bitsmoe/models/qwen3moe/bitsmoe_block.py:45, :63-64)
//   y = fp16(rank_accum) . U_down^T (+ z . W_down^T) (+ residual)   (bitsmoe/models/base_block.py:414)
// A CTA walks 128 x BN output tiles (BN = 256, or 128 or 64 when the wide tile would leave most SMs idle; a few narrow tiles
// split K over a cluster of two or four CTAs, whose sums meet in distributed shared memory).  Per tile, K is streamed in slices of 64 through a ring of stages, both operands K-major with the 128-byte swizzle that the tensor
// map writes and the MMA descriptor reads:
//   warp 0      producer: cp.async.bulk.tensor (2-D tiles) of the X slice and of two half tiles of W rows -- neighbouring
//               rows of a stack, or the same rows of a gated pair -- completing on the stage's mbarrier
//   warp 1      MMA issue: four tcgen05.mma (M = 128, N = BN, K = 16) per slice, tcgen05.commit frees the stage; the
//               accumulator alternates between two TMEM buffers, so the next tile's products run while this tile's
//               accumulator is read out
//   warps 4-11  epilogue: tcgen05.ld, residual / gated pair, rounding, and 32 x 32 blocks through shared memory into TMA
//               stores (a lane owns an output row; its own stores would touch 32 rows per instruction)
//   warps 12-15, 2, 3, and the epilogue warps before the end of a CTA's only tile: only for bf16 / fp32 activations: round the landed X slice to fp16 in place (both MMA operands have to
//               be fp16: a bf16 A with an fp16 B is not an encodable instruction).  bf16 -> fp16 is element for
//               element; an fp32 slice is twice as large as its fp16 result, and the eight lanes that hold a row read
//               the row's 256 bytes before any of them writes its 16-byte piece of the 128-byte result row.
// Every wait is bounded; a time-out raises the status word.
//
// Small batches of bf16 or fp32 rows are bound by the rounding: 550 to 600 cycles a slice of 128 rows, whatever the tile's width and
// however many warps share it; fp16 slices take 350, the rate at which an SM gets data from L2.  Measured and not taken: the rounded
// slice into tensor memory instead of shared memory (basis pair of 777 tokens 11.8 -> 11.6 us, 8192 tokens 22.1 -> 21.3, but 2048
// tokens 14.0 -> 15.2), conversion by integer shifts (777 tokens 12.9).  Basis
// pair of 300 tokens 14.9 -> 9.3 us (clusters of four), 777 tokens 15.2 -> 11.8 (of two), 2048 tokens 15.7 -> 14.0 (epilogue warps
// round too).
//
// Large ones are bound by the tensor pipe at its sustained clock.  16384 tokens, hidden 2048: router of 512 experts, basis pair
// 2 x 256 and gated pair 2 x 512 with silu as one launch 119 us (1.15 PFLOP/s; as three launches and a pass over z 192), down basis
// and shared down product 109 -> 59 us; 8192 tokens: basis pair 25 -> 23 us, down basis 30 -> 20 (TMA stores).
#include <cuda.h>

#include <cstring>
#include <utility>

#include "common.cuh"
#include "tc05.cuh"

namespace bm {

constexpr int GT_BM = 128, GT_BK = 64, GT_THREADS = 512, GT_MAX_STAGES = 8;
constexpr int GT_WARP_EPI0 = 4, GT_EPI_WARPS = 8, GT_WARP_TR0 = 12, GT_TR_WARPS = 6;    // transform: warps 12-15 and 2, 3
constexpr int GT_STORE_BYTES = 32 * 64;                       // one 32 x 32 block of 16-bit results
constexpr int GT_SMEM = 225 * 1024;                           // stages and store blocks

__host__ __device__ constexpr int gt_a_bytes(int xd) { return xd == BM_F32 ? GT_BM * GT_BK * 4 : GT_BM * GT_BK * 2; }
__host__ __device__ constexpr int gt_stage_bytes(int bn, int xd) { return gt_a_bytes(xd) + bn * GT_BK * 2; }
// Split contraction: floats between the rows that a CTA receives from one CTA of its cluster (bn / split columns, padded), and
// what is behind the stages: blocks on their way out, or the received sums.
__host__ __device__ constexpr int gt_recv_row(int bn, int split) { return bn / split + 4; }
__host__ __device__ constexpr int gt_tail_bytes(int bn, int split) {
  return split > 1 ? split * GT_BM * gt_recv_row(bn, split) * 4 : GT_EPI_WARPS * 2 * GT_STORE_BYTES;
}
// Ring depth; with rounding a multiple of the number of warp groups that round (2 or 3), see below.
__host__ __device__ constexpr int gt_stages(int bn, int xd, int split) {
  const int room = (GT_SMEM - gt_tail_bytes(bn, split)) / gt_stage_bytes(bn, xd);
  const int fit = room < GT_MAX_STAGES ? room : GT_MAX_STAGES;
  return xd == BM_F16 || fit % 3 == 0 ? fit : fit / 2 * 2;
}
__host__ __device__ constexpr int gt_tr_groups(int bn, int xd, int split) { return gt_stages(bn, xd, split) % 3 == 0 ? 3 : 2; }
// where the epilogue warps round too: 3, 4 or 2 groups of 4, 3 or 7 of the 14 warps
__host__ __device__ constexpr int gt_tr_groups_all(int bn, int xd, int split) {
  return gt_stages(bn, xd, split) % 3 == 0 ? 3 : gt_stages(bn, xd, split) % 4 == 0 ? 4 : 2;
}

struct GtSeg {
  void* C;
  int rows, c_dtype, glu, tile0, map_w, map_up;       // glu: W_up at map_up pairs with W
};
struct GtParams {
  CUtensorMap x, x2, w[GEMM_MAX_SEG + 2], w2, c[GEMM_MAX_SEG];
  GtSeg seg[GEMM_MAX_SEG];
  const void* residual;      // of stack 0
  const float* row_gate;     // factor per row of a gated pair's result, or null
  int n_seg, M, slices, slices2, tiles_n, ntiles, tma_store, beside;
  int* status;
  float4* zero;              // cleared by the epilogue warps
  int64_t zero_n;
};

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                   tc::smem_u32(dst)),
               "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(tc::smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, int x, int y, const void* src) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(reinterpret_cast<uint64_t>(map)), "r"(x),
               "r"(y), "r"(tc::smem_u32(src))
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// K-major operand tile of 128-byte rows, 8-row groups 1024 bytes apart, 128-byte swizzle
__device__ __forceinline__ uint64_t gt_desc_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>(1) << 16;              // leading byte offset: unused with swizzled K-major tiles
  d |= static_cast<uint64_t>(1024 >> 4) << 32;      // stride between 8-row groups
  d |= 1ull << 46;                                  // descriptor version of this architecture
  d |= 2ull << 61;                                  // 128-byte swizzle
  return d;
}

__device__ __forceinline__ uint32_t pack16(float a, float b, int dtype) {
  if (dtype == BM_F16) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// What output tile `tile` is: its row block, its stack and the first output row (of W) inside the stack.
struct GtTile {
  int m0, si, n0;
  bool two;                  // both halves of the tile hold W rows
};
template <int BN>
__device__ __forceinline__ GtTile gt_tile(const GtParams& p, int tile) {
  GtTile t;
  const int m_t = tile / p.tiles_n, r = tile - m_t * p.tiles_n;
  t.m0 = m_t * GT_BM;
  t.si = 0;
  while (t.si + 1 < p.n_seg && r >= p.seg[t.si + 1].tile0) ++t.si;
  const GtSeg& s = p.seg[t.si];
  t.n0 = (r - s.tile0) * (s.glu ? BN / 2 : BN);
  t.two = s.glu || t.n0 + BN / 2 < s.rows;
  return t;
}

// SPLIT > 1: a cluster of SPLIT CTAs per tile, each of which takes its share of the slices; the sums meet in shared memory, where
// a CTA owns BN / 2 / SPLIT columns of either half of the tile.
template <int BN, int XD, int SPLIT>
__global__ void __launch_bounds__(GT_THREADS, 1) gemm_tma_kernel(const __grid_constant__ GtParams p) {
  constexpr int A_BYTES = gt_a_bytes(XD), A2_BYTES = GT_BM * GT_BK * 2, H_BYTES = BN / 2 * GT_BK * 2, STAGE = A_BYTES + 2 * H_BYTES,
                NST = gt_stages(BN, XD, SPLIT);
  constexpr int TR_GROUPS = gt_tr_groups(BN, XD, SPLIT), TR_GROUPS_ALL = gt_tr_groups_all(BN, XD, SPLIT);
  // one tile per CTA: the epilogue warps have nothing to do before its end, and round slices until then
  const bool all_round = static_cast<int>(gridDim.x) >= p.ntiles * SPLIT;
  const int tr_groups = all_round ? TR_GROUPS_ALL : TR_GROUPS;
  const int tr_per = all_round ? (GT_TR_WARPS + GT_EPI_WARPS) / TR_GROUPS_ALL : GT_TR_WARPS / TR_GROUPS;
  constexpr uint32_t TMEM_COLS = 2 * BN < 32 ? 32 : 2 * BN;
  extern __shared__ unsigned char gt_raw[];
  __shared__ __align__(8) uint64_t loaded[GT_MAX_STAGES], ready[GT_MAX_STAGES], empty[GT_MAX_STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_slot;
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(gt_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int warp = tc::warp_index(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < GT_MAX_STAGES; ++i) {
      tc::mbar_init(&loaded[i], 1);
      tc::mbar_init(&ready[i], tr_per);
      tc::mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&acc_full[i], 1);
      tc::mbar_init(&acc_empty[i], GT_EPI_WARPS);
    }
    tc::mbar_init_fence();
  }
  if (warp == 2) tc::tmem_alloc(&tmem_slot, TMEM_COLS);
  if (SPLIT > 1) tc::cluster_arrive();           // waited for before anything is sent to another CTA
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem_base = tmem_slot;
  grid_launch_dependents();
  if (!p.beside) grid_wait();
  // slices of X . W, then of the second contraction: this CTA's share
  const int all = p.slices + p.slices2, rank = SPLIT > 1 ? static_cast<int>(blockIdx.x) % SPLIT : 0;
  const int s_first = all * rank / SPLIT, s_end = all * (rank + 1) / SPLIT, slices = s_end - s_first;
  const int cta = static_cast<int>(blockIdx.x) / SPLIT, grid = static_cast<int>(gridDim.x) / SPLIT;
  bool ok = true;

  if (warp == 0) {
    // ------------------------------------------------------------------ producer (the whole warp waits, one lane issues)
    uint32_t st = 0, ph = 0;
    for (int tile = cta; tile < p.ntiles && ok; tile += grid) {
      const GtTile t = gt_tile<BN>(p, tile);
      const GtSeg& sg = p.seg[t.si];
      const CUtensorMap *mw = &p.w[sg.map_w], *mu = sg.glu ? &p.w[sg.map_up] : mw;
      const int nu = sg.glu ? t.n0 : t.n0 + BN / 2;
      for (int s = s_first; s < s_end; ++s) {
        if (!(ok = tc::mbar_wait(&empty[st], ph ^ 1))) break;
        if (tc::elect_one()) {
          unsigned char* sa = smem + st * STAGE;
          const bool first = s < p.slices;
          const int k = (first ? s : s - p.slices) * GT_BK;
          tc::mbar_expect_tx(&loaded[st], (first ? A_BYTES : A2_BYTES) + (t.two ? 2 : 1) * H_BYTES);
          tma_load_2d(sa, first ? &p.x : &p.x2, k, t.m0, &loaded[st]);
          if (XD == BM_F32 && first) tma_load_2d(sa + A_BYTES / 2, &p.x, k + 32, t.m0, &loaded[st]);   // an fp32 row of 64 values is two 128-byte boxes
          tma_load_2d(sa + A_BYTES, first ? mw : &p.w2, k, t.n0, &loaded[st]);
          if (t.two) tma_load_2d(sa + A_BYTES + H_BYTES, first ? mu : &p.w2, k, nu, &loaded[st]);
        }
        __syncwarp();
        if (++st == NST) { st = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issue (the whole warp waits, one issues)
    uint32_t st = 0, ph = 0, ti = 0;
    for (int tile = cta; tile < p.ntiles && ok; tile += grid, ++ti) {
      const uint32_t ab = ti & 1u;
      const uint32_t idesc = tc::idesc_f16(GT_BM, gt_tile<BN>(p, tile).two ? BN : BN / 2);
      if (ti >= 2 && !(ok = tc::mbar_wait(&acc_empty[ab], ((ti >> 1) - 1) & 1))) break;    // read out two tiles ago
      tc::fence_after_sync();
      for (int s = 0; s < slices; ++s) {
        if (!(ok = tc::mbar_wait(XD == BM_F16 ? &loaded[st] : &ready[st], ph))) break;
        if (tc::elect_one()) {
          const uint32_t sa = tc::smem_u32(smem + st * STAGE);
          const uint64_t ad = gt_desc_sw128(sa), bd = gt_desc_sw128(sa + A_BYTES);
#pragma unroll
          for (int kk = 0; kk < GT_BK / 16; ++kk)
            tc::mma_f16(tmem_base + ab * BN, ad + 2 * kk, bd + 2 * kk, idesc, (s > 0 || kk > 0) ? 1u : 0u);
          tc::mma_commit(&empty[st]);
        }
        __syncwarp();
        if (++st == NST) { st = 0; ph ^= 1; }
      }
      if (ok && tc::elect_one()) tc::mma_commit(&acc_full[ab]);
      __syncwarp();
    }
  } else {
    const bool epi = warp >= GT_WARP_EPI0 && warp < GT_WARP_EPI0 + GT_EPI_WARPS;
    if (epi && p.zero)
      for (int64_t i = static_cast<int64_t>(blockIdx.x) * (32 * GT_EPI_WARPS) + threadIdx.x - 32 * GT_WARP_EPI0; i < p.zero_n;
           i += static_cast<int64_t>(gridDim.x) * (32 * GT_EPI_WARPS))
        p.zero[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    // ------------------------------------------------------------------ rounding of the X slice to fp16, in place
    if (XD != BM_F16 && (!epi || all_round)) {
      // Rounding one slice is a chain (wait, load, convert, store, proxy fence, arrive), so groups of warps take the slices in
      // turn and the chains overlap.  A group takes every tr_groups-th stage of the ring: it sees every use of its stages, as
      // its parity waits need.
      const int tw = warp >= GT_WARP_TR0 ? warp - GT_WARP_TR0 : warp < GT_WARP_EPI0 ? warp + 2 : warp - GT_WARP_EPI0 + GT_TR_WARPS;
      const int grp = tw / tr_per, gw = tw - grp * tr_per;
      const int total = p.ntiles > cta ? (p.ntiles - cta + grid - 1) / grid * slices : 0;
      uint32_t cur = grp, ph = 0;
      int k = s_first + grp;                     // slice of its tile
      for (int s = grp; s < total && grp < tr_groups; s += tr_groups) {
        if (!(ok = tc::mbar_wait(&loaded[cur], ph))) break;
        while (k >= s_end) k -= slices;
        unsigned char* sa = smem + cur * STAGE;
        if (k >= p.slices) {
          // second contraction: fp16 already
        } else if (XD == BM_BF16) {
          // 1024 pieces of 16 bytes, element for element (the swizzle only permutes whole pieces)
          constexpr int PIECES = GT_BM * GT_BK * 2 / 16;
          const int STEP = tr_per * 32;
#pragma unroll 1
          for (int i0 = 0; i0 < PIECES; i0 += 4 * STEP) {
            uint4 v[4];
            uint4* q = reinterpret_cast<uint4*>(sa) + i0 + gw * 32 + lane;
#pragma unroll
            for (int u = 0; u < 4; ++u)
              if (i0 + gw * 32 + u * STEP < PIECES) v[u] = q[u * STEP];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              if (i0 + gw * 32 + u * STEP >= PIECES) break;
              uint32_t* w = reinterpret_cast<uint32_t*>(&v[u]);
#pragma unroll
              for (int j = 0; j < 4; ++j) w[j] = pack16(__uint_as_float(w[j] << 16), __uint_as_float(w[j] & 0xffff0000u), BM_F16);
              q[u * STEP] = v[u];
            }
          }
        } else {
          // row r, values 8 j .. 8 j + 7: two 16-byte pieces of box j / 4 -> piece j of the result row; a row's eight lanes
          // have read before any of them overwrites the row's start
          const int j = lane & 7, c4 = 2 * (j & 3);
#pragma unroll 1
          for (int rg = gw; rg < GT_BM / 4; rg += 2 * tr_per) {
            float4 lo[2], hi[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              if (rg + u * tr_per >= GT_BM / 4) break;
              const int r = (rg + u * tr_per) * 4 + (lane >> 3), sw = r & 7;
              const unsigned char* box = sa + (j >> 2) * (A_BYTES / 2) + r * 128;
              lo[u] = *reinterpret_cast<const float4*>(box + ((c4 ^ sw) << 4));
              hi[u] = *reinterpret_cast<const float4*>(box + (((c4 + 1) ^ sw) << 4));
            }
            __syncwarp();
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              if (rg + u * tr_per >= GT_BM / 4) break;
              const int r = (rg + u * tr_per) * 4 + (lane >> 3), sw = r & 7;
              *reinterpret_cast<uint4*>(sa + r * 128 + ((j ^ sw) << 4)) =
                  make_uint4(pack16(lo[u].x, lo[u].y, BM_F16), pack16(lo[u].z, lo[u].w, BM_F16), pack16(hi[u].x, hi[u].y, BM_F16),
                             pack16(hi[u].z, hi[u].w, BM_F16));
            }
          }
        }
        tc::fence_async_smem();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&ready[cur]);
        cur += tr_groups;
        if (cur >= NST) { cur -= NST; ph ^= 1u; }
        k += tr_groups;
      }
    }
    // ------------------------------------------------------------------ epilogue
    if (epi) {
      // warp = (TMEM lane quarter q, every other block of 32 output columns)
      const int q = warp & 3, half = (warp - GT_WARP_EPI0) >> 2;
      unsigned char* stores = smem + NST * STAGE + (warp - GT_WARP_EPI0) * 2 * GT_STORE_BYTES;
      uint32_t ti = 0, sb = 0;
      for (int tile = cta; tile < p.ntiles && ok; tile += grid, ++ti) {
        const GtTile t = gt_tile<BN>(p, tile);
        const GtSeg& sg = p.seg[t.si];
        const uint32_t ab = ti & 1u;
        if (!(ok = tc::mbar_wait(&acc_full[ab], (ti >> 1) & 1))) break;
        tc::fence_after_sync();
        if (SPLIT > 1) {
          // (one tile per cluster) this warp's rows of one half of the tile -> the CTAs that own the columns
          constexpr int RW = BN / 2 / SPLIT, ROW = gt_recv_row(BN, SPLIT);
          tc::cluster_wait();
          const uint32_t mine = tc::smem_u32(smem + NST * STAGE) + ((rank * GT_BM + 32 * q + lane) * ROW + half * RW) * 4;
          const uint32_t acc = tmem_base + (static_cast<uint32_t>(32 * q) << 16) + ab * BN + half * (BN / 2);
          if (half == 0 || t.two) {
#pragma unroll
            for (int c0 = 0; c0 < BN / 2; c0 += 32) {
              float v[32];
              tc::tmem_ld32(acc + c0, v);
#pragma unroll
              for (int j = 0; j < 32; j += 4) {
                const int col = c0 + j;
                asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(tc::cluster_map(mine + (col % RW) * 4, col / RW)), "f"(v[j]), "f"(v[j + 1]),
                             "f"(v[j + 2]), "f"(v[j + 3])
                             : "memory");
              }
            }
          }
          break;
        }
        const int row0 = t.m0 + 32 * q, row = row0 + lane, N = sg.rows;
        const bool with_res = p.residual != nullptr && t.si == 0;
        const uint32_t acc = tmem_base + (static_cast<uint32_t>(32 * q) << 16) + ab * BN;
        const int blocks = (sg.glu ? BN / 2 : t.two ? BN : BN / 2) / 32;
        const float gate = sg.glu && p.row_gate && row < p.M ? p.row_gate[row] : 1.f;
#pragma unroll 1
        for (int b = half; b < blocks; b += 2) {
          const int n = t.n0 + 32 * b;
          if (n >= N) break;
          float v[32];
          tc::tmem_ld32(acc + 32 * b, v);
          if (sg.glu) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              float u[16];
              tc::tmem_ld16(acc + BN / 2 + 32 * b + 16 * h, u);
#pragma unroll
              for (int i = 0; i < 16; ++i) {
                const float g = v[16 * h + i];
                v[16 * h + i] = __fdividef(g, 1.f + __expf(-g)) * u[i] * gate;
              }
            }
          }
          if (sg.c_dtype != BM_F32 && p.tma_store) {
            // 32 rows of 64 bytes, 16-byte pieces in the order of the map's 64-byte swizzle; the block two before has left
            unsigned char* blk = stores + sb * GT_STORE_BYTES;
            sb ^= 1u;
            if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
            __syncwarp();
            unsigned char* mine = blk + lane * 64;
            const int sw = (lane >> 1) & 3;
            if (with_res) {
              const int r = lane >> 2, c = lane & 3;
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int rr = 8 * i + r;
                uint4 x = make_uint4(0u, 0u, 0u, 0u);
                if (row0 + rr < p.M && n + 8 * c < N)
                  x = __ldg(reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(p.residual) + static_cast<size_t>(row0 + rr) * N + n + 8 * c));
                *reinterpret_cast<uint4*>(blk + rr * 64 + ((c ^ ((rr >> 1) & 3)) << 4)) = x;
              }
              __syncwarp();
#pragma unroll
              for (int c2 = 0; c2 < 4; ++c2) {
                const uint4 x = *reinterpret_cast<const uint4*>(mine + ((c2 ^ sw) << 4));
                const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  const float2 f = sg.c_dtype == BM_F16 ? __half22float2(*reinterpret_cast<const __half2*>(&w[j]))
                                                        : __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[j]));
                  v[8 * c2 + 2 * j] += f.x;
                  v[8 * c2 + 2 * j + 1] += f.y;
                }
              }
            }
#pragma unroll
            for (int c = 0; c < 4; ++c)
              *reinterpret_cast<uint4*>(mine + ((c ^ sw) << 4)) =
                  make_uint4(pack16(v[8 * c], v[8 * c + 1], sg.c_dtype), pack16(v[8 * c + 2], v[8 * c + 3], sg.c_dtype),
                             pack16(v[8 * c + 4], v[8 * c + 5], sg.c_dtype), pack16(v[8 * c + 6], v[8 * c + 7], sg.c_dtype));
            tc::fence_async_smem();
            __syncwarp();
            if (lane == 0) tma_store_2d(&p.c[t.si], n, row0, blk);       // rows and columns past the matrix are clipped
          } else if (row < p.M) {
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              if (n + i < N) {
                const size_t idx = static_cast<size_t>(row) * N + n + i;
                float val = v[i];
                if (with_res) val += load_act(p.residual, sg.c_dtype, idx);
                store_act(sg.C, sg.c_dtype, idx, val);
              }
            }
          }
        }
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&acc_empty[ab]);
      }
      if (SPLIT == 1 && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
  }
  if (SPLIT > 1) {
    const bool epi = warp >= GT_WARP_EPI0 && warp < GT_WARP_EPI0 + GT_EPI_WARPS;
    if (!epi || !ok) tc::cluster_wait();         // (the epilogue warps have, unless their accumulator did not come)
    tc::cluster_arrive();
    tc::cluster_wait();                          // every share of this CTA's columns is there
    if (epi) {
      constexpr int RW = BN / 2 / SPLIT, ROW = gt_recv_row(BN, SPLIT);
      const GtTile t = gt_tile<BN>(p, cta);
      const GtSeg& sg = p.seg[t.si];
      const int i = threadIdx.x - 32 * GT_WARP_EPI0, r = i >> 1, h = i & 1, row = t.m0 + r, N = sg.rows;
      const float* recv = reinterpret_cast<const float*>(smem + NST * STAGE) + r * ROW;
      const float gate = sg.glu && p.row_gate && row < p.M ? p.row_gate[row] : 1.f;
      const bool with_res = p.residual != nullptr && t.si == 0;
      if (row < p.M && (sg.glu ? h == 0 : h == 0 || t.two)) {
#pragma unroll
        for (int c = 0; c < RW; c += 8) {
          const int n = t.n0 + (sg.glu ? 0 : h * (BN / 2)) + rank * RW + c;
          if (n >= N) break;                     // (rows of a stack come in eights)
          float v[8] = {}, u[8] = {};
#pragma unroll
          for (int src = 0; src < SPLIT; ++src)
#pragma unroll
            for (int j = 0; j < 8; j += 4) {
              const float4 a = *reinterpret_cast<const float4*>(recv + src * GT_BM * ROW + h * RW + c + j);
              v[j] += a.x; v[j + 1] += a.y; v[j + 2] += a.z; v[j + 3] += a.w;
              if (sg.glu) {
                const float4 b = *reinterpret_cast<const float4*>(recv + src * GT_BM * ROW + RW + c + j);
                u[j] += b.x; u[j + 1] += b.y; u[j + 2] += b.z; u[j + 3] += b.w;
              }
            }
          const size_t idx = static_cast<size_t>(row) * N + n;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (sg.glu) v[j] = __fdividef(v[j], 1.f + __expf(-v[j])) * u[j] * gate;
            if (with_res) v[j] += load_act(p.residual, sg.c_dtype, idx + j);
          }
          if (sg.c_dtype != BM_F32 && p.tma_store) {
            *reinterpret_cast<uint4*>(static_cast<uint16_t*>(sg.C) + idx) = make_uint4(pack16(v[0], v[1], sg.c_dtype), pack16(v[2], v[3], sg.c_dtype),
                                                                                       pack16(v[4], v[5], sg.c_dtype), pack16(v[6], v[7], sg.c_dtype));
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) store_act(sg.C, sg.c_dtype, idx + j, v[j]);
          }
        }
      }
    }
  }
  if (!ok && lane == 0 && p.status) atomicExch(p.status, BM_ERR_TIMEOUT);
  if (p.beside) grid_wait();
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 2) tc::tmem_dealloc(tmem_base, TMEM_COLS);
}

// ---- host side -------------------------------------------------------------------------------------------------------

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &qres) != cudaSuccess || qres != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<EncodeTiledFn>(f);
  }();
  return fn;
}

// [rows, cols] row-major, boxes of box_rows x box_bytes (128 or 64) with the swizzle of that width
static bool make_map(CUtensorMap* map, const void* base, int rows, int cols, int elem_bytes, int box_rows, int box_bytes) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(cols) * elem_bytes};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(box_bytes / elem_bytes), static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t estr[2] = {1, 1};
  return fn(map, elem_bytes == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(base), dims,
            strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, box_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN, int XD, int SPLIT>
static int launch_one(const GtParams& p, LaunchAfter after, int grid, cudaStream_t st) {
  const int smem = gt_stages(BN, XD, SPLIT) * gt_stage_bytes(BN, XD) + gt_tail_bytes(BN, SPLIT) + 1024;
  static PerDeviceOnce once;
  int dev = -1;
  BM_CUDA(cudaGetDevice(&dev));
  if (!once.is_done(dev)) {
    BM_CUDA(cudaFuncSetAttribute(gemm_tma_kernel<BN, XD, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    once.mark(dev);
  }
  BM_CUDA(launch_after(after, SPLIT, gemm_tma_kernel<BN, XD, SPLIT>, dim3(grid * SPLIT), GT_THREADS, smem, st, p));
  BM_LAUNCH_CHECK("gemm_tma_kernel");
  return BM_OK;
}
template <int BN, int SPLIT>
static int launch_typed(const GtParams& p, int x_dtype, LaunchAfter after, int grid, cudaStream_t st) {
  if (x_dtype == BM_F32) return launch_one<BN, BM_F32, SPLIT>(p, after, grid, st);
  if (x_dtype == BM_BF16) return launch_one<BN, BM_BF16, SPLIT>(p, after, grid, st);
  return launch_one<BN, BM_F16, SPLIT>(p, after, grid, st);
}

// Returns BM_ERR_UNSUPPORTED (without having launched anything) when the shape or the pointers do not suit tiled
// copies; the caller then takes the cp.async kernel, a product at a time.
int launch_gemm_tma(const GemmTmaArgs& a, cudaStream_t st) {
  const int xb = a.x_dtype == BM_F32 ? 4 : 2;
  auto aligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
  if (a.K <= 0 || a.K % GT_BK != 0 || a.K2 % GT_BK != 0 || a.M <= 0 || a.n_seg < 1 || a.n_seg > GEMM_MAX_SEG || !aligned(a.X) || !aligned(a.X2) ||
      !aligned(a.W2) || (a.K2 && a.n_seg != 1))
    return BM_ERR_UNSUPPORTED;
  static PerDeviceOnce once;
  static int sm_counts[MAX_DEVICES];
  int dev = -1;
  BM_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= MAX_DEVICES) return BM_ERR_UNSUPPORTED;
  if (!once.is_done(dev)) {
    BM_CUDA(cudaDeviceGetAttribute(&sm_counts[dev], cudaDevAttrMultiProcessorCount, dev));
    once.mark(dev);
  }
  GtParams p;
  memset(&p, 0, sizeof(p));
  const int tiles_m = (a.M + GT_BM - 1) / GT_BM;
  auto lay_out = [&](int bn) {
    p.tiles_n = 0;
    for (int i = 0; i < a.n_seg; ++i) {
      p.seg[i].tile0 = p.tiles_n;
      const int per = a.seg[i].W_up ? bn / 2 : bn;
      p.tiles_n += (a.seg[i].rows + per - 1) / per;
    }
    return tiles_m * p.tiles_n;
  };
  // Tile width and split of the contraction.  Where the wide tile would leave most SMs idle: what takes the fewest slices one
  // after the other.  A slice of a 128-column tile counts 1.15 of a 64-column one, two more stand for start and end, three for
  // the exchange of a split; clusters of four leave a few SMs of a group unused.  Basis pair of 2 x 256 rows, hidden 2048, bf16,
  // us at 64 / 128 / 256 columns, then 64 split in 2 / 4: 300 tokens 13.2 14.5 18.8 11.6 9.4, 777 tokens 13.5 14.6 18.9 11.8 -,
  // 2048 tokens 13.9 15.7 20.8 - -, 4096 tokens 28.3 16.2 21.4 - -, 6000 tokens 40.6 30.3 21.8 - -.
  int bn = 256, split = 1;
  if (lay_out(256) < sm_counts[dev] / 2) {
    const int slices = (a.K + a.K2) / GT_BK;
    double best = 1e30;
    for (const auto& c : {std::make_pair(64, 1), std::make_pair(128, 1), std::make_pair(64, 2), std::make_pair(64, 4)}) {
      const int tiles = lay_out(c.first), most = c.second == 4 ? sm_counts[dev] * 7 / 8 : sm_counts[dev];
      if (c.second > 1 && (tiles * c.second > most || slices < 4 * c.second)) continue;
      const int waves = (tiles * c.second + sm_counts[dev] - 1) / sm_counts[dev];
      const double cost = waves * ((slices + c.second - 1) / c.second + 2) * (c.first > 64 ? 1.15 : 1.0) + (c.second > 1 ? 3 : 0);
      if (cost < best) { best = cost; bn = c.first; split = c.second; }
    }
  }
  p.ntiles = lay_out(bn);
  if (!make_map(&p.x, a.X, a.M, a.K, xb, GT_BM, 128)) return BM_ERR_UNSUPPORTED;
  if (a.K2 && (!make_map(&p.x2, a.X2, a.M, a.K2, 2, GT_BM, 128) || !make_map(&p.w2, a.W2, a.seg[0].rows, a.K2, 2, bn / 2, 128))) return BM_ERR_UNSUPPORTED;
  p.tma_store = aligned(a.residual);
  int maps = 0;
  for (int i = 0; i < a.n_seg; ++i) {
    const GemmSeg& s = a.seg[i];
    if (s.rows <= 0 || s.rows % 8 != 0 || !aligned(s.W) || !aligned(s.W_up) || maps + 2 > GEMM_MAX_SEG + 2) return BM_ERR_UNSUPPORTED;
    GtSeg& d = p.seg[i];
    d.C = s.C; d.rows = s.rows; d.c_dtype = s.c_dtype; d.glu = s.W_up != nullptr;
    d.map_w = maps++;
    if (!make_map(&p.w[d.map_w], s.W, s.rows, a.K, 2, bn / 2, 128)) return BM_ERR_UNSUPPORTED;
    if (d.glu) {
      d.map_up = maps++;
      if (!make_map(&p.w[d.map_up], s.W_up, s.rows, a.K, 2, bn / 2, 128)) return BM_ERR_UNSUPPORTED;
    }
    if (s.c_dtype != BM_F32 && (!aligned(s.C) || !make_map(&p.c[i], s.C, a.M, s.rows, 2, 32, 64))) p.tma_store = 0;
  }
  p.residual = a.residual; p.row_gate = a.row_gate; p.n_seg = a.n_seg; p.M = a.M;
  p.slices = a.K / GT_BK; p.slices2 = a.K2 / GT_BK;
  p.status = a.status;
  p.beside = a.after == AFTER_BESIDE;
  p.zero = a.zero; p.zero_n = a.zero_n;
  const int grid = split > 1 || p.ntiles < sm_counts[dev] ? p.ntiles : sm_counts[dev];
  if (bn == 64) return split == 1 ? launch_typed<64, 1>(p, a.x_dtype, a.after, grid, st) : split == 2 ? launch_typed<64, 2>(p, a.x_dtype, a.after, grid, st) : launch_typed<64, 4>(p, a.x_dtype, a.after, grid, st);
  if (bn == 128) return launch_typed<128, 1>(p, a.x_dtype, a.after, grid, st);
  return launch_typed<256, 1>(p, a.x_dtype, a.after, grid, st);
}

int launch_gemm_basis(const GemmTcArgs& a, int problems, cudaStream_t st) {
  GemmTmaArgs t{};
  t.X = a.X; t.x_dtype = a.x_dtype; t.M = a.M; t.K = a.K; t.residual = a.residual; t.status = a.status;
  t.n_seg = problems;
  t.after = a.after; t.zero = a.zero; t.zero_n = a.zero_n;
  for (int i = 0; i < problems; ++i) t.seg[i] = GemmSeg{a.W[i], nullptr, a.C[i], a.N, a.c_dtype};
  const int rc = launch_gemm_tma(t, st);
  if (rc != BM_ERR_UNSUPPORTED) return rc;
  if (a.zero) BM_CUDA(cudaMemsetAsync(a.zero, 0, static_cast<size_t>(a.zero_n) * 16, st));
  return launch_gemm_tc(a, problems, st);
}

}  // namespace bm
