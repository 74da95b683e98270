// Quantise + bit-plane pack + runtime-layout reorder of one slab in one kernel.
//
// Restates, fused, what the reference's packer does per slab in three steps
// (bitsmoe/quant/packer.py:210-306): quantize_symmetric per (rank row, 128-column tile)
// (bitsmoe/quant/quantizer.py:30-84: sign / mean-|x| for 1 bit; 50 rounds of alternating least squares on the scale for
// 2/3/4 bits; absmax for 6/8 bits; round half to even), BitPack.pack into 32-column bit-planes
// (bitsmoe/quant/bitpack/bitpack_cuda_kernel.cu:81-121) and the [tile][stage 16 rows][micro][row][plane] reorder
// (packer.py:169-207).  One warp owns one (row, tile) group: lane l holds columns 32 m + l of the tile (m = 0..3), so
// a plane word is one __ballot_sync and lands at its final payload position directly.
//
// 256 rows x 768 columns in three bit widths: six launches of 22 us each -> one of 17 us; with the host path around it
// (tables native, one pinned copy, tables built while the device works) a matrix takes 67 us instead of 616.
#include "common.cuh"

namespace bm {

constexpr float Q_EPS = 1e-8f;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// One (rank row, 128-column tile) group by one warp: lane l holds columns 32 m + l (m = 0..3).  Quantises, writes the
// group's scale to *scale_out and its plane words (16 bits: its raw fp16 pairs) to out[micro * rows_cur * words + word].
//
// What bounds it is the serial chain of the scale refinement -- divide, round, two warp sums, three divides, 50 times --
// at a warp or two per scheduler.  The scale determines the codes and the codes the next scale, so a round that returns
// the scale it was given has reached the fixed point that the remaining rounds would keep, and the loop ends there.
__device__ __forceinline__ void quantize_pack_group(const float (&x)[MICROS], const bool (&live)[MICROS], int n_valid, int bits,
                                                    __half* scale_out, uint32_t* out, int rows_cur, int8_t* codes) {
  const int lane = threadIdx.x & 31;
  if (bits == 16) {
    if (lane == 0) *scale_out = __float2half_rn(1.f);
#pragma unroll
    for (int m = 0; m < MICROS; ++m) {
      const uint32_t h = __half_as_ushort(__float2half_rn(live[m] ? x[m] : 0.f));
      const uint32_t lo = __shfl_sync(0xffffffffu, h, (2 * lane) & 31), hi = __shfl_sync(0xffffffffu, h, (2 * lane + 1) & 31);
      if (lane < 16) out[m * rows_cur * 16 + lane] = lo | (hi << 16);
    }
    return;
  }
  // means are sums divided by the count, products and sums rounded separately (no fused multiply-add), as the
  // element-wise torch expressions of the reference round them
  // (a count that is a power of two has an exact reciprocal: its product rounds to what the quotient rounds to)
  const float n_f = static_cast<float>(n_valid), n_inv = 1.f / n_f;
  const bool pow2 = (n_valid & (n_valid - 1)) == 0;
  auto mean = [&](float sum) { return pow2 ? __fmul_rn(sum, n_inv) : __fdiv_rn(sum, n_f); };
  float sabs = 0.f;
#pragma unroll
  for (int m = 0; m < MICROS; ++m) sabs = __fadd_rn(sabs, fabsf(x[m]));
  const float mean_abs = fmaxf(mean(warp_sum(sabs)), Q_EPS);
  const int hi = (1 << (bits - 1)) - 1, lo = -hi - 1;
  float q[MICROS];
  float scale;
  if (bits == 1) {
#pragma unroll
    for (int m = 0; m < MICROS; ++m) q[m] = x[m] < 0.f ? -1.f : 1.f;
    scale = mean_abs;
  } else if (bits <= 4) {
    scale = mean_abs;
    for (int it = 0; it < 50; ++it) {
      float xq = 0.f;
      int qq = 0;      // whole and below 2^24: the same sum in any order, so the integer adder takes it in one step
#pragma unroll
      for (int m = 0; m < MICROS; ++m) {
        q[m] = fminf(fmaxf(rintf(__fdiv_rn(x[m], scale)), static_cast<float>(lo)), static_cast<float>(hi));
        xq = __fadd_rn(xq, __fmul_rn(x[m], q[m]));
        qq += static_cast<int>(q[m]) * static_cast<int>(q[m]);
      }
      const float mean_qq = mean(static_cast<float>(__reduce_add_sync(0xffffffffu, qq)));
      const float next = fmaxf(__fdiv_rn(mean(warp_sum(xq)), __fadd_rn(mean_qq, Q_EPS)), Q_EPS);
      if (next == scale) break;
      scale = next;
    }
  } else {
    float amax = 0.f;
#pragma unroll
    for (int m = 0; m < MICROS; ++m) amax = fmaxf(amax, fabsf(x[m]));
    scale = fmaxf(__fdiv_rn(warp_max(amax), static_cast<float>(hi)), Q_EPS);
#pragma unroll
    for (int m = 0; m < MICROS; ++m) q[m] = fminf(fmaxf(rintf(__fdiv_rn(x[m], scale)), static_cast<float>(lo)), static_cast<float>(hi));
  }
  if (lane == 0) *scale_out = __float2half_rn(scale);
  // stored unsigned codes (columns past the matrix hold code 0) and their planes
  const int offset = bits == 1 ? 0 : (1 << (bits - 1));
#pragma unroll
  for (int m = 0; m < MICROS; ++m) {
    const int qi = live[m] ? static_cast<int>(q[m]) : 0;
    const int u = bits == 1 ? ((qi + 1) >> 1) : (qi + offset);
    if (codes) codes[m * N_MICRO + lane] = static_cast<int8_t>(qi);
    for (int p = 0; p < bits; ++p) {
      const uint32_t word = __ballot_sync(0xffffffffu, (u >> p) & 1);
      if (lane == 0) out[m * rows_cur * bits + p] = word;
    }
  }
}

// Where row r of a slab of k rows keeps its words inside one tile's block: first word, and rows of its stage.
__device__ __forceinline__ int slab_row_word(int r, int k, int words, int* rows_cur) {
  const int full = (k / K_STAGE) * K_STAGE;
  const int s0 = r < full ? (r / K_STAGE) * K_STAGE : full;
  *rows_cur = r < full ? K_STAGE : k - full;
  return s0 * MICROS * words + (r - s0) * words;
}

__device__ __forceinline__ void load_group(const float* row, int col0, int n_valid, float (&x)[MICROS], bool (&live)[MICROS]) {
#pragma unroll
  for (int m = 0; m < MICROS; ++m) {
    const int c = m * N_MICRO + (threadIdx.x & 31);
    live[m] = c < n_valid;
    x[m] = live[m] ? row[col0 + c] : 0.f;
  }
}

// grid (ceil(k / 8), tiles), 8 warps per block.
__global__ void __launch_bounds__(256) quantize_pack_slab_kernel(const float* __restrict__ rows, int64_t ld, int k, int dim, int bits,
                                                                 uint32_t* __restrict__ payload, __half* __restrict__ scale_out,
                                                                 int8_t* __restrict__ codes_out) {
  const int r = blockIdx.x * 8 + (threadIdx.x >> 5);
  const int tile = blockIdx.y;
  if (r >= k) return;
  const int col0 = tile * N_TILE, n_valid = min(N_TILE, dim - col0);
  float x[MICROS];
  bool live[MICROS];
  load_group(rows + static_cast<int64_t>(r) * ld, col0, n_valid, x, live);
  int rows_cur;
  const int word = slab_row_word(r, k, bits, &rows_cur);
  quantize_pack_group(x, live, n_valid, bits, scale_out + static_cast<int64_t>(tile) * k + r,
                      payload + static_cast<int64_t>(tile) * k * MICROS * bits + word, rows_cur,
                      codes_out ? codes_out + static_cast<int64_t>(r) * (gridDim.y * N_TILE) + col0 : nullptr);
}

// All slabs of a matrix in one launch: the slabs of one matrix are small (64 rows x a few tiles), so one launch each
// leaves the chip to the latency of a single warp's refinement, once per slab.  grid (ceil(rows / 8), tiles); the row
// order and the slab table travel as kernel parameters.
constexpr int QM_ROWS = 1024, QM_SLABS = 32;
struct PackMatrixParams {
  const float* src;
  int64_t ld;
  const float* s;
  uint32_t* payload;
  __half* scale;
  __half* s_out;
  int dim, n_rows, row0;                // row0: stored index of the launch's first row
  struct { int bits, k, first, scale_off; int64_t word_off; } slab[QM_SLABS];
  int32_t row[QM_ROWS];                 // logical row of every stored row
  uint8_t slab_of[QM_ROWS];
};
__global__ void __launch_bounds__(256) quantize_pack_matrix_kernel(const __grid_constant__ PackMatrixParams p) {
  const int i = blockIdx.x * 8 + (threadIdx.x >> 5), tile = blockIdx.y;
  if (i >= p.n_rows) return;
  const auto& sl = p.slab[p.slab_of[i]];
  const int src = p.row[i], r = i - sl.first, words = words_per_row(sl.bits);
  if (tile == 0 && (threadIdx.x & 31) == 0) p.s_out[p.row0 + i] = __float2half_rn(p.s[src]);
  const int col0 = tile * N_TILE, n_valid = min(N_TILE, p.dim - col0);
  float x[MICROS];
  bool live[MICROS];
  load_group(p.src + src * p.ld, col0, n_valid, x, live);
  int rows_cur;
  const int word = slab_row_word(r, sl.k, words, &rows_cur);
  quantize_pack_group(x, live, n_valid, sl.bits, p.scale + sl.scale_off + tile * sl.k + r,
                      p.payload + sl.word_off + static_cast<int64_t>(tile) * sl.k * MICROS * words + word, rows_cur, nullptr);
}

}  // namespace bm

extern "C" int bm_quantize_pack_slab(const float* rows, int64_t row_stride, int32_t k, int32_t dim, int32_t bits, uint32_t* payload,
                                     uint16_t* scale, int8_t* codes, void* stream) {
  using namespace bm;
  BM_REQUIRE(k >= 0 && dim > 0 && row_stride >= dim, BM_ERR_INVALID_ARG, "quantize_pack_slab: bad sizes");
  BM_REQUIRE(bits == 1 || bits == 2 || bits == 3 || bits == 4 || bits == 6 || bits == 8, BM_ERR_UNSUPPORTED,
             "Unsupported bits=%d", bits);
  BM_REQUIRE(dim % N_MICRO == 0, BM_ERR_INVALID_ARG, "quantize_pack_slab: dim=%d must be divisible by %d", dim, N_MICRO);
  if (k == 0) return BM_OK;
  BM_REQUIRE(rows && payload && scale, BM_ERR_INVALID_ARG, "quantize_pack_slab: null pointer");
  const int tiles = (dim + N_TILE - 1) / N_TILE;
  dim3 grid((k + 7) / 8, tiles);
  quantize_pack_slab_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(rows, row_stride, k, dim, bits, payload,
                                                                                reinterpret_cast<__half*>(scale), codes);
  BM_LAUNCH_CHECK("quantize_pack_slab_kernel");
  return BM_OK;
}

extern "C" int bm_quantize_pack_matrix(const float* rank_major, int64_t row_stride, const float* s, int32_t dim, const int32_t* rows,
                                       const int32_t* slabs, int32_t n_slabs, uint32_t* payload, uint16_t* scale, uint16_t* s_out,
                                       void* stream) {
  using namespace bm;
  BM_REQUIRE(dim > 0 && row_stride >= dim && n_slabs >= 0, BM_ERR_INVALID_ARG, "quantize_pack_matrix: bad sizes");
  BM_REQUIRE(dim % N_MICRO == 0, BM_ERR_INVALID_ARG, "quantize_pack_matrix: dim=%d must be divisible by %d", dim, N_MICRO);
  if (n_slabs == 0) return BM_OK;
  BM_REQUIRE(rank_major && s && rows && slabs && payload && scale && s_out, BM_ERR_INVALID_ARG, "quantize_pack_matrix: null pointer");
  const int tiles = (dim + N_TILE - 1) / N_TILE;
  int64_t word_off = 0;
  int scale_off = 0, row0 = 0, i = 0;
  PackMatrixParams p;
  p.src = rank_major; p.ld = row_stride; p.s = s; p.payload = payload;
  p.scale = reinterpret_cast<__half*>(scale); p.s_out = reinterpret_cast<__half*>(s_out); p.dim = dim;
  while (i < n_slabs) {
    p.n_rows = 0;
    p.row0 = row0;
    int n = 0;
    for (; i < n_slabs && n < QM_SLABS; ++i, ++n) {
      const int bits = slabs[2 * i], k = slabs[2 * i + 1];
      BM_REQUIRE(supported_bits(bits), BM_ERR_UNSUPPORTED, "Unsupported bits=%d", bits);
      BM_REQUIRE(k >= 1 && k <= K_SLAB, BM_ERR_INVALID_ARG, "quantize_pack_matrix: slab of %d rows", k);
      if (p.n_rows + k > QM_ROWS) break;
      p.slab[n].bits = bits; p.slab[n].k = k; p.slab[n].first = p.n_rows;
      p.slab[n].scale_off = scale_off; p.slab[n].word_off = word_off;
      for (int r = 0; r < k; ++r) {
        p.row[p.n_rows + r] = rows[row0 + r];
        p.slab_of[p.n_rows + r] = static_cast<uint8_t>(n);
      }
      p.n_rows += k;
      row0 += k;
      scale_off += tiles * k;
      word_off += static_cast<int64_t>(tiles) * k * MICROS * words_per_row(bits);
    }
    quantize_pack_matrix_kernel<<<dim3((p.n_rows + 7) / 8, tiles), 256, 0, static_cast<cudaStream_t>(stream)>>>(p);
    BM_LAUNCH_CHECK("quantize_pack_matrix_kernel");
  }
  return BM_OK;
}
