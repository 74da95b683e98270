// Packed routed-expert forward for large token counts (prefill): fused mixed-bit grouped GEMM on the
// 5th-generation tensor cores (tcgen05.mma, accumulators in tensor memory), a pair of CTAs per work item.
//
// Work item = (expert, block of up to 2 NT of its assignments; NT = ROWS = 128 or 64 where it fits).  A persistent pair of CTAs
// (cluster of two, cta_group::2) walks the items; each CTA holds half of the item's tokens as ROWS rows (M) of every product and
// converts half of the weights, its columns (N); the tensor cores read both halves, so the converted weights never cross the
// cluster.  The tile's columns are taken a chunk (64, with 64 rows 128) at a time:
//   gate/up:  D_g[n, c] = sum_slot act_g[n, slot] * W_g[c, slot]     (N = the chunk's columns c, half from each CTA; K = row slots)
//   down:     D_d[n, slot] += sum_c z[n, c] * W_d[slot, c]           (N = 128 row slots x 1..3, 64 from each CTA; K = the chunk's columns)
// Tokens as rows make the epilogue cheap: a thread owns a token.  Tensor memory holds two gate/up accumulator pairs beside the
// down accumulator, so the products of a chunk run while the previous one is turned into z.  128 rows: a lane is a row; z goes
// back to tensor memory, over the gate sums it came from, and is the A operand of the down product there.  64 rows: lanes 0-63
// hold the lower half of an accumulator's columns, lanes 64-127 the upper half, which leaves columns for chunks of 128 and for three down
// tiles (matrices of 257 to 384 slots take this form at any load); z is an operand in shared memory.
//
// Warp roles (768 threads; the last warp completes the last warpgroup):
//   warps 0-7   epilogue (two per TMEM lane quarter, 32 columns each): tcgen05.ld D_g/D_u -> z = silu(g)*u -> fp16;
//               at the end of the item D_d * s * route weight is turned through shared memory and added to rank_accum in
//               16-byte vector reductions, beside the next item's staging.
//   warps 8-19  converters, one team of six warps per pipeline: arena words (nibble / dense 2-bit codes), read straight
//               from L2 one stage ahead into registers, -> fp16 (q * scale) operand stages of 2048 codes in the
//               canonical K-major core-matrix layout, a ring of two-stage slots per pipeline, a stage per warp.  Before an
//               item's stages they build its activation operand act[n, slot] = fp16(h[token, rank(slot)] * s(slot)).
//   warp  20    looks up the next item while the current one runs and asks L2 for its weights
//   warps 21,22 (of the even CTA) MMA issue for both CTAs, one thread each: gate products and the down product's even slot
//               tiles; up products and the odd ones.  The waits and commits of one pipeline hide behind the products of the
//               other, and they never write the same accumulator.
// The roles walk the items on their own barriers, so an item's staging runs beside the last products and sums of the one
// before.  What an MMA issuer waits for is signalled by both CTAs (mapped arrivals on the even CTA's barriers), what waits for
// MMAs is signalled in both by the commit.
//
// What bounds it.  128 rows: the MMAs.  A chunk of 64 columns is 32 of N = 64, which take about 50 cycles each whatever their
// rows (they read 4 KB of activations from shared memory), and 8 of N = 128: 2.1 K cycles of 3.6 K a chunk all in; the rest is
// the way through ring, epilogue and arrivals, and 6 K cycles an item in which the activations are staged.  64 rows: the chain of
// the converter warps (an MMA of 64 rows takes as long as one of 128, but N = 128 halves their number); a stage is about 280
// instructions at 8 cycles each, and what the instruction cache holds of 24 warps in different roles matters: a copy of the
// loop for each kind of stage took 60 us where one for all takes 40 (203 tokens), one for gate/up and down together 42.
// Stage of 8192 tokens of 128 experts (rank 256, intermediate 768): 118 us (176 before weights were converted in pairs), 2048
// tokens 59 (72), 777 tokens 45 (59), 300 tokens 40 (50); of 512 experts: 16384 tokens 235 us (318), 2048 tokens 99 (125 with 128
// rows), 1050 tokens 90 (114).
// The mapped arrivals carry no cluster-scope release: what they publish is read by the tensor core of the CTA that wrote it, behind
// the proxy fence, and is in shared memory before the arrival leaves.  The PTX memory model does not promise this order to the other CTA's
// issuer; it rests on the hardware.  A form that it does cover -- arrivals within a CTA, passed on by warps of the odd CTA with
// .release.cluster and waited for with .acquire.cluster -- gives the same bits in deterministic mode (1200 runs of 520 to 4096
// tokens, two shapes) and takes a layer call of 8192 tokens from 180 to 208 us, a block of 777 from 78 to 100, 2048 tokens of 64 experts from
// 155 to 163; with the release in the converters' own arrivals, 1.4 K cycles each, the stage of 8192 tokens takes 165 us.
//
// The down product of a chunk is issued one chunk late (G0 U0 | G1 U1 D0 | G2 U2 D1 | ...).  Every mbarrier wait is
// bounded in time.  One that gives up raises a flag in both CTAs; the roles then leave at their next wait that is not over, the
// look-up warp behind its copy, both CTAs behind the MMAs issued so far, and tensor memory is given back after that.
#include <algorithm>
#include <limits>

#include "dequant.cuh"
#include "tc05.cuh"

namespace bm {

int expected_passes(int experts, double load, int size);      // layer.cu

constexpr int XT_NT_MAX = 128;            // most tokens (assignments) of an item in a CTA: its rows of one MMA
constexpr int XT_THREADS = 768;
constexpr int XT_EPI_WARPS = 8, XT_DQ_WARP0 = 8, XT_DQ_WARPS = 12, XT_LOOKUP_WARP = 20, XT_MMA_WARP0 = 21;
constexpr int XT_TEAM = XT_DQ_WARPS / 2;  // converter warps per pipeline
// Registers per thread at launch (what 768 threads leave) and per role afterwards: the converters, which keep two stages'
// words and four independent blocks in flight, take what the roles with little state give back.
constexpr int XT_REGS = 80, XT_REGS_EPI = 80, XT_REGS_DQ = 88, XT_REGS_MISC = 56;
static_assert(32 * (XT_EPI_WARPS * XT_REGS_EPI + XT_DQ_WARPS * XT_REGS_DQ + 4 * XT_REGS_MISC) <= XT_THREADS * XT_REGS,
              "the roles' registers come out of the launch's");
constexpr int XT_ACC = 64;                // columns of tensor memory of a gate or up accumulator
// Tile columns per step, by the rows (tokens) of a CTA: 64 rows of a pair's accumulator take half as many columns as it has
__host__ __device__ constexpr int xt_chunk(int rows) { return rows > 64 ? 64 : 128; }
__host__ __device__ constexpr int xt_down_cols(int rows) { return rows > 64 ? 128 : 64; }
// Operand slots per pipeline, by the rows (tokens) of a CTA
__host__ __device__ constexpr int xt_ring(int rows) { return rows > 64 ? 4 : 6; }
constexpr int XT_RING_MAX = 6;
// A weight slot: this CTA's half of the rows of one B operand, in two stages that two warps fill.
//   gate/up  128 rows: 32 columns of the chunk x 128 row slots (four pairs of 16-slot blocks; a stage is two of them)
//            64 rows: 64 columns x 64 slots (a stage is a pair)
//   down     64 slots of a 128-slot tile x 64 columns (a stage is 32 of them)
// Bytes between 8-position chunks, padded: the 16-byte stores of a quarter warp hit distinct banks.
constexpr int XT_N32_STRIDE = 32 * 16 + 32, XT_N64_STRIDE = 64 * 16 + 32;
__host__ __device__ constexpr int xt_g_stride(int rows) { return rows > 64 ? XT_N32_STRIDE : XT_N64_STRIDE; }
constexpr int XT_D_STRIDE = XT_N64_STRIDE;
constexpr int XT_SLOT_BYTES = 16 * XT_N32_STRIDE;
static_assert(8 * XT_N64_STRIDE <= XT_SLOT_BYTES, "a slot of 64-row operands fits");
constexpr int XT_Z_STRIDE = 64 * 16 + 16, XT_Z_BYTES = 16 * XT_Z_STRIDE;      // z operand in shared memory (64 rows x 128 columns): bytes between chunks, a buffer
constexpr int XT_TURN_BYTES = 2048;       // where an epilogue warp turns its sums: 16 tokens x 32 slots (64 rows: its part of the idle z operand)
__host__ __device__ constexpr int xt_z_or_turn_bytes(int rows) { return rows > 64 ? XT_EPI_WARPS * XT_TURN_BYTES : 2 * XT_Z_BYTES; }
// bytes between 8-position chunks of the token-side operands (padded: conflict-free stores)
__host__ __device__ constexpr int xt_chunk_stride(int nt) { return nt * 16 + 16; }
constexpr int XT_MAX_E = 1024, XT_MAX_SLOTS = 3 * 128;

struct XtBars {
  uint64_t w_full[2 * XT_RING_MAX], w_empty[2 * XT_RING_MAX];     // weight slots of the pipelines
  uint64_t item_full[2], item_free[2];    // an item's description and table are there / no role needs them any more
  uint64_t act_ready, act_free;           // activation operand written / every product with it complete
  uint64_t gu_done[2];                    // gate/up accumulators of a chunk complete
  uint64_t z_ready[2], z_free[2];         // accumulators read out and z written over them / z multiplied
  uint64_t down_done, down_free;          // down sums of an item complete / read out
  uint64_t drained[2];                    // every MMA of the pipeline complete (at the end of the kernel)
};

struct XtItem {
  int tok[XT_NT_MAX];
  float rw[XT_NT_MAX];
  int n, chunk0, nchunk;
  int pad_;
};

// abort_flag[0]: a wait of this CTA or of its peer gave up; abort_flag[1]: the limit of a wait in microseconds
__device__ __noinline__ void xt_give_up(volatile int* abort_flag) {
  *abort_flag = 1;
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(tc::cluster_map(tc::smem_u32(const_cast<int*>(abort_flag)), tc::cluster_rank() ^ 1u)), "r"(1) : "memory");
}
__device__ __forceinline__ bool xt_wait_slow(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  const uint32_t addr = tc::smem_u32(bar);
  uint64_t t0 = 0;
  for (uint32_t i = 0;; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity), "r"(20000u)
        : "memory");
    if (done) return true;
    if (*abort_flag) return false;
    if ((i & 15u) == 15u) {
      const uint64_t now = tc::global_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > static_cast<uint64_t>(abort_flag[1]) * 1000u) { xt_give_up(abort_flag); return false; }
    }
  }
}
// Bounded wait: one probe inline (the common case in a running pipeline), the time-limited loop out of line.
__device__ __forceinline__ bool xt_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  uint32_t done;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(done)
               : "r"(tc::smem_u32(bar)), "r"(parity)
               : "memory");
  return done ? true : xt_wait_slow(bar, parity, abort_flag);
}

// How a group's words become weights (dequant.cuh), in registers: the converters hold one copy of their code for nibble and
// dense words.  With a copy for each the instruction cache does not hold what 24 warps in different roles run.
struct XtFields {
  uint32_t mlo, mhi, shift, blo, bhi;
  bool nib;
  __device__ __forceinline__ explicit XtFields(bool n) : nib(n) {
    const uint32_t off = n ? FAST_NIB_OFFSET : FAST_DENSE_OFFSET;
    mlo = n ? 0x000F000Fu : 0x00030003u;
    mhi = mlo << 4;
    shift = n ? 8u : 2u;
    blo = 0x64006400u + off * 0x00010001u;
    bhi = 0x54005400u + off * 0x00100010u;
  }
};
__device__ __forceinline__ uint32_t xt_weight(uint32_t w, uint32_t mask, uint32_t magic, uint32_t sub, __half2 scale) {
  uint32_t v;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(v) : "r"(w), "r"(mask), "r"(magic));
  const __half2 o = __hmul2(__hsub2(*reinterpret_cast<const __half2*>(&v), *reinterpret_cast<const __half2*>(&sub)), scale);
  return *reinterpret_cast<const uint32_t*>(&o);
}
// The two blocks of a pair -> the two 16-byte chunks (rows g and g + 8 of the block) of an 8-position chunk.  s[4]: scales of
// row g and of row g + 8, positions 0-7 and 8-15 (a[]) of the first block, b[] of the second.
__device__ __forceinline__ void xt_convert(const DqMagic& k, const XtFields& f, const uint2& w, __half2 a0, __half2 a1, __half2 a2, __half2 a3, __half2 b0,
                                           __half2 b1, __half2 b2, __half2 b3, unsigned char* dst) {
  const uint32_t y = f.nib ? w.y : w.x >> 8, xs = w.x >> f.shift, ys = y >> f.shift;
  *reinterpret_cast<uint4*>(dst) = make_uint4(xt_weight(w.x, f.mlo, k.lo, f.blo, a0), xt_weight(xs, f.mlo, k.lo, f.blo, a2),
                                              xt_weight(y, f.mlo, k.lo, f.blo, b0), xt_weight(ys, f.mlo, k.lo, f.blo, b2));
  *reinterpret_cast<uint4*>(dst + 128) = make_uint4(xt_weight(w.x, f.mhi, k.hi, f.bhi, a1), xt_weight(xs, f.mhi, k.hi, f.bhi, a3),
                                                    xt_weight(y, f.mhi, k.hi, f.bhi, b1), xt_weight(ys, f.mhi, k.hi, f.bhi, b3));
}

struct XtSmem {
  unsigned char* act;     // [2][nchunks][nt rows] canonical K-major, 16-byte chunks
  unsigned char* z;       // 128 rows: [8 epilogue warps][XT_TURN_BYTES]; 64 rows: [2][16 chunks][64 rows]
  unsigned char* ring;    // [2 pipelines][ring][XT_SLOT_BYTES]
  int* prefix;            // [E + 1] items before each expert
  unsigned char* tab;     // [2 items] token-side table of the item's expert (TokTab)
};

__host__ __device__ inline size_t xt_act_bytes(int max_slots, int nt) { return static_cast<size_t>(2) * (max_slots / 8) * xt_chunk_stride(nt); }
__host__ __device__ inline size_t xt_smem_bytes(int max_slots, int num_experts, int tab_bytes, int nt, int rows) {
  size_t o = align_up_c(xt_act_bytes(max_slots, nt), 128) + xt_z_or_turn_bytes(rows);
  o += static_cast<size_t>(2 * xt_ring(rows)) * XT_SLOT_BYTES;
  o += align_up_c(static_cast<size_t>(num_experts + 1) * 4, 128);     // items before each expert
  o += static_cast<size_t>(2) * tab_bytes;
  // the MMAs read 128 operand rows whatever nt is: rows past nt of the last chunk lie in what follows the operand
  return o;
}

// Units of work.  Items that fill whole rounds of the grid are units of their own; the items of the last, partial round
// are cut along the tile columns so that the round's pairs share them evenly (their down sums meet in rank_accum anyway).
struct XtUnits {
  int full, split, per, n_units;
  __device__ __forceinline__ XtUnits(int n_items, int grid, int n_chunks) {
    const int rem = n_items % grid;
    full = n_items - rem;
    split = rem ? grid / rem : 1;
    split = split > n_chunks ? n_chunks : split;
    per = (n_chunks + split - 1) / split;
    split = (n_chunks + per - 1) / per;
    n_units = full + rem * split;
  }
};

struct XtArgs {
  const unsigned char* arena;
  const unsigned char* toktab;
  const __half* h_gate;
  const __half* h_up;
  const int32_t* token_indices;
  const int32_t* expert_offsets;
  const float* route_w;
  float* rank_accum;
  long long* acc64;
  int* status;
  int h_rank, rank_out, T, num_experts, n_tiles, max_slots, nt, tab_bytes;
  int wait_limit_us;
  int vec_add;            // every row of rank_accum starts on a 16-byte boundary (and takes fp32 adds)
};

// Locates unit `u` and copies what the roles need; one warp, an item ahead of the roles.
__device__ __forceinline__ void xt_load_item(XtItem& item, unsigned char* tab, uint64_t* bar, int u, const XtUnits& units, int n_chunks,
                                             const XtSmem& sm, const XtArgs& A, int lane, int rank) {
  int it = u, chunk0 = 0, nchunk = n_chunks;
  if (u >= units.full) {
    const int r = u - units.full, part = r % units.split;
    it = units.full + r / units.split;
    chunk0 = part * units.per;
    nchunk = min(units.per, n_chunks - chunk0);
  }
  int lo = 0, hi = A.num_experts - 1;           // last expert e with prefix[e] <= it
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (sm.prefix[mid] <= it) lo = mid; else hi = mid - 1;
  }
  const int e = lo;
  if (lane == 0) {
    tc::mbar_expect_tx(bar, A.tab_bytes);
    tc::bulk_g2s(tab, A.toktab + static_cast<size_t>(e) * A.tab_bytes, A.tab_bytes, bar);
  }
  // an expert's assignments are spread evenly over its items, an item's over the two CTAs
  const int begin = A.expert_offsets[e], cnt = A.expert_offsets[e + 1] - begin, parts = sm.prefix[e + 1] - sm.prefix[e], j = it - sm.prefix[e];
  int a0 = begin + static_cast<int>(static_cast<int64_t>(cnt) * j / parts);
  const int both = begin + static_cast<int>(static_cast<int64_t>(cnt) * (j + 1) / parts) - a0, first = (both + 1) >> 1;
  const int n = rank ? both - first : first;
  a0 += rank ? first : 0;
  int tk[XT_NT_MAX / 32];
  float rw[XT_NT_MAX / 32];
#pragma unroll
  for (int q = 0; q < XT_NT_MAX / 32; ++q) {
    const int i = lane + 32 * q;
    tk[q] = i < n ? A.token_indices[a0 + i] : -1;
    rw[q] = i < n ? A.route_w[a0 + i] : 0.f;
  }
#pragma unroll
  for (int q = 0; q < XT_NT_MAX / 32; ++q) {
    const bool good = tk[q] >= 0 && tk[q] < A.T;
    item.tok[lane + 32 * q] = good ? tk[q] : 0;
    item.rw[lane + 32 * q] = good ? rw[q] : 0.f;
  }
  if (lane == 0) { item.n = n; item.chunk0 = chunk0; item.nchunk = nchunk; }
}

// One converter stage's words and scales, on their way from L2.
struct XtPre {
  uint2 w[4];
  uint4 s[2];
};

// WIDE: more than 256 row slots a matrix (64 rows); a step then has more stages than the warps can keep apart by their place in it.
template <int ROWS, bool WIDE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(XT_THREADS, 1) experts_tc_kernel(const __grid_constant__ XtArgs A) {
  extern __shared__ __align__(128) unsigned char xt_raw[];
  __shared__ __align__(8) XtBars bars;
  __shared__ XtItem items[2];             // this item and the next one (looked up while this one runs)
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag_s[2];
  volatile int* abort_flag = abort_flag_s;
  const int warp = tc::warp_index(), lane = threadIdx.x & 31;
  const int rank = static_cast<int>(tc::cluster_rank()), pair = static_cast<int>(blockIdx.x) >> 1, n_pairs = static_cast<int>(gridDim.x) >> 1;
  constexpr uint32_t ring = xt_ring(ROWS);
  const int nt = A.nt, h_rank = A.h_rank, num_experts = A.num_experts;
  const int cs = xt_chunk_stride(nt);     // bytes between 8-position chunks of act
  constexpr int D_COLS = xt_down_cols(ROWS);      // of tensor memory per 128-slot tile of the down product
  constexpr int CH = xt_chunk(ROWS), PER_TILE = N_TILE / CH, G_STRIDE = xt_g_stride(ROWS);
  const int n_chunks = A.n_tiles * PER_TILE;
  const uint32_t act_m_bytes = static_cast<uint32_t>(A.max_slots / 8) * cs;
  const TokTab lay(h_rank, A.max_slots);
  XtSmem sm;
  {
    unsigned char* base = xt_raw;
    sm.act = base;
    size_t o = align_up_c(xt_act_bytes(A.max_slots, nt), 128);
    sm.z = base + o; o += xt_z_or_turn_bytes(ROWS);
    sm.ring = base + o; o += static_cast<size_t>(2 * ring) * XT_SLOT_BYTES;
    sm.prefix = reinterpret_cast<int*>(base + o);
    o += align_up_c(static_cast<size_t>(num_experts + 1) * 4, 128);
    sm.tab = base + o;
  }
  if (threadIdx.x == 0) {
    // what the MMA issuers (of the even CTA) wait for is signalled by both CTAs, what waits for MMAs by their commits
    for (int i = 0; i < 2 * XT_RING_MAX; ++i) { tc::mbar_init(&bars.w_full[i], 4); tc::mbar_init(&bars.w_empty[i], 1); }
    tc::mbar_init(&bars.act_ready, 2 * XT_DQ_WARPS);
    tc::mbar_init(&bars.act_free, 2);
    tc::mbar_init(&bars.down_done, 2);
    tc::mbar_init(&bars.down_free, 2 * XT_EPI_WARPS);
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&bars.item_full[i], 2);
      tc::mbar_init(&bars.item_free[i], XT_EPI_WARPS + XT_DQ_WARPS + (rank == 0 ? 2 : 0));
      tc::mbar_init(&bars.gu_done[i], 2);
      tc::mbar_init(&bars.z_ready[i], 2 * XT_EPI_WARPS);
      tc::mbar_init(&bars.z_free[i], 2);
      tc::mbar_init(&bars.drained[i], 1);
    }
    tc::mbar_init_fence();
    abort_flag_s[0] = A.wait_limit_us == 0;
    abort_flag_s[1] = A.wait_limit_us;
  }
  tc::cluster_arrive();
  grid_launch_dependents();
  grid_wait();
  // items before each expert (an item = up to 2 nt consecutive assignments of one expert): every thread loads
  // its experts' counts in parallel, one warp then scans them
  for (int e = threadIdx.x; e < num_experts; e += XT_THREADS) {
    const int o0 = A.expert_offsets[e], o1 = A.expert_offsets[e + 1];
    sm.prefix[e + 1] = (o1 - o0 + 2 * nt - 1) / (2 * nt);
  }
  __syncthreads();
  if (warp == 1) {
    int carry = 0;
    for (int base = 0; base < num_experts; base += 32) {
      const int e = base + lane;
      int v = e < num_experts ? sm.prefix[e + 1] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int n = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += n;
      }
      if (e < num_experts) sm.prefix[e + 1] = carry + v;
      carry += __shfl_sync(0xffffffffu, v, 31);
    }
    if (lane == 0) sm.prefix[0] = 0;
  }
  tc::cluster_wait();                     // both CTAs run and their barriers are set up
  if (warp == 0) tc::tmem_alloc_pair(&tmem_slot, 512);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem_base = tmem_slot;
  const XtUnits units(sm.prefix[num_experts], n_pairs, n_chunks);
  const uint32_t lead_bars = tc::cluster_map(tc::smem_u32(&bars), 0);      // the barriers of the CTA that issues the MMAs
  auto lead = [&](const uint64_t* bar) { return lead_bars + static_cast<uint32_t>(reinterpret_cast<const char*>(bar) - reinterpret_cast<const char*>(&bars)); };
  // tensor memory: two times gate (64 columns) and up (64), then the down product's slot tiles
  const uint32_t d_down = tmem_base + 2 * 2 * XT_ACC;
  constexpr int lag = 1;                  // chunks that the down product of a chunk is issued late

  // The roles run through this CTA's items independently; what they share is guarded by barriers only.  Item number
  // `round` uses description and table buffer round & 1.  After a wait that gave up, every further wait gives up too.
  uint32_t round = 0;
  uint32_t gu_round = 0;    // chunks so far
#define XT_ITEM_BEGIN                                                                                        \
  const uint32_t ib = round & 1u;                                                                            \
  if (!xt_wait(&bars.item_full[ib], (round >> 1) & 1u, abort_flag)) break;                                   \
  const XtItem& item = items[ib];                                                                            \
  const unsigned char* tab = sm.tab + ib * lay.bytes;                                                        \
  const TokTabHead& head = *reinterpret_cast<const TokTabHead*>(tab);                                        \
  const FastExpert& fe = head.fe;                                                                            \
  const int nchunk = item.nchunk;

  if (warp < XT_EPI_WARPS) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(XT_REGS_EPI));
    // -------------------------------------------------------------------- epilogue
    // warp = (TMEM lane quarter q, half of the columns there); a thread owns a token.  128 rows: quarter q is tokens 32 q ..
    // 32 q + 31.  64 rows: lanes 64-127 hold the same tokens as lanes 0-63 and the upper half of every product's columns.
    const int q = warp & 3, half = warp >> 2, upper = ROWS > 64 ? 0 : q >> 1, n0 = 32 * (ROWS > 64 ? q : q & 1), n = n0 + lane;
    const uint32_t lane_sel = static_cast<uint32_t>(32 * q) << 16;
    // four runs of 512 bytes that no other epilogue warp writes
    unsigned char* turn = ROWS > 64 ? sm.z + warp * XT_TURN_BYTES : sm.z + 4 * (2 * upper + half) * XT_Z_STRIDE + n0 * 16;
    constexpr int TURN_STEP = ROWS > 64 ? 512 : XT_Z_STRIDE;
    for (int u = pair; u < units.n_units; u += n_pairs, ++round) {
      XT_ITEM_BEGIN
      const int n_tok = item.n;
      const bool busy = n0 < n_tok;                               // any token in this quarter
      bool ok = true;
      for (int t = 0; t < nchunk && ok; ++t) {
        const uint32_t g = gu_round + t, b = g & 1u;
        ok = xt_wait(&bars.gu_done[b], (g >> 1) & 1u, abort_flag);
        if (!ok) break;
        tc::fence_after_sync();
        if (busy) {
          // z in the contraction order of the down weights (pos32): piece c of eight holds columns 2c, 2c+1, 2c+8, 2c+9 of both
          // of this warp's blocks of 16
          uint32_t zp[16];
          const uint32_t d_gate = tmem_base + 2 * b * XT_ACC + lane_sel + 32 * half, d_up = d_gate + XT_ACC;
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {          // 16 columns at a time: 32 of both would hold 64 registers
            float gv[16], uv[16];
            tc::tmem_ld16(d_gate + 16 * hh, gv);
            tc::tmem_ld16(d_up + 16 * hh, uv);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const __half2 h2 = __floats2half2_rn(silu_mul(gv[2 * i], uv[2 * i]), silu_mul(gv[2 * i + 1], uv[2 * i + 1]));
              zp[4 * (i & 3) + 2 * hh + (i >> 2)] = *reinterpret_cast<const uint32_t*>(&h2);
            }
          }
          if (ROWS > 64) {
            tc::tmem_st16(d_gate, zp);              // over the first half of the gate sums that this warp has read
          } else {
            unsigned char* dst = sm.z + b * XT_Z_BYTES + 4 * (2 * upper + half) * XT_Z_STRIDE + n * 16;
#pragma unroll
            for (int c = 0; c < 4; ++c) *reinterpret_cast<uint4*>(dst + c * XT_Z_STRIDE) = make_uint4(zp[4 * c], zp[4 * c + 1], zp[4 * c + 2], zp[4 * c + 3]);
            tc::fence_async_smem();
          }
        }
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive_cluster(lead(&bars.z_ready[b]));
      }
      gu_round += nchunk;
      if (ok) ok = xt_wait(&bars.down_done, round & 1u, abort_flag);
      if (ok && busy) {
        tc::fence_after_sync();
        const int rank_out = A.rank_out, nslots_d = fe.m[2].nslots;
        const float* s_d = reinterpret_cast<const float*>(tab + lay.s_d);
        const int16_t *rank_d = reinterpret_cast<const int16_t*>(tab + lay.rank_d), *oct_d = reinterpret_cast<const int16_t*>(tab + lay.oct_d);
        const float rw = n < n_tok ? item.rw[n] : 0.f;
        // D_d * s * route weight -> rank_accum.  A thread owns a token: adding straight from the registers would touch a
        // 32-byte sector per lane and instruction.  32 slots of 16 tokens at a time go through shared memory, so that an instruction adds 128 bytes of each of four tokens (128 KB in 5.1 K cycles of an SM, 8.1 K
        // with 64 bytes of eight).  Octets of slots that are not an aligned octet of ranks, rows that do not start on
        // 16-byte boundaries, and the deterministic mode add element by element.
        for (int col = 32 * half; col < XT_MAX_SLOTS; col += ROWS > 64 ? 64 : 128) {
          // 64 rows: 64 columns of a 128-slot tile, which are its lower or its upper slots
          const int s0 = col + 64 * upper;
          if (s0 >= nslots_d) break;
          float v[32];
          tc::tmem_ld32(d_down + lane_sel + (ROWS > 64 ? col : col >> 1 & ~63 | 32 * half), v);
          const bool whole = s0 + 16 < nslots_d;          // the matrix may end after 16 of the 32 slots
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const float4 sv = i < 16 || whole ? *reinterpret_cast<const float4*>(s_d + s0 + i) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[i] *= sv.x * rw; v[i + 1] *= sv.y * rw; v[i + 2] *= sv.z * rw; v[i + 3] *= sv.w * rw;
          }
          // piece c (four slots) of token row r of sixteen, in an order that puts a row's eight pieces into distinct banks
          auto at = [&](int c, int r) { return turn + (c >> 1) * TURN_STEP + (16 * (c & 1) + (r ^ c)) * 16; };
          const int piece = lane & 7, o = piece >> 1;
          const int r0 = A.vec_add && (o < 2 || whole) ? oct_d[(s0 >> 3) + o] : -1;
          const uint32_t odd = __ballot_sync(0xffffffffu, r0 < 0) & 0x55u;      // octets (by their first piece) that go element by element
#pragma unroll
          for (int ph = 0; ph < 2; ++ph) {
            const int first = n0 + 16 * ph, rows = min(16, n_tok - first);
            if (rows <= 0) break;
            __syncwarp();                            // the pieces before have been read
            if ((lane >> 4) == ph) {
#pragma unroll
              for (int c = 0; c < 8; ++c) *reinterpret_cast<float4*>(at(c, lane & 15)) = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
            }
            __syncwarp();
            if (r0 >= 0) {
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const int row = 4 * j + (lane >> 3);
                const float4 x = *reinterpret_cast<const float4*>(at(piece, row));
                if (row < rows)
                  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(A.rank_accum + static_cast<int64_t>(item.tok[first + row]) * rank_out +
                                                                                     r0 + 4 * (piece & 1)),
                               "f"(x.x), "f"(x.y), "f"(x.z), "f"(x.w)
                               : "memory");
              }
            }
            if (odd && (lane & 15) < rows) {          // two lanes a token: the even and the odd octets
              for (int o2 = lane >> 4; o2 < (whole ? 4 : 2); o2 += 2) {
                if (!((odd >> (2 * o2)) & 1u)) continue;
                for (int i = 0; i < 8; ++i) {
                  const int r = rank_d[s0 + 8 * o2 + i];
                  if (r >= 0)
                    acc_add(A.rank_accum, A.acc64, static_cast<int64_t>(item.tok[first + (lane & 15)]) * rank_out + r,
                            *reinterpret_cast<const float*>(at(2 * o2 + (i >> 2), lane & 15) + 4 * (i & 3)));
                }
              }
            }
          }
        }
        tc::fence_before_sync();
        tc::fence_async_smem();
      }
      __syncwarp();
      if (lane == 0) { tc::mbar_arrive_cluster(lead(&bars.down_free)); tc::mbar_arrive(&bars.item_free[ib]); }
      if (!ok) break;
    }
  } else if (warp < XT_DQ_WARP0 + XT_DQ_WARPS) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(XT_REGS_DQ));
    // -------------------------------------------------------------------- activation operand and converters
    // Team 0 (six warps) feeds pipeline 0, team 1 pipeline 1.  Step t of an item is `n` stages of a team: a stage per two pairs
    // of blocks (64 rows: per pair) of chunk t's gate (up) product, then a stage (64 slots x 32 columns) per 32 columns and
    // 128-slot tile of chunk t - lag's down product; stages 2 i and 2 i + 1 share a ring slot.  Warp w of the team takes stages w,
    // w + 6, ... of every step: at 256 slots a matrix and 128 rows that is one stage, the same of every chunk, whose addresses and
    // kinds of words are worked out once per item.  A stage is four 16 x 32 blocks; lane (g, t4) turns its words of each into two
    // 16-byte pieces.
    const int dw = warp - XT_DQ_WARP0;
    const int team = dw / XT_TEAM, wt = dw - team * XT_TEAM, g = lane >> 2, t4 = lane & 3;
    uint64_t* w_empty = &bars.w_empty[team * ring];
    const uint32_t w_full = lead(&bars.w_full[team * ring]);
    unsigned char* ring0 = sm.ring + team * ring * XT_SLOT_BYTES;
    const DqMagic magic;
    uint32_t item_seq = 0;                    // ring slots that the pipeline has used before this item
    uint32_t seen = 0;                        // every use of a slot before this one is known to be multiplied
    for (int u = pair; u < units.n_units; u += n_pairs, ++round) {
      XT_ITEM_BEGIN
      if (round > 0 && !xt_wait(&bars.act_free, (round - 1) & 1u, abort_flag)) break;
      {
        // act[m][chunk][n] = 8 consecutive contraction positions of token n: fp16(h[token, rank(slot)] * s(slot)).
        // A warp takes tokens; a lane owns an octet of ranks, which the arena layout keeps together: one 16-byte load, four
        // multiplications, one 16-byte store (pieces of one row are 16 bytes apart modulo 128: no bank conflicts).  Octets
        // that straddle two groups of rows follow rank by rank.  Operand rows past the item's tokens keep whatever they
        // hold: they only reach accumulator rows that nobody reads.
        const int n_tok = item.n, n_oct = h_rank >> 3;
        const int16_t* pos_r = reinterpret_cast<const int16_t*>(tab + lay.pos_r);
        const __half* s_r = reinterpret_cast<const __half*>(tab + lay.s_r);
        const int16_t* oct_r = reinterpret_cast<const int16_t*>(tab + lay.oct_r);
        for (int o0 = 0; o0 < n_oct; o0 += 32) {
          const int o = o0 + lane;
          int dst[2];
          uint4 sc[2];
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            const int c = o < n_oct ? oct_r[m * n_oct + o] : -1;
            dst[m] = c < 0 ? -1 : static_cast<int>(m * act_m_bytes) + c * cs;
            sc[m] = c < 0 ? make_uint4(0u, 0u, 0u, 0u) : *reinterpret_cast<const uint4*>(s_r + m * h_rank + 8 * o);
          }
          for (int n0 = dw; n0 < n_tok; n0 += 4 * XT_DQ_WARPS) {
            uint4 hv[4][2];                     // four tokens per round: eight loads in flight per lane
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int n = min(n0 + j * XT_DQ_WARPS, n_tok - 1);
              const int64_t row = static_cast<int64_t>(item.tok[n]) * h_rank + 8 * o;
#pragma unroll
              for (int m = 0; m < 2; ++m)
                if (dst[m] >= 0) hv[j][m] = __ldg(reinterpret_cast<const uint4*>((m ? A.h_up : A.h_gate) + row));
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int n = n0 + j * XT_DQ_WARPS;
              if (n >= n_tok) break;
#pragma unroll
              for (int m = 0; m < 2; ++m)
                if (dst[m] >= 0) {
                  uint4 r;
                  const __half2 *hp = reinterpret_cast<const __half2*>(&hv[j][m]), *sp = reinterpret_cast<const __half2*>(&sc[m]);
                  __half2* rp = reinterpret_cast<__half2*>(&r);
#pragma unroll
                  for (int k = 0; k < 4; ++k) rp[k] = __hmul2(hp[k], sp[k]);       // one rounding of the exact product
                  *reinterpret_cast<uint4*>(sm.act + dst[m] + n * 16) = r;
                }
            }
          }
        }
        const int tid_s = threadIdx.x - XT_DQ_WARP0 * 32;
        for (int m = 0; m < 2; ++m)
          for (int w = 0; w < (n_oct + 31) >> 5; ++w)
            for (uint32_t left = head.broken[m][w]; left; left &= left - 1) {
              const int o = 32 * w + __ffs(left) - 1;
              for (int i = tid_s; i < 8 * n_tok; i += XT_DQ_WARPS * 32) {
                const int n = i >> 3, rk = 8 * o + (i & 7), pos = pos_r[m * h_rank + rk];
                if (pos >= 0)
                  *reinterpret_cast<__half*>(sm.act + m * act_m_bytes + (pos >> 3) * cs + (pos & 7) * 2 + n * 16) =
                      __hmul((m ? A.h_up : A.h_gate)[static_cast<int64_t>(item.tok[n]) * h_rank + rk], s_r[m * h_rank + rk]);
              }
            }
        // Slots that the octets above do not reach.  Padding: the weights are zero, the activations have to be finite.  A
        // rank that several slots hold: each slot has weights and a factor of its own.
        if (head.loose) {
          for (int m = 0; m < 2; ++m) {
            const int nslots = fe.m[m].nslots;
            const int16_t* rank_t = reinterpret_cast<const int16_t*>(A.arena + fe.m[m].tab_off);
            const __half* s_t = reinterpret_cast<const __half*>(rank_t + nslots);
            for (int i = dw; i < nslots; i += XT_DQ_WARPS) {
              const int rk = rank_t[i], pos = slot_pos(i);
              const bool live = rk >= 0 && rk < h_rank;
              if (live && pos_r[m * h_rank + rk] == pos) continue;
              const __half sv = live ? s_t[i] : __float2half(0.f);
              for (int n = lane; n < n_tok; n += 32)
                *reinterpret_cast<__half*>(sm.act + m * act_m_bytes + (pos >> 3) * cs + (pos & 7) * 2 + n * 16) =
                    live ? __hmul((m ? A.h_up : A.h_gate)[static_cast<int64_t>(item.tok[n]) * h_rank + rk], sv) : sv;
            }
          }
        }
        // Every ring slot of the item before is multiplied; known before this item may begin, for the parities' sake (see acquire).
        if (round > 0 && !xt_wait(&bars.down_done, (round - 1) & 1u, abort_flag)) break;
        seen = item_seq;
        tc::fence_async_smem();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive_cluster(lead(&bars.act_ready));
      }
      // everything about the expert in registers: the barriers' memory clobbers would have it read again every stage
      const int chunk0 = item.chunk0, nblk_d = fe.m[2].nslots >> 4, n_mt = (nblk_d + 7) >> 3;
      const int npairs = fe.m[team].nslots >> 5, nib_pairs = fe.m[team].nblk[0] >> 1, nib_d = fe.m[2].nblk[0];
      constexpr int GP = ROWS > 64 ? 2 : 1, DS = CH / 32;       // pairs of a gate/up stage, stages of a down tile
      const int slots_gu = (npairs + 2 * GP - 1) / (2 * GP), slots_d = ((n_mt - team + 1) >> 1) * (DS / 2), per_step = slots_gu + slots_d;
      const int unit_bytes = fe.unit_bytes;
      const unsigned char* unit0 = A.arena + fe.unit_base;
      const int scale_gu = fe.sec_off[team] + t4 * 16, words_gu = fe.sec_off[3 + team], scale_d = fe.sec_off[2] + g * 4, words_d = fe.sec_off[5];
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&bars.item_free[ib]);
      // A stage: `kind` bit p: words of pair p (down: of block p) are nibbles; `live`: its pairs (blocks); offsets of its words and
      // scales in the unit block and of its pieces in a ring slot.
      struct Stage { int kind, live, w_off[2], s_off, dst_off; bool gu; };
      auto describe = [&](int i) -> Stage {
        Stage st;
        st.gu = i < 2 * slots_gu;
        if (st.gu) {
          st.live = min(GP, npairs - GP * i);    // an odd last stage has an empty partner in its slot
          st.s_off = scale_gu + GP * i * 64;
          st.kind = 0;
#pragma unroll
          for (int p = 0; p < GP; ++p) {
            const int pr = GP * i + p;
            const bool nib = pr < nib_pairs;
            st.kind |= nib ? 1 << p : 0;
            st.w_off[p] = words_gu + (nib ? pr * 2048 + 4 / GP * rank * 256 + lane * 8 : nib_pairs * 2048 + (pr - nib_pairs) * 1024 + 4 / GP * rank * 128 + lane * 4);
          }
          st.dst_off = (i & 1) * 4 * GP * G_STRIDE + t4 * G_STRIDE + g * 16;
        } else {
          const int j = i - 2 * slots_gu, mb0 = 8 * (team + 2 * (j / DS)) + 4 * rank, pr = j % DS;
          st.live = min(4, nblk_d - mb0);        // blocks; slots past the matrix: accumulator columns that nobody reads
          st.kind = (1 << min(max(nib_d - mb0, 0), 4)) - 1;
          st.s_off = scale_d + mb0 * 32;
          st.w_off[0] = words_d + (mb0 * 4 + pr) * 256 + lane * 8;                                              // of a nibble block
          st.w_off[1] = words_d + nib_d * 1024 + ((mb0 - nib_d) * 4 + pr) * 128 + lane * 4;                     // of a dense block
          st.dst_off = (j & 1) * 4 * XT_D_STRIDE + t4 * XT_D_STRIDE + g * 16;
        }
        return st;
      };
      // its words and scales of chunk `c` of the item, whatever their kinds
      auto fetch = [&](const Stage& st, int c, XtPre& p) {
        const int ch = chunk0 + c, odd = ch % PER_TILE;
        const unsigned char* b = unit0 + static_cast<int64_t>(ch / PER_TILE) * unit_bytes;
        if (st.gu) {
#pragma unroll
          for (int q = 0; q < GP; ++q) {
            if (q >= st.live) break;
            p.s[q] = __ldg(reinterpret_cast<const uint4*>(b + st.s_off + q * 64));
            if (st.kind & (1 << q)) {
              const uint2* w = reinterpret_cast<const uint2*>(b + st.w_off[q] + odd * 1024);
#pragma unroll
              for (int x = 0; x < 4 / GP; ++x) p.w[4 / GP * q + x] = __ldg(w + 32 * x);
            } else {
              const uint32_t* w = reinterpret_cast<const uint32_t*>(b + st.w_off[q] + odd * 512);
#pragma unroll
              for (int x = 0; x < 4 / GP; ++x) p.w[4 / GP * q + x].x = __ldg(w + 32 * x);
            }
          }
        } else {
          uint32_t* ps = reinterpret_cast<uint32_t*>(p.s);
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            if (v >= st.live) break;
            ps[v] = __ldg(reinterpret_cast<const uint32_t*>(b + st.s_off + v * 32));
            if (st.kind & (1 << v)) p.w[v] = __ldg(reinterpret_cast<const uint2*>(b + st.w_off[0] + odd * 512 + v * 1024));
            else p.w[v].x = __ldg(reinterpret_cast<const uint32_t*>(b + st.w_off[1] + odd * 256 + v * 512));
          }
        }
      };
      auto convert = [&](const Stage& st, const XtPre& p, unsigned char* dst) {
        if (st.gu) {
#pragma unroll
          for (int q = 0; q < GP; ++q) {
            if (q >= st.live) break;
            const __half2* sp = reinterpret_cast<const __half2*>(&p.s[q]);
            const XtFields f(st.kind & (1 << q));
#pragma unroll
            for (int x = 0; x < 4 / GP; ++x)
              xt_convert(magic, f, p.w[4 / GP * q + x], sp[0], sp[0], sp[1], sp[1], sp[2], sp[2], sp[3], sp[3], dst + q * 4 * G_STRIDE + x * 256);
          }
        } else {
          const __half2* sp = reinterpret_cast<const __half2*>(p.s);
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            if (v >= st.live) break;
            const __half2 lo = __low2half2(sp[v]), hi = __high2half2(sp[v]);
            xt_convert(magic, XtFields(st.kind & (1 << v)), p.w[v], lo, hi, lo, hi, lo, hi, lo, hi, dst + v * 256);
          }
        }
      };
      // The use `seq` of a ring slot may begin once use seq - ring is multiplied.  The parity of the slot's barrier tells that
      // from the use before only if the warp knows use seq - 2 ring to be multiplied: a warp's uses lie at most a ring apart,
      // and the first one of an item less than two rings behind the last one of the item before.
      auto acquire = [&](uint32_t seq) -> bool {
        if (static_cast<int>(seq - seen) < static_cast<int>(ring)) return true;
        const uint32_t before = seq - ring;
        seen = before + 1;
        return xt_wait(&w_empty[before % ring], (before / ring) & 1u, abort_flag);
      };
      // Stage i of step t.  Up to 256 slots a warp takes the same stages of every step (the ring covers what lies between them),
      // so that one which takes a single stage describes it once; beyond, the item's stages in turn, three ring slots apart.
      bool ok = true;
      int i = WIDE ? wt - XT_TEAM : wt, t = 0;
      auto step = [&]() -> bool {
        if (WIDE) {
          i += XT_TEAM - (t == nchunk ? 2 * slots_gu : 0);
          for (int nt = 0; t < nchunk + lag; ++t, i -= nt) {
            nt = (t < nchunk ? 2 * slots_gu : 0) + (t >= lag ? 2 * slots_d : 0);
            if (i < nt) break;
          }
          if (t == nchunk) i += 2 * slots_gu;
        } else {
          do {
            i += XT_TEAM;
            if (i >= 2 * per_step) { i = wt; ++t; }
          } while (t < nchunk + lag && !(i < 2 * slots_gu ? t < nchunk : t >= lag));
        }
        return t < nchunk + lag;
      };
      XtPre p;
      Stage st;
      bool more = WIDE ? step() : i < 2 * per_step && (i < 2 * slots_gu || step());
      if (more) {
        st = describe(i);
        fetch(st, st.gu ? t : t - lag, p);
      }
      while (more) {
        // the use of a ring slot that this stage fills: steps before t, then this step's order (the last one has no gate / up)
        const uint32_t pos = item_seq + t * per_step - (t > 0 ? slots_d : 0) + (i >> 1) - (t == nchunk ? slots_gu : 0);
        if (!(ok = acquire(pos))) break;
        convert(st, p, ring0 + (pos % ring) * XT_SLOT_BYTES + st.dst_off);
        const int i_was = i;
        more = step();
        if (more) {
          if (i != i_was) st = describe(i);
          fetch(st, st.gu ? t : t - lag, p);      // on its way while the converted stage is published and the next one is waited for
        }
        tc::fence_async_smem();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive_cluster(w_full + (pos % ring) * 8);
      }
      item_seq += nchunk * per_step;
      if (!ok) break;
    }
  } else {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(XT_REGS_MISC));
  if (warp == XT_LOOKUP_WARP) {
    // -------------------------------------------------------------------- descriptions, an item ahead of the roles
    for (int u = pair; u < units.n_units; u += n_pairs, ++round) {
      const uint32_t ib = round & 1u;
      if (round >= 2 && !xt_wait(&bars.item_free[ib], ((round >> 1) - 1) & 1u, abort_flag)) break;
      xt_load_item(items[ib], sm.tab + ib * lay.bytes, &bars.item_full[ib], u, units, n_chunks, sm, A, lane, rank);
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&bars.item_full[ib]);
      // the copy lands whatever the other roles do: waited for also when one of them has given up
      if (!tc::mbar_wait(&bars.item_full[ib], (round >> 1) & 1u)) { xt_give_up(abort_flag); break; }
      // the weights on their way to L2, one tile per lane, every other one by this CTA (sizes and offsets are multiples of 16 bytes)
      const FastExpert& fe = reinterpret_cast<const TokTabHead*>(sm.tab + ib * lay.bytes)->fe;
      const int t0 = items[ib].chunk0 / PER_TILE, t1 = (items[ib].chunk0 + items[ib].nchunk + PER_TILE - 1) / PER_TILE;
      for (int t = t0 + 2 * lane + rank; t < t1; t += 64)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(A.arena + fe.unit_base + static_cast<int64_t>(t) * fe.unit_bytes),
                     "r"(fe.unit_bytes)
                     : "memory");
      __syncwarp();
    }
  } else if (warp < XT_MMA_WARP0 + 2 && rank == 0) {
    // -------------------------------------------------------------------- MMA issue for both CTAs, one thread per pipeline
    // The whole warp waits (a lone waiting lane wakes up several times slower); one issues.
    const int pl = warp - XT_MMA_WARP0;
    const uint32_t idesc_gu = tc::idesc_f16(2 * ROWS, CH), idesc_d = tc::idesc_f16(2 * ROWS, 128);
    // descriptors: constant upper part, start-address field advanced per block
    const uint64_t a_desc = tc::smem_desc_kmajor(tc::smem_u32(sm.act) + pl * act_m_bytes, cs, 128);
    const uint32_t ring0 = tc::smem_u32(sm.ring) + pl * ring * XT_SLOT_BYTES;
    const uint64_t gu_desc = tc::smem_desc_kmajor(ring0, G_STRIDE, 128), dn_desc = tc::smem_desc_kmajor(ring0, XT_D_STRIDE, 128);
    uint64_t* w_full = &bars.w_full[pl * ring];
    uint64_t* w_empty = &bars.w_empty[pl * ring];
    const uint32_t a_step = (2 * cs) >> 4;       // descriptor units per 16 contraction positions
    const uint64_t z_desc = tc::smem_desc_kmajor(tc::smem_u32(sm.z), XT_Z_STRIDE, 128);
    uint32_t seq = 0;                            // uses of ring slots so far
    for (int u = pair; u < units.n_units; u += n_pairs, ++round) {
      XT_ITEM_BEGIN
      const int npairs = fe.m[pl].nslots >> 5, n_mt = ((fe.m[2].nslots >> 4) + 7) >> 3;   // 128-slot tiles of the down product (<= 3)
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&bars.item_free[ib]);
      bool ok = xt_wait(&bars.act_ready, round & 1u, abort_flag);
      tc::fence_after_sync();
      for (int t = 0; t < nchunk + lag && ok; ++t) {
        if (t < nchunk) {
          const uint32_t g = gu_round + t, b = g & 1u, k = g >> 1;
          if (k >= 1) ok = xt_wait(&bars.z_free[b], (k - 1) & 1u, abort_flag);     // the z written over this accumulator is multiplied
          tc::fence_after_sync();
          const uint32_t d_acc = tmem_base + (2 * b + pl) * XT_ACC;
          uint64_t ad = a_desc;
          constexpr int SP = ROWS > 64 ? 4 : 2;       // pairs of a slot
          for (int pr = 0; pr < npairs && ok; pr += SP, ++seq) {
            const uint32_t sl = seq % ring;
            if (!(ok = xt_wait(&w_full[sl], (seq / ring) & 1u, abort_flag))) break;
            if (tc::elect_one()) {
              const uint64_t bd = gu_desc + ((sl * XT_SLOT_BYTES) >> 4);
#pragma unroll
              for (int h = 0; h < 2 * SP; ++h)    // 16 slots each
                if (h < 2 || pr + (h >> 1) < npairs)
                  tc::mma_f16_pair(d_acc, ad + h * a_step, bd + ((h * 2 * G_STRIDE) >> 4), idesc_gu, pr > 0 || h > 0 ? 1u : 0u);
              tc::mma_commit_pair(&w_empty[sl]);
            }
            __syncwarp();
            ad += 2 * SP * a_step;
          }
          if (!ok) break;
          if (tc::elect_one()) {
            tc::mma_commit_pair(&bars.gu_done[b]);
            if (t == nchunk - 1) tc::mma_commit_pair(&bars.act_free);
          }
          __syncwarp();
        }
        if (t >= lag) {
          const uint32_t g = gu_round + t - lag, b = g & 1u;
          if (t == lag && round > 0) ok = xt_wait(&bars.down_free, (round - 1) & 1u, abort_flag);   // the last item's sums are read out
          if (ok) ok = xt_wait(&bars.z_ready[b], (g >> 1) & 1u, abort_flag);
          tc::fence_after_sync();
          const uint32_t d_z = tmem_base + 2 * b * XT_ACC;      // columns 0-31 of the chunk, and 32-63 32 columns on
          for (int mt = pl; mt < n_mt && ok; mt += 2)
            for (int kp = 0; kp < CH / 64; ++kp, ++seq) {      // 64 columns of z per slot
              const uint32_t sl = seq % ring;
              if (!(ok = xt_wait(&w_full[sl], (seq / ring) & 1u, abort_flag))) break;
              if (tc::elect_one()) {
                const uint64_t bd = dn_desc + ((sl * XT_SLOT_BYTES) >> 4);
#pragma unroll
                for (int h = 0; h < 4; ++h) {         // 16 columns of z each
                  const uint32_t add = t > lag || kp > 0 || h > 0 ? 1u : 0u;
                  if (ROWS > 64)
                    tc::mma_f16_pair_ta(d_down + mt * D_COLS, d_z + 32 * (h >> 1) + 8 * (h & 1), bd + ((h * 2 * XT_D_STRIDE) >> 4), idesc_d, add);
                  else
                    tc::mma_f16_pair(d_down + mt * D_COLS, z_desc + ((b * XT_Z_BYTES + (4 * kp + h) * 2 * XT_Z_STRIDE) >> 4), bd + ((h * 2 * XT_D_STRIDE) >> 4), idesc_d, add);
                }
                tc::mma_commit_pair(&w_empty[sl]);
              }
              __syncwarp();
            }
          if (ok && tc::elect_one()) {
            tc::mma_commit_pair(&bars.z_free[b]);
            if (t == nchunk + lag - 1) tc::mma_commit_pair(&bars.down_done);
          }
          __syncwarp();
        }
      }
      gu_round += nchunk;
      if (!ok) break;
    }
    if (tc::elect_one()) tc::mma_commit_pair(&bars.drained[pl]);
    __syncwarp();
  }
  }
  // Every role of both CTAs comes here on its own, also when a wait gave up.  Nothing of the pair is in flight behind the
  // last commits, and neither CTA leaves while the other may still signal its barriers.
  tc::fence_before_sync();
  __syncthreads();
  if (warp == XT_MMA_WARP0)
    for (int i = 0; i < 2; ++i)
      if (!tc::mbar_wait(&bars.drained[i], 0)) xt_give_up(abort_flag);
  tc::cluster_arrive();
  tc::cluster_wait();
  if (warp == 0) tc::tmem_dealloc_pair(tmem_base, 512);
  if (threadIdx.x == 0 && *abort_flag) atomicExch(A.status, BM_ERR_TIMEOUT);
#undef XT_ITEM_BEGIN
}

// Item size and ring depth for a layer: the first candidate whose activation operand (2 KB per token at 256 row slots per
// matrix) and stages fit shared memory.  Tensor memory holds two gate/up buffers of 128 columns and 128 (64 rows: 64) per 128 slots of
// the down product: with 128 rows up to 256 slots.
struct XtPlan { int nt; size_t smem; };
constexpr size_t XT_SMEM_LIMIT = 227 * 1024 - 3072;     // dynamic part: the static part (two item descriptions, barriers) stays below 3 KB
static bool xt_plan(const bm_layer* L, int rows, XtPlan* out) {
  if (!L->toktab_dev || L->num_experts > XT_MAX_E || L->intermediate % N_TILE != 0 || L->max_slots > XT_MAX_SLOTS) return false;
  if (2 * 2 * XT_ACC + (L->max_slots + 127) / 128 * xt_down_cols(rows) > 512) return false;      // columns of tensor memory
  for (int nt = rows; nt >= 16; nt -= 16) {
    const size_t smem = xt_smem_bytes(L->max_slots, L->num_experts, TokTab(L->rank_in, L->max_slots).bytes, nt, rows);
    if (smem <= XT_SMEM_LIMIT) {
      *out = XtPlan{nt, smem};
      return true;
    }
  }
  return false;
}

// Whether the layer's largest expert fits the tensor path's shared- and tensor-memory budget (AUTO falls back to the
// decode path otherwise).
bool experts_tc_fits(const bm_layer* L) {
  XtPlan p;
  return xt_plan(L, 64, &p) || xt_plan(L, 128, &p);
}

// The stage as a model, us: the tiles and units of the pair with the most, items of `2 nt` assignments spread evenly.  Fits to thirteen layer shapes (8
// to 512 experts, 4 to 16 tiles, rank 128 to 384) at 17 to 180 assignments an expert, off by 4 %.
static double xt_us(const bm_layer* L, int rows, int nt, double load) {
  const int pairs = L->sms / 2, items = std::max(1, expected_passes(L->num_experts, load, 2 * nt)), rest = items % pairs, full = items / pairs;
  const int split = rest ? std::min(L->n_tiles, pairs / rest) : 1, last = rest ? (L->n_tiles + split - 1) / split : 0;
  const double tiles = full * L->n_tiles + last, more = full - (rest == 0), slots = L->max_slots / 256.0;
  if (L->max_slots > 256) return 14.7 + 3.6 * tiles + 2.6 * more;
  return rows == 64 ? 11.9 + (0.9 + 1.3 * slots) * tiles + 3.1 * more : 14.4 + (1.1 + 1.55 * slots) * tiles + 5.8 * more;
}
// Rows of a CTA for this load.  More than 256 slots: always 64 (128 experts of 6 tiles and rank 384, 32 assignments each 57 us against 89 with 128
// rows, which left tensor memory for one pair of accumulators only; 128 each 96 / 94; 256 each 142 / 158).  Else the smaller estimate: with 64 rows
// an item is half as large and a quarter cheaper, so that they pay until many experts need a second one.  us with 64 / with 128: 128 experts of 6 tiles,
// 64 each 41 / 51, 120 each 48 / 53, 128 each 58 / 52, 150 each 66 / 53, 256 each 84 / 74; 512 of 4 tiles, 108 each 99 / 125, 136 each 153 / 126; 64 of 11 tiles
// and rank 128, 112 each 31 / 35, 128 each 41 / 35.  Under skewed loads the two are 3 % apart between 100 and
// 150 each, 64 rows ahead where experts are few (hence the 8 %).
static int xt_rows(const bm_layer* L, double load, double* us) {
  XtPlan few, many;
  const bool fits = xt_plan(L, 64, &few);
  const double t64 = fits ? xt_us(L, 64, few.nt, load) : 0.0;
  if (fits && L->max_slots > 256) { *us = t64; return 64; }
  const double t128 = xt_plan(L, 128, &many) ? xt_us(L, 128, many.nt, load) : std::numeric_limits<double>::infinity();
  const bool take64 = fits && t64 <= 1.08 * t128;
  *us = take64 ? t64 : t128;
  return take64 ? 64 : 128;
}
double experts_tc_us(const bm_layer* L, double load, int* rows) {
  double us;
  *rows = xt_rows(L, load, &us);
  return us;
}

template <int ROWS, bool WIDE>
static int xt_launch(XtArgs a, size_t smem, cudaStream_t st) {
  static PerDeviceOnce once;
  static int grids[MAX_DEVICES];
  int dev = -1;
  BM_CUDA(cudaGetDevice(&dev));
  BM_REQUIRE(dev >= 0 && dev < MAX_DEVICES, BM_ERR_UNSUPPORTED, "experts_tc: device ordinal %d out of range", dev);
  if (!once.is_done(dev)) {
    BM_CUDA(cudaFuncSetAttribute(experts_tc_kernel<ROWS, WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(XT_SMEM_LIMIT)));
    BM_CUDA(cudaDeviceGetAttribute(&grids[dev], cudaDevAttrMultiProcessorCount, dev));
    grids[dev] &= ~1;
    cudaFuncAttributes fa;
    BM_CUDA(cudaFuncGetAttributes(&fa, experts_tc_kernel<ROWS, WIDE>));
    BM_REQUIRE(fa.numRegs >= XT_REGS, BM_ERR_UNSUPPORTED, "experts_tc: built with %d registers per thread, %d expected", fa.numRegs, XT_REGS);
    once.mark(dev);
  }
  BM_CUDA(launch_after(AFTER_READS, /*cluster: the kernel's own*/ 1, experts_tc_kernel<ROWS, WIDE>, dim3(grids[dev]), XT_THREADS, smem, st, a));
  BM_LAUNCH_CHECK("experts_tc_kernel");
  return BM_OK;
}

int launch_experts_tc(const bm_layer* L, const __half* h_gate, const __half* h_up, const int32_t* token_indices,
                      const int32_t* expert_offsets, const float* route_w, int T, int expected_assign, int rows, float* rank_accum, long long* acc64,
                      cudaStream_t st) {
  BM_REQUIRE(L->num_experts <= XT_MAX_E, BM_ERR_UNSUPPORTED, "experts_tc: more than %d experts", XT_MAX_E);
  BM_REQUIRE(L->intermediate % N_TILE == 0, BM_ERR_UNSUPPORTED, "experts_tc: intermediate size must be a multiple of %d", N_TILE);
  BM_REQUIRE(L->max_slots <= XT_MAX_SLOTS, BM_ERR_UNSUPPORTED, "experts_tc: %d row slots exceed the tensor-memory budget", L->max_slots);
  BM_REQUIRE(L->rank_in % 8 == 0 && ((reinterpret_cast<uintptr_t>(h_gate) | reinterpret_cast<uintptr_t>(h_up)) & 15u) == 0,
             BM_ERR_UNSUPPORTED, "experts_tc: rank-space rows must be 16-byte aligned (rank %d)", L->rank_in);
  double us;
  if (rows == 0) rows = xt_rows(L, static_cast<double>(expected_assign) / L->num_experts, &us);
  XtPlan plan;
  BM_REQUIRE(xt_plan(L, rows, &plan), BM_ERR_UNSUPPORTED, "experts_tc: the layer's largest expert does not fit in shared memory");
  XtArgs a{};
  a.toktab = L->toktab_dev;
  a.tab_bytes = TokTab(L->rank_in, L->max_slots).bytes;
  a.arena = static_cast<const unsigned char*>(L->arena);
  a.h_gate = h_gate; a.h_up = h_up; a.h_rank = L->rank_in;
  a.token_indices = token_indices; a.expert_offsets = expert_offsets; a.route_w = route_w;
  a.rank_accum = rank_accum; a.acc64 = acc64; a.status = L->status_dev;
  // an octet's two 16-byte adds need the row's start, and so rank_out and the base, at multiples of four floats
  a.vec_add = acc64 == nullptr && L->rank_out % 4 == 0 && (reinterpret_cast<uintptr_t>(rank_accum) & 15u) == 0;
  a.wait_limit_us = L->wait_limit_us;
  a.rank_out = L->rank_out; a.T = T; a.num_experts = L->num_experts; a.n_tiles = L->n_tiles; a.max_slots = L->max_slots;
  a.nt = plan.nt;
  if (L->max_slots > 256) return xt_launch<64, true>(a, plan.smem, st);
  return rows > 64 ? xt_launch<128, false>(a, plan.smem, st) : xt_launch<64, false>(a, plan.smem, st);
}

}  // namespace bm
