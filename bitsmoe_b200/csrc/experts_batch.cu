// Packed routed-expert forward for batches of some tokens per expert: weights on the tensor cores (mma.sync) with 16 tokens a pass.
//
// Work unit = (expert, pass of up to 16 of its assignments, range of its 128-column tiles); passes that fill whole rounds of the
// grid (two CTAs an SM) are units of their own, those of the last, partial round are cut along the tiles, evenly.  A unit gathers its
// tokens' rows once into the operand hs = fp16(h[rank] * s) (16-byte octets, as the tensor path stages them).  Per tile the eight
// warps turn the section's words into A fragments -- fp16(q * scale), the very weights the tensor path multiplies -- for two
// blocks of eight tokens: gate and up into z = silu(g) * u (shared memory), one barrier, down into accumulators that stay in
// registers to the end of the unit and leave as one fp32 atomic per (slot, token).  One thread copies the sections a ring ahead
// (cp.async.bulk); the tile's barrier says which slots are free, so there is no producer warp and a thread has 128 registers.
//
// What bounds it: issue slots.  Turning a word into fp16(q * scale) takes 3.5 instructions for two codes and mma.sync holds a
// scheduler 8.5 cycles, which do not overlap: a tile costs an SM 2.7 K cycles and 0.8 K for every eight tokens (gate and up 1.9 K of
// them at 16).  The decode kernel (experts_decode.cu), with less work per code and its weights' scale in the operand, takes 2.8 K
// with eight tokens, but a second pass doubles that.  128 tokens on 128 experts of six tiles (8 each) 31.1 -> 22.7 us, 64 experts of
// eleven tiles 31.3 -> 22.7.  The stage takes as long as its longest CTA, 7.3 us and 5.2 a tile; a second unit costs 4.8 (operand, sums, the way
// through the ring).  148 passes on 296 CTAs leave a CTA three of six tiles (22.9 us); cut by an integer quotient 149 to 295 left one all six
// (37.7), in even shares 149 to 197 passes take 28 to 31 us, 198 to 246 36, and behind whole rounds 445 64 instead of 70.  203 tokens are 145 +- 3
// passes, one load in eight more than 148.
// Measured and not taken: 32 tokens a pass (203 tokens 33 us, 256 tokens 33 against 39, skewed 300 tokens 53 against 39), a third CTA
// per SM (80 registers: 203 tokens 27.5), the scale in the operand instead of the weights (203 tokens 27).  Against 64 bits the stage
// is off by 4.2e-4 (203 tokens; the decode kernel by 4.7e-4, whose operand is rounded twice).
//
// Every wait is bounded; one that gives up raises a flag, the warps agree at the next barrier to leave, and the status word reports
// BM_ERR_TIMEOUT behind the copies under way.
#include "dequant.cuh"
#include "tc05.cuh"

namespace bm {

constexpr int BT_THREADS = 256, BT_WARPS = 8;
constexpr int BT_MAX_E = 1024;                 // four experts a thread in the prefix of passes
constexpr int BT_MAX_RING = 6;                 // section slots
constexpr int BT_NP = 2, BT_NT = 8 * BT_NP;    // blocks of eight tokens, tokens of a pass
constexpr uint64_t BT_DRAIN_LIMIT_NS = 100000000;

// Dynamic shared memory of one CTA (bytes)
struct BtLayout {
  int ring, hs, z, tab, soff, pbase, total;
  int hs_row, hs_m, z_buf;                     // a token's row, a matrix, a buffer
};
__host__ __device__ inline BtLayout bt_layout(int max_slots, int sec_bytes, int ring, int num_experts, int tab_bytes) {
  BtLayout L;
  L.hs_row = (max_slots + 63) / 64 * 128;      // whole groups of eight 16-byte pieces: bt_piece permutes inside them
  L.hs_m = BT_NT * L.hs_row;
  L.z_buf = BT_NT * N_TILE * 2;
  int o = 0;
  L.ring = o;  o += ring * sec_bytes;
  L.hs = o;    o += 2 * L.hs_m;
  L.z = o;     o += 2 * L.z_buf;
  L.tab = o;   o += 2 * static_cast<int>(align_up_c(static_cast<size_t>(tab_bytes), 128));
  L.soff = o;  o += static_cast<int>(align_up_c(static_cast<size_t>(num_experts + 1) * 4, 16));
  L.pbase = o; o += static_cast<int>(align_up_c(static_cast<size_t>(num_experts + 4) * 4, 16));
  L.total = o;
  return L;
}
// Whether a last round of `all` tiles is handed out in even shares: where the longest one is shorter than `per`, the tiles of a pass's part.
__host__ __device__ __forceinline__ bool bt_even_shares(int all, int per, int grid) { return all <= (per - 1) * grid; }
// a / b of whole numbers, a < 2^19: (a + 1/2) / b lies at least 1 / 2b from the next whole number, which two roundings and the quotient's 2 ulp
// stay below.  A fifth of an integer division's latency.
__device__ __forceinline__ int bt_div(int a, int b) { return static_cast<int>(__fdividef(static_cast<float>(a) + 0.5f, static_cast<float>(b))); }
// Place of 16-byte piece c of token row n: the rows that a quarter warp reads (n, n + 1) lie in distinct banks.
__device__ __forceinline__ int bt_piece(int n, int c) { return (c ^ ((n & 1) << 2)) * 16; }

struct BtArgs {
  const unsigned char* arena;
  const unsigned char* toktab;
  const FastExpert* fast;
  const __half* h_gate;
  const __half* h_up;
  const int32_t* token_indices;
  const int32_t* expert_offsets;
  const float* route_w;
  float* rank_accum;
  long long* acc64;
  int* status;
  int h_rank, rank_out, T, num_experts, n_tiles, max_slots, sec_bytes, ring, tab_bytes;
  int wait_limit_us;
};

struct BtUnit {
  FastExpert fe;
  int tok[BT_NT];
  float rw[BT_NT];
  int npass, tile0, ntiles, pad_;
};

__device__ __noinline__ bool bt_wait_slow(uint32_t addr, uint32_t parity, volatile int* abort_flag) {
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
    if ((i & 7u) == 7u) {
      const uint64_t now = tc::global_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > static_cast<uint64_t>(abort_flag[1]) * 1000u) { *abort_flag = 1; return false; }
    }
  }
}
__device__ __forceinline__ bool bt_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  const uint32_t addr = tc::smem_u32(bar);
  uint32_t done;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(done)
               : "r"(addr), "r"(parity)
               : "memory");
  return done ? true : bt_wait_slow(addr, parity, abort_flag);
}

__device__ __forceinline__ void bt_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ __half2 bt_h2(uint32_t v) { return *reinterpret_cast<const __half2*>(&v); }

// `npairs` pairs of blocks of one group against the token-side operand, from pair `p0` of the matrix on.  `wp`: this lane's
// word(s) of the first pair, pairs `stride` bytes apart; `sp`: its scales of pair p0; `hp`: row g of the operand.
template <bool DENSE>
__device__ __forceinline__ void bt_pairs(const DqMagic& magic, const unsigned char* wp, const unsigned char* sp, const unsigned char* hp, int hs_row, int p0,
                                         int npairs, int g, int t, float (&acc)[BT_NP][4]) {
  constexpr int STRIDE = DENSE ? 1024 : 2048;
  if (npairs <= 0) return;
  uint2 w;
  if (DENSE) w.x = *reinterpret_cast<const uint32_t*>(wp);
  else w = *reinterpret_cast<const uint2*>(wp);
  uint4 s = *reinterpret_cast<const uint4*>(sp);
#pragma unroll 2
  for (int p = 0; p < npairs; ++p) {
    uint4 b[BT_NP];
#pragma unroll
    for (int nb = 0; nb < BT_NP; ++nb) b[nb] = *reinterpret_cast<const uint4*>(hp + nb * 8 * hs_row + bt_piece(g, 4 * (p0 + p) + t));
    uint32_t a0[4], a1[4];
    dequant_block<DENSE>(magic, w.x, bt_h2(s.x), bt_h2(s.x), bt_h2(s.y), bt_h2(s.y), a0);
    dequant_block<DENSE>(magic, DENSE ? w.x >> 8 : w.y, bt_h2(s.z), bt_h2(s.z), bt_h2(s.w), bt_h2(s.w), a1);
    if (p + 1 < npairs) {
      wp += STRIDE;
      sp += 64;
      if (DENSE) w.x = *reinterpret_cast<const uint32_t*>(wp);
      else w = *reinterpret_cast<const uint2*>(wp);
      s = *reinterpret_cast<const uint4*>(sp);
    }
#pragma unroll
    for (int nb = 0; nb < BT_NP; ++nb) bt_mma(acc[nb], a0, b[nb].x, b[nb].y);
#pragma unroll
    for (int nb = 0; nb < BT_NP; ++nb) bt_mma(acc[nb], a1, b[nb].z, b[nb].w);
  }
}

// MAXMB: 16-slot blocks of the down matrix per warp (2: up to 256 slots, 4: up to 512)
template <int MAXMB>
__global__ void __launch_bounds__(BT_THREADS, 2) experts_batch_kernel(const __grid_constant__ BtArgs A) {
  extern __shared__ __align__(128) unsigned char bt_smem[];
  __shared__ BtUnit info[2];
  __shared__ __align__(8) uint64_t bar_full[BT_MAX_RING], bar_tab[2];
  __shared__ int warp_tot[BT_WARPS], abort_s[2], n_units_s;
  volatile int* abort_flag = abort_s;
  const int tid = threadIdx.x, warp = tc::warp_index(), lane = tid & 31, g = lane >> 2, t = lane & 3;
  const BtLayout lay = bt_layout(A.max_slots, A.sec_bytes, A.ring, A.num_experts, A.tab_bytes);
  const TokTab tl(A.h_rank, A.max_slots);
  const int tab_stride = static_cast<int>(align_up_c(static_cast<size_t>(A.tab_bytes), 128));
  int* soff = reinterpret_cast<int*>(bt_smem + lay.soff);        // expert_offsets
  int* pbase = reinterpret_cast<int*>(bt_smem + lay.pbase);      // passes before each expert
  if (tid == 0) {
    for (int i = 0; i < A.ring; ++i) tc::mbar_init(&bar_full[i], 1);
    tc::mbar_init(&bar_tab[0], 1);
    tc::mbar_init(&bar_tab[1], 1);
    tc::mbar_init_fence();
    abort_s[0] = A.wait_limit_us == 0;
    abort_s[1] = A.wait_limit_us;
  }
  // everything above runs while the kernel before this one (launched with programmatic serialisation) drains
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // ---- passes per expert and their exclusive prefix: four consecutive experts a thread
  int total;
  {
    const int e0 = tid * 4;
    int o[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) o[i] = e0 + i <= A.num_experts ? A.expert_offsets[e0 + i] : 0;
    int pass[4], sum = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int cnt = e0 + i < A.num_experts ? o[i + 1] - o[i] : 0;
      pass[i] = cnt > 0 ? (cnt + BT_NT - 1) / BT_NT : 0;
      sum += pass[i];
      if (e0 + i <= A.num_experts) soff[e0 + i] = o[i];
    }
    if (e0 + 4 == A.num_experts) soff[e0 + 4] = o[4];
    int incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += n;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    int before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < BT_WARPS; ++w) {
      const int n = warp_tot[w];
      if (w < warp) before += n;
      all += n;
    }
    total = all;
    int run = before + incl - sum;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (e0 + i < A.num_experts) pbase[e0 + i] = run;
      run += pass[i];
    }
    __syncthreads();
  }
  // Passes that fill whole rounds of the grid are units of their own.  Those of the last, partial round are cut along the tiles: into equal
  // parts, a part a CTA, or, where that leaves the longest part a tile more than an even share of all, into such shares of the passes laid
  // end to end, which may hold the end of one pass and the start of the next (two units).  One warp works it out: divisions in all eight
  // took 0.4 us of issue slots.
  const int grid = static_cast<int>(gridDim.x), cta = static_cast<int>(blockIdx.x);
  const int rounds = total / grid, rem = total - rounds * grid;
  int last_pass = 0, last_tile = 0, last_ntiles[2] = {0, 0};      // this CTA's units of the last round: the second one starts the next pass
  if (warp == 0 && rem) {
    const int parts = min(bt_div(grid, rem), A.n_tiles), per = bt_div(A.n_tiles + parts - 1, parts), all = rem * A.n_tiles;
    if (bt_even_shares(all, per, grid)) {
      const int first = cta * all / grid, end = (cta + 1) * all / grid;
      last_pass = first / A.n_tiles;
      last_tile = first - last_pass * A.n_tiles;
      last_ntiles[0] = min(end - first, A.n_tiles - last_tile);
      last_ntiles[1] = end - first - last_ntiles[0];
    } else {
      const int used = bt_div(A.n_tiles + per - 1, per);
      last_pass = bt_div(cta, used);
      last_tile = (cta - last_pass * used) * per;
      last_ntiles[0] = last_pass < rem ? min(per, A.n_tiles - last_tile) : 0;
    }
  }
  if (tid == 0) n_units_s = rounds + (last_ntiles[0] > 0) + (last_ntiles[1] > 0);

  const DqMagic magic;
  // ---- unit look-up (warp 0): issued with `begin`, in shared memory after `finish`
  constexpr int FE_WORDS = sizeof(FastExpert) / 4, FE_LANES = (FE_WORDS + 31) / 32;
  uint32_t nx_fe[FE_LANES];
  int nx_tok = 0, nx_n = 0, nx_tile0 = 0, nx_ntiles = 0;
  float nx_rw = 0.f;
  int looked_up = 0;                            // units whose tables are on their way or there
  auto look_up = [&](int it) {
    int pu = cta + it * grid, tile0 = 0, ntl = A.n_tiles;
    if (it >= rounds) {
      const bool second = it > rounds;
      pu = rounds * grid + last_pass + second;
      tile0 = second ? 0 : last_tile;
      ntl = second ? last_ntiles[1] : last_ntiles[0];
    }
    int lo = 0, hi = A.num_experts - 1;           // last expert whose prefix is <= pu
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (pbase[mid] <= pu) lo = mid; else hi = mid - 1;
    }
    // an expert's assignments are spread evenly over its passes
    const int e = lo, begin = soff[e], cnt = soff[e + 1] - begin, parts = (cnt + BT_NT - 1) / BT_NT, j = pu - pbase[e];
    int a0 = begin, end = begin + cnt;
    if (parts > 1) {      // (64-bit divisions)
      a0 = begin + static_cast<int>(static_cast<int64_t>(cnt) * j / parts);
      end = begin + static_cast<int>(static_cast<int64_t>(cnt) * (j + 1) / parts);
    }
    ++looked_up;
    nx_n = end - a0;
    nx_tile0 = tile0;
    nx_ntiles = ntl;
#pragma unroll
    for (int i = 0; i < FE_LANES; ++i) {
      const int w = lane + 32 * i;
      nx_fe[i] = w < FE_WORDS ? reinterpret_cast<const uint32_t*>(&A.fast[e])[w] : 0u;
    }
    nx_tok = lane < nx_n ? A.token_indices[a0 + lane] : -1;
    nx_rw = lane < nx_n ? A.route_w[a0 + lane] : 0.f;
    if (lane == 0) {
      tc::mbar_expect_tx(&bar_tab[it & 1], A.tab_bytes);
      tc::bulk_g2s(bt_smem + lay.tab + (it & 1) * tab_stride, A.toktab + static_cast<size_t>(e) * A.tab_bytes, A.tab_bytes, &bar_tab[it & 1]);
    }
  };
  auto look_up_done = [&](int it) {
    BtUnit& s = info[it & 1];
#pragma unroll
    for (int i = 0; i < FE_LANES; ++i) {
      const int w = lane + 32 * i;
      if (w < FE_WORDS) reinterpret_cast<uint32_t*>(&s.fe)[w] = nx_fe[i];
    }
    const bool good = nx_tok >= 0 && nx_tok < A.T;
    if (lane < BT_NT) {
      s.tok[lane] = good ? nx_tok : 0;
      s.rw[lane] = good ? nx_rw : 0.f;
    }
    if (lane == 0) { s.npass = nx_n; s.tile0 = nx_tile0; s.ntiles = nx_ntiles; }
    __syncwarp();
  };
  // ---- copies (one thread): the sections gate, up, down of every tile of this CTA's units in turn, one ring slot each
  const uint32_t R = static_cast<uint32_t>(A.ring);
  uint32_t is_seq = 0, is_slot = 0;             // next section to copy, its slot
  int is_unit = 0, is_tile = 0, is_m = 0;       // ... its unit (of this CTA), tile of the unit, matrix
  auto issue = [&](uint32_t limit, int known) {      // sections before `limit`, of units before `known`
    while (is_seq < limit && is_unit < known) {
      const BtUnit& s = info[is_unit & 1];
      const FastMat& m = s.fe.m[is_m];
      const uint32_t bytes = static_cast<uint32_t>(m.nslots) * 2u + static_cast<uint32_t>(m.words) * 4u;
      tc::mbar_expect_tx(&bar_full[is_slot], bytes);
      tc::bulk_g2s(bt_smem + lay.ring + is_slot * A.sec_bytes,
                   A.arena + s.fe.unit_base + static_cast<int64_t>(s.tile0 + is_tile) * s.fe.unit_bytes + s.fe.sec_off[is_m], bytes, &bar_full[is_slot]);
      ++is_seq;
      if (++is_slot == R) is_slot = 0;
      if (++is_m == 3) {
        is_m = 0;
        if (++is_tile == s.ntiles) { is_tile = 0; ++is_unit; }
      }
    }
  };
  uint32_t rs = 0, rp = 0;                      // ring slot and phase of the next section to read
  uint32_t used = 0;                            // sections that every warp has read
  auto advance = [&]() { if (++rs == R) { rs = 0; rp ^= 1u; } };
  bool ok = A.wait_limit_us != 0, leave = false;      // this warp's waits; what the warps decided
  int it = 0;
  if (warp == 0 && rounds + last_ntiles[0] > 0) {
    look_up(0);
    look_up_done(0);
    if (lane == 0) issue(R, 1);
  }
  __syncthreads();
  const int n_units = n_units_s;                // of this CTA
  for (; it < n_units; ++it) {
    const BtUnit& si = info[it & 1];
    const FastExpert& fe = si.fe;
    const int npass = si.npass, ntl = si.ntiles;
    const bool more = it + 1 < n_units;
    const unsigned char* tab = bt_smem + lay.tab + (it & 1) * tab_stride;
    ok = ok && bt_wait(&bar_tab[it & 1], (it >> 1) & 1, abort_flag);
    // ---- operand rows hs[m][n][position] = fp16(h[token, rank] * s).  A lane owns an octet of ranks, which the arena layout
    // keeps together: one 16-byte load, four multiplications, one 16-byte store.  Rows past npass keep whatever they hold.
    if (ok) {
      const TokTabHead& head = *reinterpret_cast<const TokTabHead*>(tab);
      const int16_t* pos_r = reinterpret_cast<const int16_t*>(tab + tl.pos_r);
      const __half* s_r = reinterpret_cast<const __half*>(tab + tl.s_r);
      const int16_t* oct_r = reinterpret_cast<const int16_t*>(tab + tl.oct_r);
      const int n_oct = A.h_rank >> 3;
      unsigned char* hs = bt_smem + lay.hs;
      for (int o0 = 0; o0 < n_oct; o0 += 32) {
        const int o = o0 + lane;
        int piece[2];
        uint4 sc[2];
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          piece[m] = o < n_oct ? oct_r[m * n_oct + o] : -1;
          sc[m] = piece[m] < 0 ? make_uint4(0u, 0u, 0u, 0u) : *reinterpret_cast<const uint4*>(s_r + m * A.h_rank + 8 * o);
        }
        uint4 hv[BT_NP][2];                      // this warp's tokens: warp, warp + 8, ...
#pragma unroll
        for (int j = 0; j < BT_NP; ++j) {
          const int n = warp + 8 * j;
          const int64_t row = static_cast<int64_t>(si.tok[n]) * A.h_rank + 8 * o;
#pragma unroll
          for (int m = 0; m < 2; ++m)
            if (n < npass && piece[m] >= 0) hv[j][m] = __ldg(reinterpret_cast<const uint4*>((m ? A.h_up : A.h_gate) + row));
        }
#pragma unroll
        for (int j = 0; j < BT_NP; ++j) {
          const int n = warp + 8 * j;
#pragma unroll
          for (int m = 0; m < 2; ++m)
            if (n < npass && piece[m] >= 0) {
              uint4 r;
              const __half2 *hp = reinterpret_cast<const __half2*>(&hv[j][m]), *sp = reinterpret_cast<const __half2*>(&sc[m]);
              __half2* rp2 = reinterpret_cast<__half2*>(&r);
#pragma unroll
              for (int k = 0; k < 4; ++k) rp2[k] = __hmul2(hp[k], sp[k]);       // one rounding of the exact product
              *reinterpret_cast<uint4*>(hs + m * lay.hs_m + n * lay.hs_row + bt_piece(n, piece[m])) = r;
            }
        }
      }
      auto put = [&](int m, int n, int pos, __half v) {
        *reinterpret_cast<__half*>(hs + m * lay.hs_m + n * lay.hs_row + bt_piece(n, pos >> 3) + (pos & 7) * 2) = v;
      };
      for (int m = 0; m < 2; ++m)
        for (int w = 0; w < (n_oct + 31) >> 5; ++w)
          for (uint32_t left = head.broken[m][w]; left; left &= left - 1) {
            const int o = 32 * w + __ffs(left) - 1;
            for (int i = tid; i < 8 * npass; i += BT_THREADS) {
              const int n = i >> 3, rk = 8 * o + (i & 7), pos = pos_r[m * A.h_rank + rk];
              if (pos >= 0) put(m, n, pos, __hmul((m ? A.h_up : A.h_gate)[static_cast<int64_t>(si.tok[n]) * A.h_rank + rk], s_r[m * A.h_rank + rk]));
            }
          }
      // Slots that the octets above do not reach.  Padding: the weights are zero, the activations have to be finite.  A
      // rank that several slots hold: each slot has weights and a factor of its own.
      if (head.loose) {
        for (int m = 0; m < 2; ++m) {
          const int nslots = fe.m[m].nslots;
          const int16_t* rank_t = reinterpret_cast<const int16_t*>(A.arena + fe.m[m].tab_off);
          const __half* s_t = reinterpret_cast<const __half*>(rank_t + nslots);
          for (int i = warp; i < nslots; i += BT_WARPS) {
            const int rk = rank_t[i], pos = slot_pos(i);
            const bool live = rk >= 0 && rk < A.h_rank;
            if (live && pos_r[m * A.h_rank + rk] == pos) continue;
            const __half sv = live ? s_t[i] : __float2half(0.f);
            for (int n = lane; n < npass; n += 32)
              put(m, n, pos, live ? __hmul((m ? A.h_up : A.h_gate)[static_cast<int64_t>(si.tok[n]) * A.h_rank + rk], sv) : sv);
          }
        }
      }
    }
    if ((leave = __syncthreads_or(!ok))) break;
    // every warp is done with the unit before: its ring slots, its description and its tables
    if (tid == 0) issue(used + R, it + 1);
    if (warp == 0 && more) look_up(it + 1);

    float dacc[MAXMB][BT_NP][4];
#pragma unroll
    for (int i = 0; i < MAXMB; ++i)
#pragma unroll
      for (int nb = 0; nb < BT_NP; ++nb)
#pragma unroll
        for (int j = 0; j < 4; ++j) dacc[i][nb][j] = 0.f;
    const int nblk_d = fe.m[2].nslots >> 4, nib_d = fe.m[2].nblk[0];

    for (int i = 0; i < ntl; ++i) {
      // ---- gate / up: this warp owns columns 16 warp .. 16 warp + 15 of the tile
      float acc[2][BT_NP][4];
#pragma unroll
      for (int m = 0; m < 2; ++m) {
#pragma unroll
        for (int nb = 0; nb < BT_NP; ++nb)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[m][nb][j] = 0.f;
        if (ok) ok = bt_wait(&bar_full[rs], rp, abort_flag);
        if (ok) {
          // scales per slot, then nibble words [pair][x][lane][2], dense words [pair][x][lane]
          const unsigned char* sec = bt_smem + lay.ring + rs * A.sec_bytes;
          const unsigned char* words = sec + fe.m[m].nslots * 2;
          const unsigned char* hp = bt_smem + lay.hs + m * lay.hs_m + g * lay.hs_row;
          const int nib = fe.m[m].nblk[0] >> 1, den = fe.m[m].nblk[1] >> 1;
          bt_pairs<false>(magic, words + (warp * 32 + lane) * 8, sec + 16 * t, hp, lay.hs_row, 0, nib, g, t, acc[m]);
          bt_pairs<true>(magic, words + nib * 2048 + (warp * 32 + lane) * 4, sec + nib * 64 + 16 * t, hp, lay.hs_row, nib, den, g, t, acc[m]);
        }
        advance();
      }
      // ---- z = silu(g) * u as the down product's operand.  A thread has columns g and g + 8 of tokens 2 t and 2 t + 1;
      // with its neighbour of the next column it makes pairs of columns: lanes of even g store the even tokens.
      unsigned char* zb = bt_smem + lay.z + (i & 1) * lay.z_buf;
      {
        const int n_row = 2 * t + (g & 1);
#pragma unroll
        for (int nb = 0; nb < BT_NP; ++nb) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float z0 = silu_mul(acc[0][nb][2 * h], acc[1][nb][2 * h]), z1 = silu_mul(acc[0][nb][2 * h + 1], acc[1][nb][2 * h + 1]);
            const float other = __shfl_xor_sync(0xffffffffu, g & 1 ? z0 : z1, 4);
            const __half2 v = g & 1 ? __floats2half2_rn(other, z1) : __floats2half2_rn(z0, other);
            const int pos = slot_pos(16 * warp + (g & ~1) + 8 * h), n = 8 * nb + n_row;
            *reinterpret_cast<__half2*>(zb + n * (N_TILE * 2) + bt_piece(n, pos >> 3) + (pos & 7) * 2) = v;
          }
        }
      }
      if (warp == 0 && i == 0 && more) look_up_done(it + 1);
      if ((leave = __syncthreads_or(!ok))) break;
      // every warp has read this tile's gate and up sections and the down section before them
      if (tid == 0) issue(used + 2 + R, more ? it + 2 : it + 1);
      used += 3;
      // ---- down: slot blocks round-robin over the warps, contraction over the tile's 128 columns
      ok = bt_wait(&bar_full[rs], rp, abort_flag);
      if (ok) {
        const unsigned char* sec = bt_smem + lay.ring + rs * A.sec_bytes;
        const unsigned char* words = sec + fe.m[2].nslots * 2;
        const unsigned char* zrow = zb + g * (N_TILE * 2);
        uint32_t sc[MAXMB];
#pragma unroll
        for (int i2 = 0; i2 < MAXMB; ++i2) sc[i2] = warp + 8 * i2 < nblk_d ? *reinterpret_cast<const uint32_t*>(sec + (warp + 8 * i2) * 32 + 4 * g) : 0u;     // rows g and g + 8
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          uint4 b[BT_NP];
#pragma unroll
          for (int nb = 0; nb < BT_NP; ++nb) b[nb] = *reinterpret_cast<const uint4*>(zrow + nb * 8 * (N_TILE * 2) + bt_piece(g, 4 * p + t));
#pragma unroll
          for (int i2 = 0; i2 < MAXMB; ++i2) {
            const int mb = warp + 8 * i2;
            if (mb >= nblk_d) break;
            const __half2 lo = __low2half2(bt_h2(sc[i2])), hi = __high2half2(bt_h2(sc[i2]));
            uint32_t a0[4], a1[4];
            // nibble words [mblock][pair][lane][2], dense words [mblock][pair][lane]
            if (mb < nib_d) {
              const uint2 w = *reinterpret_cast<const uint2*>(words + ((mb * 4 + p) * 32 + lane) * 8);
              dequant_block<false>(magic, w.x, lo, hi, lo, hi, a0);
              dequant_block<false>(magic, w.y, lo, hi, lo, hi, a1);
            } else {
              const uint32_t w = *reinterpret_cast<const uint32_t*>(words + nib_d * 1024 + (((mb - nib_d) * 4 + p) * 32 + lane) * 4);
              dequant_block<true>(magic, w, lo, hi, lo, hi, a0);
              dequant_block<true>(magic, w >> 8, lo, hi, lo, hi, a1);
            }
#pragma unroll
            for (int nb = 0; nb < BT_NP; ++nb) bt_mma(dacc[i2][nb], a0, b[nb].x, b[nb].y);
#pragma unroll
            for (int nb = 0; nb < BT_NP; ++nb) bt_mma(dacc[i2][nb], a1, b[nb].z, b[nb].w);
          }
        }
      }
      advance();
    }
    if (leave) break;
    // ---- rank_accum[token, rank] += sum over the unit's tiles * s * route weight
    if (ok) {
      const float* s_d = reinterpret_cast<const float*>(tab + tl.s_d);
      const int16_t* rank_d = reinterpret_cast<const int16_t*>(tab + tl.rank_d);
#pragma unroll
      for (int i2 = 0; i2 < MAXMB; ++i2) {
        const int mb = warp + 8 * i2;
        if (mb >= nblk_d) break;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int slot = mb * 16 + g + 8 * h, rk = rank_d[slot];
          if (rk < 0 || rk >= A.rank_out) continue;
          const float sv = s_d[slot];
#pragma unroll
          for (int nb = 0; nb < BT_NP; ++nb)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              const int n = 8 * nb + 2 * t + q;
              if (n < npass) acc_add(A.rank_accum, A.acc64, static_cast<int64_t>(si.tok[n]) * A.rank_out + rk, dacc[i2][nb][2 * h + q] * sv * si.rw[n]);
            }
        }
      }
    }
  }
  if (!leave) leave = __syncthreads_or(!ok);
  // A CTA that gives up leaves behind the copies it has started (or behind the limit of this wait): the sections in the last R
  // slots, and the tables of the unit at hand and of the next one.
  if (leave && tid == 0) {
    const uint32_t first = is_seq > R ? is_seq - R : 0;
    for (uint32_t s = first; s < is_seq; ++s) tc::mbar_wait(&bar_full[s % R], (s / R) & 1u, BT_DRAIN_LIMIT_NS);
    for (int j = max(looked_up - 2, 0); j < looked_up; ++j) tc::mbar_wait(&bar_tab[j & 1], (j >> 1) & 1, BT_DRAIN_LIMIT_NS);
    atomicExch(A.status, BM_ERR_TIMEOUT);
  }
}

bool experts_batch_even_shares(int all, int per, int grid) { return bt_even_shares(all, per, grid); }

// Ring depth and grid for this layer on the current device; bat_ring = 0 where the layer does not suit the kernel.
int plan_experts_batch(bm_layer* L) {
  L->bat_ring = 0;
  int dev = -1, sm_count = 0, smem_sm = 0;
  BM_CUDA(cudaGetDevice(&dev));
  BM_CUDA(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev));
  L->sms = sm_count;
  if (!L->fast_ok || !L->toktab_dev || L->num_experts > BT_MAX_E || L->intermediate % N_TILE != 0 || L->max_slots > 512 || L->rank_in % 8 != 0) return BM_OK;
  BM_CUDA(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
  const void* kernel = L->max_slots <= 256 ? reinterpret_cast<const void*>(experts_batch_kernel<2>) : reinterpret_cast<const void*>(experts_batch_kernel<4>);
  cudaFuncAttributes fa;
  BM_CUDA(cudaFuncGetAttributes(&fa, kernel));
  const int room = smem_sm / 2 - 1024 - static_cast<int>(fa.sharedSizeBytes), tab = TokTab(L->rank_in, L->max_slots).bytes;
  L->bat_sec_bytes = static_cast<int>(align_up_c(static_cast<size_t>(L->max_slots) * 2 + static_cast<size_t>(L->max_words) * 4, 128));
  for (int ring = BT_MAX_RING; ring >= 3 && !L->bat_ring; --ring) {
    const int total = bt_layout(L->max_slots, L->bat_sec_bytes, ring, L->num_experts, tab).total;
    if (total > room) continue;
    L->bat_ring = ring;
    L->bat_smem = total;
    L->bat_grid = 2 * sm_count;
  }
  if (!L->bat_ring) return BM_OK;
  BM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, room));
  BM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
  return BM_OK;
}

int launch_experts_batch(const bm_layer* L, const __half* h_gate, const __half* h_up, const int32_t* token_indices, const int32_t* expert_offsets,
                         const float* route_w, int T, float* rank_accum, long long* acc64, cudaStream_t st) {
  BM_REQUIRE(L->bat_ring, BM_ERR_UNSUPPORTED, "experts_batch: the layer does not suit this kernel");
  BM_REQUIRE(((reinterpret_cast<uintptr_t>(h_gate) | reinterpret_cast<uintptr_t>(h_up)) & 15u) == 0, BM_ERR_INVALID_ARG,
             "experts_batch: h_gate / h_up rows must be 16-byte aligned");
  BtArgs a{};
  a.arena = static_cast<const unsigned char*>(L->arena);
  a.toktab = L->toktab_dev;
  a.fast = L->fast_dev;
  a.h_gate = h_gate; a.h_up = h_up;
  a.token_indices = token_indices; a.expert_offsets = expert_offsets; a.route_w = route_w;
  a.rank_accum = rank_accum; a.acc64 = acc64; a.status = L->status_dev;
  a.h_rank = L->rank_in; a.rank_out = L->rank_out; a.T = T; a.num_experts = L->num_experts; a.n_tiles = L->n_tiles; a.max_slots = L->max_slots;
  a.tab_bytes = TokTab(L->rank_in, L->max_slots).bytes;
  a.sec_bytes = L->bat_sec_bytes; a.ring = L->bat_ring;
  a.wait_limit_us = L->wait_limit_us;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(L->bat_grid);
  cfg.blockDim = dim3(BT_THREADS);
  cfg.dynamicSmemBytes = L->bat_smem;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  BM_CUDA(cudaLaunchKernelEx(&cfg, L->max_slots <= 256 ? experts_batch_kernel<2> : experts_batch_kernel<4>, a));
  BM_LAUNCH_CHECK("experts_batch_kernel");
  return BM_OK;
}

}  // namespace bm
