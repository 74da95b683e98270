// C ABI glue: error reporting, layer planning / creation over the reference's buffers,
// stage entry points and the composed layer forward.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <new>
#include <string>

#include "skinny.cuh"

namespace bm {

static thread_local char g_err[512] = "";

int set_error(int status, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return status;
}

static std::atomic<unsigned long long> g_launches{0};
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

// from the other translation units
int launch_gemm_nt(const GemmArgs& g, int problems, cudaStream_t st);
void plan_fast(const bm_layer* L, size_t base_bytes, FastPlan* P);
int build_fast(bm_layer* L, const FastPlan& P, cudaStream_t st);
size_t fast_build_scratch_bytes(const FastPlan& P);
int launch_arena_decode(const bm_layer* L, int e, int w, int8_t* codes, cudaStream_t st);
int plan_experts_decode(bm_layer* L);
int launch_experts_decode(const bm_layer* L, const __half* h_gate, const __half* h_up, const int32_t* token_indices,
                          const int32_t* expert_offsets, const float* route_w, int T, int num_assign, float* rank_accum,
                          long long* acc64, cudaStream_t st);
int plan_experts_batch(bm_layer* L);
int launch_experts_batch(const bm_layer* L, const __half* h_gate, const __half* h_up, const int32_t* token_indices, const int32_t* expert_offsets,
                         const float* route_w, int T, float* rank_accum, long long* acc64, cudaStream_t st);
bool experts_batch_even_shares(int all, int per, int grid);
bool experts_tc_fits(const bm_layer* L);
double experts_tc_us(const bm_layer* L, double load, int* rows);
int expected_passes(int experts, double load, int size);
int launch_experts_tc(const bm_layer* L, const __half* h_gate, const __half* h_up, const int32_t* token_indices,
                      const int32_t* expert_offsets, const float* route_w, int T, int expected_assign, int rows, float* rank_accum, long long* acc64,
                      cudaStream_t st);
int launch_experts_generic(const bm_layer* L, const __half* h_gate, const __half* h_up, const int32_t* token_indices,
                           const int32_t* expert_offsets, const float* route_w, int T, float* rank_accum,
                           long long* acc64, cudaStream_t st);

static const char* which_name(int w) { return w == 0 ? "gate" : (w == 1 ? "up" : "down"); }

// Pinned host memory for the meta read-back.  The copies of a layer (three for each of 384 matrices at 128
// experts) run behind one another and are waited for once: one blocking copy each made the build 33 ms, this way it is 17.
struct PinnedInts {
  int32_t* p = nullptr;
  ~PinnedInts() { if (p) cudaFreeHost(p); }
};

static int check_matrix(const bm_matrix_t& m, int which, int expert) {
  BM_REQUIRE(m.n_slabs >= 0 && m.n_tile_rows >= 0 && m.n_rows >= 0 && m.payload_words >= 0 && m.n_scales >= 0,
             BM_ERR_INVALID_ARG, "%s[%d]: negative buffer length", which_name(which), expert);
  BM_REQUIRE(!m.n_slabs || (m.slab_meta && m.payload && m.rank_idx && m.scale && m.s), BM_ERR_INVALID_ARG, "%s[%d]: null buffer",
             which_name(which), expert);
  BM_REQUIRE(!m.n_tile_rows || m.tile_meta, BM_ERR_INVALID_ARG, "%s[%d]: null tile_meta", which_name(which), expert);
  return BM_OK;
}
// ints of a matrix's meta: slab rows, tile rows and, where the row order matters, the rows' ranks
static size_t meta_ints(const bm_matrix_t& m, bool ranks) {
  return static_cast<size_t>(m.n_slabs) * 4 + static_cast<size_t>(m.n_tile_rows) * 3 + (ranks && m.n_slabs ? m.n_rows : 0);
}
static int fetch_matrix(const bm_matrix_t& m, bool ranks, int32_t* to) {
  auto copy = [&](const int32_t* from, size_t n) {
    int32_t* dst = to;
    to += n;
    return n ? cudaMemcpyAsync(dst, from, n * 4, cudaMemcpyDeviceToHost, nullptr) : cudaSuccess;
  };
  BM_CUDA(copy(m.slab_meta, static_cast<size_t>(m.n_slabs) * 4));
  BM_CUDA(copy(m.tile_meta, static_cast<size_t>(m.n_tile_rows) * 3));
  if (ranks && m.n_slabs) BM_CUDA(copy(m.rank_idx, m.n_rows));
  return BM_OK;
}

// Takes one matrix's fetched meta over and checks every offset the kernels will use.
static int ingest_matrix(const bm_matrix_t& m, int which, int expert, int intermediate, const int32_t* meta, bool ranks, MatHost* out) {
  const int n_tiles = (intermediate + N_TILE - 1) / N_TILE;
  out->n_rows = m.n_rows;
  out->slabs.clear();
  const int32_t* slab = meta;
  meta += static_cast<size_t>(m.n_slabs) * 4;
  out->tile_meta.assign(meta, meta + static_cast<size_t>(m.n_tile_rows) * 3);
  meta += out->tile_meta.size();
  out->rank_idx.assign(static_cast<size_t>(m.n_rows), -1);
  if (ranks && m.n_slabs) out->rank_idx.assign(meta, meta + m.n_rows);
  for (int i = 0; i < m.n_slabs; ++i) {
    SlabHost s;
    s.bits = slab[i * 4 + 0];
    s.k_slab = slab[i * 4 + 1];
    s.rank_off = slab[i * 4 + 2];
    s.tile_off = slab[i * 4 + 3];
    s.tile_end = (i + 1 < m.n_slabs) ? slab[(i + 1) * 4 + 3] : m.n_tile_rows;
    BM_REQUIRE(supported_bits(s.bits), BM_ERR_UNSUPPORTED, "%s[%d] slab %d: Unsupported bits=%d", which_name(which), expert,
               i, s.bits);
    BM_REQUIRE(s.k_slab >= 1 && s.rank_off >= 0 && s.rank_off + s.k_slab <= m.n_rows, BM_ERR_INVALID_ARG,
               "%s[%d] slab %d: rows [%d, %d) outside rank_idx of %d", which_name(which), expert, i, s.rank_off,
               s.rank_off + s.k_slab, m.n_rows);
    BM_REQUIRE(s.tile_off >= 0 && s.tile_off <= s.tile_end && s.tile_end <= m.n_tile_rows &&
                   s.tile_end - s.tile_off <= n_tiles,
               BM_ERR_INVALID_ARG, "%s[%d] slab %d: tile range [%d, %d) invalid (tile_meta rows %d, tiles per row %d)",
               which_name(which), expert, i, s.tile_off, s.tile_end, m.n_tile_rows, n_tiles);
    const int64_t wpt = static_cast<int64_t>(s.k_slab) * MICROS * words_per_row(s.bits);
    for (int t = s.tile_off; t < s.tile_end; ++t) {
      const int64_t pack_off = out->tile_meta[t * 3 + 0], scale_off = out->tile_meta[t * 3 + 1];
      const int n_valid = out->tile_meta[t * 3 + 2];
      BM_REQUIRE(pack_off >= 0 && pack_off + wpt <= m.payload_words, BM_ERR_INVALID_ARG,
                 "%s[%d] slab %d tile %d: payload [%lld, %lld) outside %lld words", which_name(which), expert, i,
                 t - s.tile_off, (long long)pack_off, (long long)(pack_off + wpt), (long long)m.payload_words);
      BM_REQUIRE(scale_off >= 0 && scale_off + s.k_slab <= m.n_scales, BM_ERR_INVALID_ARG,
                 "%s[%d] slab %d tile %d: scales outside buffer", which_name(which), expert, i, t - s.tile_off);
      BM_REQUIRE(n_valid >= 1 && n_valid <= N_TILE && (t - s.tile_off) * N_TILE + n_valid <= intermediate,
                 BM_ERR_INVALID_ARG, "%s[%d] slab %d tile %d: n_valid=%d does not fit intermediate=%d",
                 which_name(which), expert, i, t - s.tile_off, n_valid, intermediate);
    }
    out->slabs.push_back(s);
  }
  out->bytes = m.payload_words * 4 + m.n_scales * 2 + static_cast<int64_t>(m.n_rows) * (2 + 4) +
               static_cast<int64_t>(m.n_tile_rows) * 12 + static_cast<int64_t>(m.n_slabs) * 16;
  return BM_OK;
}

static int check_desc(const bm_layer_desc_t* d) {
  BM_REQUIRE(d != nullptr, BM_ERR_INVALID_ARG, "null layer descriptor");
  BM_REQUIRE(d->num_experts >= 0, BM_ERR_INVALID_ARG, "num_experts must be >= 0");
  BM_REQUIRE(d->intermediate > 0, BM_ERR_INVALID_ARG, "intermediate_size must be > 0");
  BM_REQUIRE(d->rank_out > 0, BM_ERR_INVALID_ARG, "rank_out must be > 0");
  BM_REQUIRE(d->rank_in > 0, BM_ERR_INVALID_ARG, "rank_in must be > 0");
  BM_REQUIRE(d->intermediate % N_MICRO == 0, BM_ERR_INVALID_ARG, "intermediate_size=%d must be divisible by %d",
             d->intermediate, N_MICRO);
  BM_REQUIRE(d->act_type == 0, BM_ERR_UNSUPPORTED, "only SiLU act_type=0 is currently supported");
  BM_REQUIRE(d->num_experts == 0 || (d->gate && d->up && d->down), BM_ERR_INVALID_ARG, "null matrix tables");
  return BM_OK;
}

// arena = [ExpertDev table][status flag][arena layout ...][build scratch]
static size_t table_bytes(int num_experts) {
  return align_up(sizeof(ExpertDev) * static_cast<size_t>(num_experts > 0 ? num_experts : 1), 256);
}
static size_t base_bytes(int num_experts) { return table_bytes(num_experts) + 256; }

static size_t arena_need(const bm_layer* L, FastPlan* P) {
  plan_fast(L, base_bytes(L->num_experts), P);
  return P->ok ? P->total + fast_build_scratch_bytes(*P) : base_bytes(L->num_experts);
}

// `ranks`: the rows' ranks too.  They order the arena's rows; its size does not depend on them.
static int build_host(const bm_layer_desc_t* d, bool ranks, bm_layer* L) {
  int rc = check_desc(d);
  if (rc) return rc;
  L->num_experts = d->num_experts;
  L->hidden = d->hidden;
  L->intermediate = d->intermediate;
  L->rank_in = d->rank_in;
  L->rank_out = d->rank_out;
  L->n_tiles = (d->intermediate + N_TILE - 1) / N_TILE;
  L->vh_gate = reinterpret_cast<const __half*>(d->vh_gate);
  L->vh_up = reinterpret_cast<const __half*>(d->vh_up);
  L->u_down = reinterpret_cast<const __half*>(d->u_down);
  L->max_rows = 1;
  const bm_matrix_t* tabs[3] = {d->gate, d->up, d->down};
  size_t total = 0;
  for (int w = 0; w < 3; ++w)
    for (int e = 0; e < d->num_experts; ++e) {
      if ((rc = check_matrix(tabs[w][e], w, e))) return rc;
      total += meta_ints(tabs[w][e], ranks);
    }
  PinnedInts meta;
  if (total) {
    BM_CUDA(cudaHostAlloc(reinterpret_cast<void**>(&meta.p), total * 4, cudaHostAllocDefault));
    int32_t* to = meta.p;
    for (int w = 0; w < 3 && !rc; ++w)
      for (int e = 0; e < d->num_experts && !rc; ++e) {
        rc = fetch_matrix(tabs[w][e], ranks, to);
        to += meta_ints(tabs[w][e], ranks);
      }
    const cudaError_t done = cudaStreamSynchronize(nullptr);      // also on error: the copies write into `meta`
    if (rc) return rc;
    BM_CUDA(done);
  }
  const int32_t* from = meta.p;
  for (int w = 0; w < 3; ++w) {
    L->host[w].resize(d->num_experts);
    L->src[w].assign(tabs[w], tabs[w] + d->num_experts);
    for (int e = 0; e < d->num_experts; ++e) {
      rc = ingest_matrix(tabs[w][e], w, e, d->intermediate, from, ranks, &L->host[w][e]);
      if (rc) return rc;
      from += meta_ints(tabs[w][e], ranks);
      if (tabs[w][e].n_rows > L->max_rows) L->max_rows = tabs[w][e].n_rows;
    }
  }
  return BM_OK;
}

// int8 codes of one matrix, decoded through slab/tile meta: one thread per (row, column).
__global__ void decode_codes_kernel(MatDev md, int intermediate, int8_t* __restrict__ codes) {
  const int64_t total = static_cast<int64_t>(md.n_rows) * intermediate;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int row = static_cast<int>(i / intermediate), col = static_cast<int>(i - static_cast<int64_t>(row) * intermediate);
    int8_t q = 0;
    for (int sl = 0; sl < md.n_slabs; ++sl) {
      const int bits = md.slab_meta[sl * 4 + 0], k_slab = md.slab_meta[sl * 4 + 1];
      const int rank_off = md.slab_meta[sl * 4 + 2], tile_off = md.slab_meta[sl * 4 + 3];
      if (row < rank_off || row >= rank_off + k_slab) continue;
      const int tile_end = (sl + 1 < md.n_slabs) ? md.slab_meta[(sl + 1) * 4 + 3] : md.n_tile_rows;
      const int t = tile_off + col / N_TILE;
      if (t >= tile_end || bits == 16) break;
      const int cc = col % N_TILE;
      if (cc >= md.tile_meta[t * 3 + 2]) break;
      const int r = row - rank_off, s0 = (r / K_STAGE) * K_STAGE, rows_cur = min(K_STAGE, k_slab - s0);
      const uint32_t* w = md.payload + md.tile_meta[t * 3 + 0] + s0 * MICROS * bits + (cc / N_MICRO) * rows_cur * bits +
                          (r - s0) * bits;
      int u = 0;
      for (int p = 0; p < bits; ++p) u |= static_cast<int>((w[p] >> (cc % N_MICRO)) & 1u) << p;
      q = static_cast<int8_t>(bits == 1 ? 2 * u - 1 : u - (1 << (bits - 1)));
      break;
    }
    codes[i] = q;
  }
}

static MatDev to_dev(const bm_matrix_t& m) {
  MatDev d;
  d.payload = m.payload;
  d.rank_idx = m.rank_idx;
  d.tile_meta = m.tile_meta;
  d.slab_meta = m.slab_meta;
  d.scale = reinterpret_cast<const __half*>(m.scale);
  d.s = reinterpret_cast<const __half*>(m.s);
  d.n_slabs = m.n_slabs;
  d.n_tile_rows = m.n_tile_rows;
  d.n_rows = m.n_rows;
  d.pad_ = 0;
  return d;
}

struct Carver {
  unsigned char* base;
  size_t off = 0, cap;
  Carver(void* p, size_t c) : base(static_cast<unsigned char*>(p)), cap(c) {}
  template <typename T>
  T* take(size_t n) {
    T* r = reinterpret_cast<T*>(base + off);
    off += align_up(n * sizeof(T), 256);
    return r;
  }
};

struct LayerWs {
  int32_t* topk_idx; float* topk_w; int32_t* token_indices; int32_t* expert_offsets; float* route_flat;
  int32_t* tile_table; int32_t* counts; __half* h_gate; __half* h_up; float* rank_accum;
  void* route_ws; size_t route_ws_bytes; void* experts_ws; size_t experts_ws_bytes; size_t total;
};

constexpr int TILE_ROWS = 128;

static LayerWs carve_layer_ws(const bm_layer* L, void* ws, int T, int k) {
  Carver c(ws, 0);
  LayerWs w;
  const size_t A = static_cast<size_t>(T) * k;
  const int max_tiles = bm_route_max_tiles(T, k, L->num_experts, TILE_ROWS);
  w.topk_idx = c.take<int32_t>(A);
  w.topk_w = c.take<float>(A);
  w.token_indices = c.take<int32_t>(A);
  w.expert_offsets = c.take<int32_t>(L->num_experts + 1);
  w.route_flat = c.take<float>(A);
  w.tile_table = c.take<int32_t>(static_cast<size_t>(max_tiles) * 3);
  w.counts = c.take<int32_t>(2);
  w.h_gate = c.take<__half>(static_cast<size_t>(T) * L->rank_in);
  w.h_up = c.take<__half>(static_cast<size_t>(T) * L->rank_in);
  w.rank_accum = c.take<float>(static_cast<size_t>(T) * L->rank_out);
  w.route_ws_bytes = bm_route_build_workspace_bytes(T, k, L->num_experts);
  w.route_ws = c.take<unsigned char>(w.route_ws_bytes);
  w.experts_ws_bytes = bm_experts_workspace_bytes(L, T, static_cast<int32_t>(A), BM_PATH_AUTO);
  w.experts_ws = c.take<unsigned char>(w.experts_ws_bytes);
  w.total = c.off;
  return w;
}

}  // namespace bm

using namespace bm;

extern "C" int bm_abi_version(void) { return 2; }
extern "C" const char* bm_last_error(void) { return g_err; }
extern "C" uint64_t bm_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }
extern "C" int bm_arena_layout_version(void) { return 4; }   // 4: octets of ranks kept together, down scales by fragment rows
extern "C" const char* bm_status_string(int s) {
  switch (s) {
    case BM_OK: return "ok";
    case BM_ERR_INVALID_ARG: return "invalid argument";
    case BM_ERR_UNSUPPORTED: return "unsupported";
    case BM_ERR_CUDA: return "CUDA error";
    case BM_ERR_WORKSPACE: return "workspace too small";
    case BM_ERR_TIMEOUT: return "device wait timed out";
    default: return "unknown status";
  }
}

extern "C" int bm_layer_plan(const bm_layer_desc_t* desc, size_t* arena_bytes) {
  BM_REQUIRE(arena_bytes != nullptr, BM_ERR_INVALID_ARG, "null arena_bytes");
  bm_layer tmp;
  const int rc = build_host(desc, false, &tmp);
  if (rc) return rc;
  FastPlan P;
  *arena_bytes = arena_need(&tmp, &P);
  return BM_OK;
}

extern "C" int bm_layer_create(const bm_layer_desc_t* desc, void* arena, size_t arena_bytes, void* stream,
                               bm_layer_t** out) {
  BM_REQUIRE(out != nullptr, BM_ERR_INVALID_ARG, "null output handle");
  *out = nullptr;
  bm_layer* L = new (std::nothrow) bm_layer();
  BM_REQUIRE(L != nullptr, BM_ERR_INVALID_ARG, "out of host memory");
  int rc = build_host(desc, true, L);
  if (rc) { delete L; return rc; }
  FastPlan P;
  const size_t need = arena_need(L, &P);
  if (arena == nullptr || arena_bytes < need || (reinterpret_cast<uintptr_t>(arena) & 255u)) {
    delete L;
    return set_error(BM_ERR_WORKSPACE, "layer arena must be 256-byte aligned and hold %zu bytes (%zu given)", need, arena_bytes);
  }
  cudaGetDevice(&L->device);
  L->arena = arena;
  L->arena_bytes = arena_bytes;
  L->experts_dev = static_cast<ExpertDev*>(arena);
  std::vector<ExpertDev> tab(desc->num_experts);
  for (int e = 0; e < desc->num_experts; ++e) {
    tab[e].m[0] = to_dev(desc->gate[e]);
    tab[e].m[1] = to_dev(desc->up[e]);
    tab[e].m[2] = to_dev(desc->down[e]);
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  L->status_dev = reinterpret_cast<int*>(static_cast<unsigned char*>(arena) + table_bytes(desc->num_experts));
  cudaError_t ce = cudaMemsetAsync(L->status_dev, 0, 256, st);
  if (ce == cudaSuccess && desc->num_experts)
    ce = cudaMemcpyAsync(L->experts_dev, tab.data(), sizeof(ExpertDev) * tab.size(), cudaMemcpyHostToDevice, st);
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(st);
  if (ce != cudaSuccess) {
    delete L;
    return set_error(BM_ERR_CUDA, "uploading the expert table failed: %s", cudaGetErrorString(ce));
  }
  if (P.ok) {
    L->fast_host = P.experts;
    L->fast_dev = reinterpret_cast<const FastExpert*>(static_cast<unsigned char*>(arena) + P.table_off);
    L->max_unit_bytes = P.max_unit_bytes;
    L->max_slots = P.max_slots;
    L->max_words = P.max_words;
    rc = build_fast(L, P, st);
    if (rc) { delete L; return rc; }
    L->fast_ok = true;
    rc = plan_experts_decode(L);
    if (!rc) rc = plan_experts_batch(L);
    if (rc) { delete L; return rc; }
  }
  *out = L;
  return BM_OK;
}

extern "C" int bm_layer_destroy(bm_layer_t* layer) {
  delete layer;
  return BM_OK;
}

extern "C" int64_t bm_layer_expert_bytes(const bm_layer_t* L, int32_t e) {
  if (!L || e < 0 || e >= L->num_experts) return -1;
  return L->host[0][e].bytes + L->host[1][e].bytes + L->host[2][e].bytes;
}

extern "C" int bm_layer_set_option(bm_layer_t* L, int32_t option, int32_t value) {
  BM_REQUIRE(L != nullptr, BM_ERR_INVALID_ARG, "set_option: null layer");
  if (option == BM_OPT_DETERMINISTIC) {
    BM_REQUIRE(value == 0 || value == 1, BM_ERR_INVALID_ARG, "set_option: the deterministic mode is 0 or 1");
    L->deterministic = value != 0;
    return BM_OK;
  }
  if (option == BM_OPT_WAIT_LIMIT_US) {
    BM_REQUIRE(value >= 0 && value <= DEFAULT_WAIT_LIMIT_US, BM_ERR_INVALID_ARG, "set_option: the wait limit must be 0..%d us", DEFAULT_WAIT_LIMIT_US);
    L->wait_limit_us = value;
    return BM_OK;
  }
  BM_REQUIRE(option == BM_OPT_DECODE_CTAS_PER_SM, BM_ERR_INVALID_ARG, "set_option: unknown option %d", option);
  BM_REQUIRE(value >= 0 && value <= 3, BM_ERR_INVALID_ARG, "set_option: CTAs per SM must be 0..3");
  const bm_layer saved = *L;
  L->dec_force_ctas = value;
  const int rc = plan_experts_decode(L);
  if (rc || (saved.dec_ok && !L->dec_ok)) {
    *L = saved;
    return rc ? rc : set_error(BM_ERR_UNSUPPORTED, "set_option: %d CTAs per SM do not fit this layer", value);
  }
  return BM_OK;
}

extern "C" int bm_layer_has_fast_layout(const bm_layer_t* L) { return L && L->fast_ok ? 1 : 0; }

extern "C" int bm_layer_status(const bm_layer_t* L, void* stream) {
  BM_REQUIRE(L != nullptr, BM_ERR_INVALID_ARG, "layer_status: null layer");
  int flag = 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  BM_CUDA(cudaMemcpyAsync(&flag, L->status_dev, sizeof(int), cudaMemcpyDeviceToHost, st));
  BM_CUDA(cudaStreamSynchronize(st));
  if (flag != 0) {
    BM_CUDA(cudaMemsetAsync(L->status_dev, 0, sizeof(int), st));
    return set_error(BM_ERR_TIMEOUT, "a kernel of this layer gave up a bounded wait; its outputs are undefined");
  }
  return BM_OK;
}

extern "C" int bm_layer_decode_codes(const bm_layer_t* L, int32_t e, int32_t which, int32_t source, int8_t* codes,
                                     void* stream) {
  BM_REQUIRE(L && codes, BM_ERR_INVALID_ARG, "decode_codes: null pointer");
  BM_REQUIRE(e >= 0 && e < L->num_experts && which >= 0 && which < 3, BM_ERR_INVALID_ARG, "decode_codes: bad index");
  if (source == 1) {
    BM_REQUIRE(L->fast_ok, BM_ERR_UNSUPPORTED, "decode_codes: this layer has no arena layout");
    return launch_arena_decode(L, e, which, codes, static_cast<cudaStream_t>(stream));
  }
  const MatDev md = to_dev(L->src[which][e]);
  const int64_t total = static_cast<int64_t>(md.n_rows) * L->intermediate;
  if (total == 0) return BM_OK;
  const int blocks = static_cast<int>((total + 255) / 256 < 148 * 8 ? (total + 255) / 256 : 148 * 8);
  decode_codes_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(md, L->intermediate, codes);
  BM_LAUNCH_CHECK("decode_codes_kernel");
  return BM_OK;
}

// With `zero` the buffer (16-byte units) is cleared on the way.
static int basis_project(const bm_layer_t* L, const void* x, int x_dtype, int32_t T, uint16_t* h_gate, uint16_t* h_up, LaunchAfter after, float4* zero,
                         int64_t zero_n, cudaStream_t st) {
  BM_REQUIRE(L != nullptr, BM_ERR_INVALID_ARG, "basis_project: null layer");
  BM_REQUIRE(L->vh_gate && L->vh_up, BM_ERR_INVALID_ARG, "missing shared_vh basis for packed routed experts");
  BM_REQUIRE(T >= 0 && x_dtype >= BM_F16 && x_dtype <= BM_F32, BM_ERR_INVALID_ARG, "basis_project: bad arguments");
  if (T == 0) return BM_OK;
  BM_REQUIRE(x && h_gate && h_up, BM_ERR_INVALID_ARG, "basis_project: null pointer");
  // On its own, the skinny product up to 160 tokens, whose chunks of 64 still fit the device at once (bf16, us against the tiled one: 128 tokens
  // 7.8 / 9.0, 160 tokens 8.9 / 9.1, 203 tokens 12.4 / 9.1); the tiled one runs beside the launches before it.
  const bool tiled = L->hidden % 64 == 0 && L->rank_in % 8 == 0 && aligned16(x, L->vh_gate, L->vh_up);
  if (T <= (!tiled ? SKINNY_MAX_TOKENS : after == AFTER_ALL ? 160 : 0) && L->hidden % 128 == 0) {
    SkinnyArgs a{};
    a.seg[0] = SkSeg{L->vh_gate, nullptr, h_gate, L->rank_in, BM_F16, 0, 0};
    a.seg[1] = SkSeg{L->vh_up, nullptr, h_up, L->rank_in, BM_F16, 0, 0};
    a.n_seg = 2;
    a.X = x; a.N = T; a.K = L->hidden; a.x_dtype = x_dtype; a.splits = 8;
    a.zero = zero; a.zero_n = static_cast<int>(zero_n);
    const int rc = launch_skinny_nt(a, st);
    if (rc != BM_ERR_UNSUPPORTED) return rc;       // shape does not tile (e.g. a very wide hidden size): the general GEMMs take it
  }
  if (L->hidden % 64 == 0 && aligned16(x, L->vh_gate, L->vh_up)) {
    GemmTcArgs t{};
    t.X = x; t.W[0] = L->vh_gate; t.W[1] = L->vh_up; t.C[0] = h_gate; t.C[1] = h_up; t.residual = nullptr;
    t.M = T; t.N = L->rank_in; t.K = L->hidden; t.x_dtype = x_dtype; t.c_dtype = BM_F16; t.status = L->status_dev;
    t.after = after; t.zero = zero; t.zero_n = zero_n;
    return launch_gemm_basis(t, 2, st);
  }
  GemmArgs g{};
  g.A[0] = g.A[1] = x;
  g.B[0] = L->vh_gate;
  g.B[1] = L->vh_up;
  g.C[0] = h_gate;
  g.C[1] = h_up;
  g.residual = nullptr;
  g.a_dtype = x_dtype;
  g.c_dtype = BM_F16;
  g.round_a_f16 = 0;
  g.M = T;
  g.N = L->rank_in;
  g.K = L->hidden;
  if (zero) BM_CUDA(cudaMemsetAsync(zero, 0, static_cast<size_t>(zero_n) * 16, st));
  return launch_gemm_nt(g, 2, st);
}

extern "C" int bm_basis_project(const bm_layer_t* L, const void* x, int x_dtype, int32_t T, uint16_t* h_gate,
                                uint16_t* h_up, void* stream) {
  bm::NvtxRange nvtx_range("bm_basis_project");
  return basis_project(L, x, x_dtype, T, h_gate, h_up, AFTER_ALL, nullptr, 0, static_cast<cudaStream_t>(stream));
}

// fixed-point accumulators -> fp32 rank_accum (deterministic mode)
__global__ void __launch_bounds__(256) acc64_to_f32_kernel(const long long* __restrict__ acc64, float* __restrict__ out, int64_t n) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n; i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    out[i] = static_cast<float>(static_cast<double>(acc64[i]) * (1.0 / static_cast<double>(ACC_FIXED_SCALE)));
}

static size_t experts_ws_need(const bm_layer_t* L, int32_t T) {
  return (L && L->deterministic) ? align_up(sizeof(long long) * static_cast<size_t>(T) * L->rank_out, 256) : 0;
}

extern "C" size_t bm_experts_workspace_bytes(const bm_layer_t* L, int32_t T, int32_t num_assign, int32_t path) {
  (void)num_assign; (void)path;
  return T > 0 ? experts_ws_need(L, T) : 0;
}

// Passes of `size` assignments that the experts need together, where each has a Poisson number of them, `load` on average (choices
// spread evenly over the experts): experts * sum over j of P(more than j * size).
int bm::expected_passes(int experts, double load, int size) {
  double passes = 0.0;
  if (size > load + 5.0 * std::sqrt(load) + 5.0) return static_cast<int>(experts * (1.0 - std::exp(-load)) + 0.5);      // one at most
  if (load > 32.0) {      // a normal number is close enough, and its sum has few terms
    for (int n = 0;; n += size) {
      const double more = 0.5 * std::erfc((n + 0.5 - load) / std::sqrt(2.0 * load));
      if (more < 1e-4) return static_cast<int>(experts * passes + 0.5);
      passes += more;
    }
  }
  double p = std::exp(-load), at_most = p;
  for (int n = 0, next = 0; 1.0 - at_most >= 1e-4;) {
    if (n == next) {
      passes += 1.0 - at_most;
      next += size;
    }
    at_most += p *= load / ++n;
  }
  return static_cast<int>(experts * passes + 0.5);
}
// What the two kernels of passes take, us, as a model: both are as slow as their longest CTA.  `slots`: row slots of a matrix in units of 256.
// The costs of a unit and of a tile are fits to the stage of twelve layer shapes (8 to 512 experts, 4 to 16 tiles, rank 128 to 384) at 3 to
// 32 assignments an expert (off by 4 to 8 %, most of it where the passes are about to need another round, so that each takes the mean of
// three numbers of passes); choices spread evenly.  With the tensor path's estimate (experts_tc.cu) they choose the kernel: over these
// shapes at 3 to 64 assignments an expert the layer call takes 1.003 of the fastest kernel's time, 1.008 where the experts' shares fall as
// rank^-0.5 and 1.035 as 1 / rank, which nobody on the host knows.
template <typename F>
static double mean_near(int passes, F tiles) {
  double sum = 0.0;
  for (const double q : {0.95, 1.0, 1.05}) sum += tiles(std::max(1, static_cast<int>(q * passes + 0.5)));
  return sum / 3.0;
}
// experts_decode_kernel: a first round is cut along the tiles, later ones are not.  A round of at most half of the grid has an SM to a CTA.
static double decode_us(const bm_layer* L, double load, double slots) {
  const int grid = L->dec_grid, tiles = L->n_tiles;
  const double longest = mean_near(expected_passes(L->num_experts, load, FAST_MAX_TOK), [&](int passes) {
    const int rest = passes % grid, full = passes / grid;
    if (full == 0) {
      const int split = std::min(tiles, grid / passes), per = (tiles + split - 1) / split;
      return 8 * passes * ((tiles + per - 1) / per) <= 3 * grid ? 0.5 * per : per;
    }
    return full * tiles + (rest == 0 ? 0.0 : 2 * rest <= grid ? 0.65 * tiles : tiles) + 0.9 * (full - (rest == 0));
  });
  return 5.0 + 2.0 * slots + 1.95 * (1.0 + slots) * longest * (L->dec_ctas == 1 ? 0.6 : 1.0);
}
// experts_batch_kernel: the last round is cut, evenly where that saves a tile, and a second unit costs nearly one.  Inside a call its start
// hides less behind the launches before it than the other one's (1.5 us).
static double batch_us(const bm_layer* L, double load, double slots) {
  const int grid = L->bat_grid, tiles = L->n_tiles;
  return 4.5 + 4.5 * slots + mean_near(expected_passes(L->num_experts, load, 2 * FAST_MAX_TOK), [&](int passes) {
    const int rest = passes % grid, full = passes / grid;
    const int split = rest ? std::min(tiles, grid / rest) : 1, per = (tiles + split - 1) / split;
    const bool even = rest && experts_batch_even_shares(rest * tiles, per, grid);
    const double last = rest == 0 ? 0.0 : even ? static_cast<double>(rest) * tiles / grid : full == 0 && 3 * rest * ((tiles + per - 1) / per) <= grid ? 0.5 * per : per;
    const int more = full - (rest == 0) + even;      // units after the first
    return (0.9 + 4.3 * slots) * (full * tiles + last) + 4.8 * slots * more;
  });
}
// The kernel for `expected` assignments of at most `num_assign`: the one with the smallest estimate that the layer allows.  us of the stage with passes of
// 8 / of 16 / on tcgen05: 128 experts of 6 tiles, 4 assignments each 18.9 / 22.2 / 38, 7 each 31.0 / 23.1 / 38, 14 each 31.5 / 31.2 / 38, 20 each
// 46.6 / 36.5 / 38.8, 28 each 57 / 38.8 / 39.5; 160 of 12 tiles, 8 each 56.3 / 48.4 / 74, 24 each 105 / 78.7 / 74.7; 16 of 4 tiles, 8 each 9.0 / 10.5 / 13, 32
// each 10.8 / 12.6 / 14.2; 512 of 4 tiles, 7 each 50.7 / 51.5 / 85, 20 each 99.9 / 82.8 / 85.8.
static int choose_path(const bm_layer* L, int32_t num_assign, int32_t expected, int* rows) {
  const double load = static_cast<double>(expected) / L->num_experts, slots = L->max_slots / 256.0;
  const bool decode = L->fast_ok && L->dec_ok && num_assign / FAST_MAX_TOK + L->num_experts < 60000;
  int path = BM_PATH_GENERIC;
  double best = std::numeric_limits<double>::infinity();
  auto take = [&](int candidate, double us) { if (us < best) { best = us; path = candidate; } };
  const bool tensor = L->fast_ok && experts_tc_fits(L);
  if (tensor && (load > 8.0 || !(decode || L->bat_ring))) take(BM_PATH_TENSOR, experts_tc_us(L, load, rows));
  if (load <= 64.0 || !tensor) {
    if (decode) take(BM_PATH_DECODE, decode_us(L, load, slots));
    if (L->bat_ring && (load > 4.0 || !decode)) take(BM_PATH_BATCH, batch_us(L, load, slots));      // (up to 4 one pass of 8 is enough for nearly every expert)
  }
  return path;
}

// `num_assign` bounds the list's length, `expected` is what the choice of a kernel takes it for.
static int experts_forward_impl(const bm_layer_t* L, const uint16_t* h_gate, const uint16_t* h_up,
                                const int32_t* token_indices, const int32_t* expert_offsets, const float* route_weights,
                                int32_t T, int32_t num_assign, int32_t expected, float* rank_accum, int32_t path, bool already_zero,
                                void* workspace, size_t workspace_bytes, void* stream) {
  BM_REQUIRE(L != nullptr, BM_ERR_INVALID_ARG, "experts_forward: null layer");
  BM_REQUIRE(T >= 0 && num_assign >= 0, BM_ERR_INVALID_ARG, "experts_forward: negative sizes");
  BM_REQUIRE(path >= BM_PATH_AUTO && path <= BM_PATH_BATCH, BM_ERR_INVALID_ARG, "experts_forward: unknown path %d", path);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (T == 0) return BM_OK;
  BM_REQUIRE(rank_accum, BM_ERR_INVALID_ARG, "experts_forward: null rank_accum");
  long long* acc64 = nullptr;
  const int64_t n_acc = static_cast<int64_t>(T) * L->rank_out;
  if (L->deterministic) {
    const size_t need = experts_ws_need(L, T);
    BM_REQUIRE(workspace && workspace_bytes >= need && (reinterpret_cast<uintptr_t>(workspace) & 15u) == 0, BM_ERR_WORKSPACE,
               "experts_forward: the deterministic mode needs a 16-byte aligned workspace of %zu bytes (%zu given)", need, workspace_bytes);
    acc64 = static_cast<long long*>(workspace);
    BM_CUDA(cudaMemsetAsync(acc64, 0, sizeof(long long) * static_cast<size_t>(n_acc), st));
  } else if (!already_zero) {
    BM_CUDA(cudaMemsetAsync(rank_accum, 0, sizeof(float) * static_cast<size_t>(n_acc), st));
  }
  int rc = BM_OK;
  if (num_assign == 0 || L->num_experts == 0) {
    if (acc64) BM_CUDA(cudaMemsetAsync(rank_accum, 0, sizeof(float) * static_cast<size_t>(n_acc), st));
    return BM_OK;
  }
  BM_REQUIRE(h_gate && h_up && token_indices && expert_offsets && route_weights, BM_ERR_INVALID_ARG,
             "experts_forward: null pointer");
  BM_REQUIRE(path != BM_PATH_TENSOR || L->fast_ok, BM_ERR_UNSUPPORTED,
             "experts_forward: the tensor path needs 1- to 4-bit rows and full tiles; this layer has neither");
  BM_REQUIRE(path != BM_PATH_DECODE || L->fast_ok, BM_ERR_UNSUPPORTED,
             "experts_forward: the decode path needs 1- to 4-bit rows and full tiles; this layer has neither");
  BM_REQUIRE(path != BM_PATH_BATCH || L->fast_ok, BM_ERR_UNSUPPORTED,
             "experts_forward: the batch path needs 1- to 4-bit rows and full tiles; this layer has neither");
  const __half* hg = reinterpret_cast<const __half*>(h_gate);
  const __half* hu = reinterpret_cast<const __half*>(h_up);
  int rows = 0;      // of the tensor path's CTAs, where the choice has looked at them
  if (path == BM_PATH_AUTO) path = choose_path(L, num_assign, expected, &rows);
  if (path == BM_PATH_TENSOR)
    rc = launch_experts_tc(L, hg, hu, token_indices, expert_offsets, route_weights, T, expected, rows, rank_accum, acc64, st);
  else if (path == BM_PATH_BATCH)
    rc = launch_experts_batch(L, hg, hu, token_indices, expert_offsets, route_weights, T, rank_accum, acc64, st);
  else if (path == BM_PATH_DECODE)
    rc = launch_experts_decode(L, hg, hu, token_indices, expert_offsets, route_weights, T, num_assign, rank_accum, acc64, st);
  else
    rc = launch_experts_generic(L, hg, hu, token_indices, expert_offsets, route_weights, T, rank_accum, acc64, st);
  if (rc) return rc;
  if (acc64) {
    const int blocks = static_cast<int>((n_acc + 255) / 256 < 148 * 8 ? (n_acc + 255) / 256 : 148 * 8);
    acc64_to_f32_kernel<<<blocks, 256, 0, st>>>(acc64, rank_accum, n_acc);
    BM_LAUNCH_CHECK("acc64_to_f32_kernel");
  }
  return BM_OK;
}

extern "C" int bm_experts_forward(const bm_layer_t* L, const uint16_t* h_gate, const uint16_t* h_up,
                                  const int32_t* token_indices, const int32_t* expert_offsets,
                                  const float* route_weights, int32_t T, int32_t num_assign, float* rank_accum,
                                  int32_t path, void* workspace, size_t workspace_bytes, void* stream) {
  bm::NvtxRange nvtx_range("bm_experts_forward");
  return experts_forward_impl(L, h_gate, h_up, token_indices, expert_offsets, route_weights, T, num_assign, num_assign, rank_accum, path,
                              false, workspace, workspace_bytes, stream);
}

extern "C" int bm_experts_forward_expecting(const bm_layer_t* L, const uint16_t* h_gate, const uint16_t* h_up,
                                            const int32_t* token_indices, const int32_t* expert_offsets,
                                            const float* route_weights, int32_t T, int32_t num_assign, int32_t num_expected,
                                            float* rank_accum, int32_t path, void* workspace, size_t workspace_bytes, void* stream) {
  bm::NvtxRange nvtx_range("bm_experts_forward");
  BM_REQUIRE(num_expected >= 0 && num_expected <= num_assign, BM_ERR_INVALID_ARG, "experts_forward: %d assignments expected of at most %d",
             num_expected, num_assign);
  return experts_forward_impl(L, h_gate, h_up, token_indices, expert_offsets, route_weights, T, num_assign, num_expected, rank_accum, path,
                              false, workspace, workspace_bytes, stream);
}

// y = fp16(rank_accum) . U_down^T (+ (z * sigmoid(gate)) . W_down^T of a shared expert) (+ residual), one launch.
static int combine_small(const bm_layer_t* L, const float* rank_accum, int T, const __half* w_down, int w_bf16, const float* z, const float* gate,
                         int inter, const void* residual, void* y, int y_dtype, bool overlap, cudaStream_t st) {
  SkinnyArgs a{};
  a.overlap = overlap;
  a.seg[0] = SkSeg{L->u_down, nullptr, y, L->hidden, y_dtype, 0, 0};
  a.n_seg = 1;
  a.X = rank_accum; a.N = T; a.K = L->rank_out; a.x_dtype = BM_F32;
  a.W2 = w_down; a.w2_bf16 = w_bf16; a.X2 = z; a.x2_gate = gate; a.K2 = inter;
  a.residual = residual;
  a.splits = 1;
  return launch_skinny_nt(a, st);
}

static int combine_down_basis(const bm_layer_t* L, const float* rank_accum, int32_t T, const void* residual, void* y, int y_dtype, LaunchAfter after,
                              cudaStream_t st) {
  BM_REQUIRE(L != nullptr, BM_ERR_INVALID_ARG, "combine: null layer");
  BM_REQUIRE(L->u_down, BM_ERR_INVALID_ARG, "missing shared_u_down for packed routed experts");
  BM_REQUIRE(T >= 0 && y_dtype >= BM_F16 && y_dtype <= BM_F32, BM_ERR_INVALID_ARG, "combine: bad arguments");
  if (T == 0) return BM_OK;
  BM_REQUIRE(rank_accum && y, BM_ERR_INVALID_ARG, "combine: null pointer");
  // Up to two chunks of 64 tokens go to the skinny product (us against the tiled one: 64 tokens 5.1 / 6.1, 128 tokens 6.1 / 6.1, 203 tokens 7.9 / 6.2).
  const bool tiled = L->rank_out % 64 == 0 && L->hidden % 8 == 0 && aligned16(rank_accum, L->u_down);
  if ((T <= 128 || (T <= SKINNY_MAX_TOKENS && !tiled)) && skinny_fits(L->rank_out, 0, 1)) {
    const int rc = combine_small(L, rank_accum, T, nullptr, 0, nullptr, nullptr, 0, residual, y, y_dtype, after != AFTER_ALL, st);
    if (rc != BM_ERR_UNSUPPORTED) return rc;
  }
  if (L->rank_out % 64 == 0 && aligned16(rank_accum, L->u_down)) {
    GemmTcArgs t{};
    t.X = rank_accum; t.W[0] = t.W[1] = L->u_down; t.C[0] = t.C[1] = y; t.residual = residual;
    t.M = T; t.N = L->hidden; t.K = L->rank_out; t.x_dtype = BM_F32; t.c_dtype = y_dtype; t.status = L->status_dev;
    t.after = after;
    return launch_gemm_basis(t, 1, st);
  }
  GemmArgs g{};
  g.A[0] = g.A[1] = rank_accum;
  g.B[0] = g.B[1] = L->u_down;
  g.C[0] = g.C[1] = y;
  g.residual = residual;
  g.a_dtype = BM_F32;
  g.c_dtype = y_dtype;
  g.round_a_f16 = 1;
  g.M = T;
  g.N = L->hidden;
  g.K = L->rank_out;
  return launch_gemm_nt(g, 1, st);
}

extern "C" int bm_combine_down_basis(const bm_layer_t* L, const float* rank_accum, int32_t T, const void* residual,
                                     void* y, int y_dtype, void* stream) {
  bm::NvtxRange nvtx_range("bm_combine_down_basis");
  return combine_down_basis(L, rank_accum, T, residual, y, y_dtype, AFTER_ALL, static_cast<cudaStream_t>(stream));
}

extern "C" size_t bm_layer_workspace_bytes(const bm_layer_t* L, int32_t T, int32_t k) {
  if (!L || T < 0 || k <= 0) return 0;
  return carve_layer_ws(L, nullptr, T, k).total;
}

// A decode batch in three or four launches, each starting while the one before drains:
//   1. everything that multiplies x -- the basis projection and, for a whole block, router logits, the shared expert's
//      gated pair and its token gate -- with the expert stage's accumulator cleared on the way; given logits are routed
//      by one more cluster of the same grid
//   2. routing of computed logits (whole block only)
//   3. packed experts
//   4. down basis, shared expert's down product and residual
// BM_ERR_UNSUPPORTED, with nothing launched, when a shape does not tile; the general path takes it.
//
// Up to how many tokens, where the chain of tiled products (forward_large, the general layer path) takes the sizes.  The limits are
// crossovers of three shapes of hidden size 2048, us a call of these launches / of the chain.  Layer of 128 experts, fp16: 56 tokens 29.8 / 31.3, 72 32.3 /
// 32.0, 112 37.8 / 36.2; of 64 experts, bf16, whose rows the chain rounds in shared memory: 112 tokens 36.5 / 37.4, 129 39.7 / 37.9.  Block of 128
// experts, bf16: 64 tokens 37.5 / 38.7, 80 39.8 / 39.2, 112 46.2 / 43.9; of 512 experts and a gated shared one: 40 tokens 52.7 / 53.5, 48 71.0 / 71.3, 64
// 80.1 / 73.1.  Other shapes cross elsewhere, as the first launch grows with rows, hidden size and chunks of 64 tokens and the routing cluster
// with tokens times experts.  Earlier: layers of 160 experts and hidden size 5120 (56 tokens 57.2 / 52.3, 112 83.6 / 71.6), of 512 experts (56: 54.5 /
// 49.3); blocks of 256 experts and hidden size 4096 (24: 66.4 / 65.1, 72: 140 / 98), of 160 and 5120 (48: 59.5 / 57.7, 72: 94.9 / 70.3); with a gated shared
// expert blocks of 16 to 128 experts (40: 36.9 / 34.2, 44.4 / 43.7, 46.4 / 44.1) and of 256 (24: 81.7 / 75.0, 40: 138 / 110).  Later, by 0.9 us at most: fp16
// layers of 16 and 64 experts up to 128 and 96 tokens.
static int small_tokens(const bm_layer_t* L, const bm_block_dense_t* d, int x_dtype) {
  const bool shared = d && d->sh_intermediate > 0;
  if (L->hidden % 64 != 0 || L->rank_in % 8 != 0 || L->rank_out % 64 != 0 || (shared && d->sh_intermediate % 64 != 0) || (d && L->num_experts % 8 != 0))
    return SKINNY_MAX_TOKENS;
  if (d) return shared ? 48 : 80;
  return x_dtype == BM_F16 ? 64 : 128;
}
static int forward_small(const bm_layer_t* L, const bm_block_dense_t* d, const void* x, int x_dtype, void* logits, int logits_dtype, int T,
                         int k, int renorm, int weight_round, const void* residual, void* y, int path, const LayerWs& w, float* z, float* gate,
                         cudaStream_t st) {
  const bool shared = d && d->sh_intermediate > 0;
  if (!x || !y || !logits || x_dtype < BM_F16 || x_dtype > BM_F32 || logits_dtype < BM_F16 || logits_dtype > BM_F32) return BM_ERR_UNSUPPORTED;
  if (T > small_tokens(L, d, x_dtype) || L->hidden % 128 != 0 || (reinterpret_cast<uintptr_t>(x) & 15u) || !L->vh_gate || !L->vh_up || !L->u_down ||
      !skinny_fits(L->hidden, 0, 8) || !skinny_fits(L->rank_out, shared ? d->sh_intermediate : 0, 1) || !route_small_fits(T, L->num_experts, k))
    return BM_ERR_UNSUPPORTED;
  auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  if (!aligned(L->vh_gate) || !aligned(L->vh_up) || !aligned(L->u_down)) return BM_ERR_UNSUPPORTED;
  if (d && !(aligned(d->gate_w) && aligned(d->sh_gate) && aligned(d->sh_up) && aligned(d->sh_down) && aligned(d->sh_token_gate)))
    return BM_ERR_UNSUPPORTED;
  const size_t acc_bytes = sizeof(float) * static_cast<size_t>(T) * L->rank_out;     // rank_out is a multiple of 16 here
  auto h = [](const uint16_t* p) { return reinterpret_cast<const __half*>(p); };
  RouteSmallArgs r{};
  r.logits = logits; r.logits_dtype = logits_dtype;
  r.T = T; r.E = L->num_experts; r.k = k; r.renorm = renorm; r.weight_round = weight_round;
  r.token_indices = w.token_indices; r.expert_offsets = w.expert_offsets; r.route_flat = w.route_flat;
  SkinnyArgs a{};
  const int bf16 = d && d->w_dtype == BM_BF16;
  int n = 0;
  if (d) a.seg[n++] = SkSeg{h(d->gate_w), nullptr, logits, L->num_experts, logits_dtype, bf16, 0};
  a.seg[n++] = SkSeg{L->vh_gate, nullptr, w.h_gate, L->rank_in, BM_F16, 0, 0};
  a.seg[n++] = SkSeg{L->vh_up, nullptr, w.h_up, L->rank_in, BM_F16, 0, 0};
  if (shared) {
    a.seg[n++] = SkSeg{h(d->sh_gate), h(d->sh_up), z, d->sh_intermediate, BM_F32, bf16, 0};
    if (d->sh_token_gate) a.seg[n++] = SkSeg{h(d->sh_token_gate), nullptr, gate, 1, BM_F32, bf16, 0};
  }
  a.n_seg = n;
  a.X = x; a.N = T; a.K = L->hidden; a.x_dtype = x_dtype; a.splits = 8;
  a.zero = reinterpret_cast<float4*>(w.rank_accum); a.zero_n = static_cast<int>(acc_bytes / 16);
  if (!d) a.route = r;
  int rc = launch_skinny_nt(a, st);
  if (rc) return rc;
  if (d && (rc = launch_route_small(r, st))) return rc;
  rc = experts_forward_impl(L, reinterpret_cast<const uint16_t*>(w.h_gate), reinterpret_cast<const uint16_t*>(w.h_up), w.token_indices,
                            w.expert_offsets, w.route_flat, T, T * k, T * k, w.rank_accum, path, true, w.experts_ws, w.experts_ws_bytes, st);
  if (rc) return rc;
  return combine_small(L, w.rank_accum, T, shared ? h(d->sh_down) : nullptr, bf16, z, shared && d->sh_token_gate ? gate : nullptr,
                       shared ? d->sh_intermediate : 0, residual, y, x_dtype, true, st);
}

// Assignments of T tokens that the packed experts get where choices spread evenly over the routed ones.
static int32_t expected_assign(const bm_layer_t* L, int32_t T, int32_t k, int32_t num_routed) {
  return static_cast<int32_t>(static_cast<int64_t>(T) * k * std::min(L->num_experts, num_routed) / num_routed);
}

extern "C" int bm_layer_forward(const bm_layer_t* L, const void* x, int x_dtype, const void* logits, int logits_dtype,
                                int32_t T, int32_t num_routed, int32_t k, int32_t renorm, int32_t weight_round,
                                const int32_t* global_to_local, const void* residual, void* y, int32_t path,
                                void* workspace, size_t workspace_bytes, void* stream) {
  bm::NvtxRange nvtx_range("bm_layer_forward");
  BM_REQUIRE(L != nullptr, BM_ERR_INVALID_ARG, "layer_forward: null layer");
  BM_REQUIRE(T >= 0 && k > 0 && num_routed > 0, BM_ERR_INVALID_ARG, "layer_forward: bad sizes");
  BM_REQUIRE(global_to_local != nullptr || num_routed == L->num_experts, BM_ERR_INVALID_ARG,
             "layer_forward: %d routed experts but %d packed and no id map", num_routed, L->num_experts);
  if (T == 0) return BM_OK;
  const LayerWs w = carve_layer_ws(L, workspace, T, k);
  BM_REQUIRE(workspace && workspace_bytes >= w.total && (reinterpret_cast<uintptr_t>(workspace) & 255u) == 0,
             BM_ERR_WORKSPACE, "layer_forward: workspace must be 256-byte aligned and hold %zu bytes (%zu given)", w.total,
             workspace_bytes);
  if (global_to_local == nullptr) {
    const int rc = forward_small(L, nullptr, x, x_dtype, const_cast<void*>(logits), logits_dtype, T, k, renorm, weight_round, residual, y, path,
                                 w, nullptr, nullptr, static_cast<cudaStream_t>(stream));
    if (rc != BM_ERR_UNSUPPORTED) return rc;
  }
  // One stream, every launch set up while the one before it runs.  The basis projection depends only on x and runs beside the
  // routing's placement, which takes a cluster; the accumulator of the expert stage is cleared by its idle warps.
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int rc = route_tokens(logits, logits_dtype, T, num_routed, k, renorm, weight_round, global_to_local, L->num_experts, TILE_ROWS, w.topk_idx, w.topk_w,
                        w.token_indices, w.expert_offsets, w.route_flat, /*tile_table=*/nullptr, /*counts=*/nullptr, w.route_ws, w.route_ws_bytes,
                        AFTER_ALL, /*beside_follows=*/true, st);
  if (rc) return rc;
  const size_t acc_bytes = sizeof(float) * static_cast<size_t>(T) * L->rank_out;
  const bool zeroed = acc_bytes % 16 == 0;
  rc = basis_project(L, x, x_dtype, T, reinterpret_cast<uint16_t*>(w.h_gate), reinterpret_cast<uint16_t*>(w.h_up), AFTER_BESIDE,
                     zeroed ? reinterpret_cast<float4*>(w.rank_accum) : nullptr, static_cast<int64_t>(acc_bytes / 16), st);
  if (rc) return rc;
  // Dropped assignments (experts that are not packed) leave a shorter list; the kernels walk
  // expert_offsets, so passing the upper bound T*k as num_assign is safe.  The kernel is chosen for the packed experts' share of the
  // routed ones (a shard of 64 of 128 experts, 96 tokens, top 8: six each, not twelve; stage 17.4 -> 15.0 us).
  rc = experts_forward_impl(L, reinterpret_cast<const uint16_t*>(w.h_gate), reinterpret_cast<const uint16_t*>(w.h_up),
                            w.token_indices, w.expert_offsets, w.route_flat, T, T * k, expected_assign(L, T, k, num_routed), w.rank_accum, path, zeroed, w.experts_ws,
                            w.experts_ws_bytes, stream);
  if (rc) return rc;
  return combine_down_basis(L, w.rank_accum, T, residual, y, x_dtype == BM_F32 ? BM_F32 : x_dtype, AFTER_READS, st);
}

// bf16 weights -> fp16, several matrices per launch (piece i: n[i] groups of eight values)
struct CastArgs { const uint4* src[5]; uint4* dst[5]; int n[5]; };
__global__ void __launch_bounds__(256) cast_weights_kernel(const __grid_constant__ CastArgs a) {
  const int p = blockIdx.y;
  grid_launch_dependents();
  for (int i = blockIdx.x * 256 + threadIdx.x; i < a.n[p]; i += gridDim.x * 256) {
    uint4 v = __ldg(a.src[p] + i);
    uint32_t* o = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const __half2 h = __floats2half2_rn(__uint_as_float(o[j] << 16), __uint_as_float(o[j] & 0xffff0000u));
      o[j] = *reinterpret_cast<const uint32_t*>(&h);
    }
    a.dst[p][i] = v;
  }
}

// Extra workspace of a block on the general path: the shared expert's contribution (y is written by the last launch
// only), its intermediates, and fp16 copies of bf16 weights.
struct BlockWs { void* res; void* dense_ws; size_t dense_ws_bytes; uint16_t* w[5]; size_t total; };
static BlockWs carve_block_ws(const bm_layer_t* L, const bm_block_dense_t* d, int num_routed, void* base, int T) {
  Carver c(base, 0);
  BlockWs w{};
  const size_t H = static_cast<size_t>(L->hidden), I = d->sh_intermediate > 0 ? d->sh_intermediate : 0;
  if (I) {
    w.res = c.take<uint16_t>(static_cast<size_t>(T) * H);
    w.dense_ws_bytes = bm_dense_mlp_workspace_bytes(T, static_cast<int32_t>(I));
    w.dense_ws = c.take<unsigned char>(w.dense_ws_bytes);
  }
  if (d->w_dtype == BM_BF16) {
    const size_t n[5] = {static_cast<size_t>(num_routed) * H, I * H, I * H, I * H, H};
    for (int i = 0; i < 5; ++i) w.w[i] = c.take<uint16_t>(n[i]);
  }
  w.total = c.off;
  return w;
}

// A prefill batch of a whole block: everything that multiplies x in one launch (router logits, basis projection, the shared
// expert's gated pair), routing, packed experts, and both down products in one launch.  BM_ERR_UNSUPPORTED, with nothing
// launched that matters, when a shape or pointer does not suit the tiled-copy GEMM.
static int forward_large(const bm_layer_t* L, const bm_block_dense_t& d, const void* x, int x_dtype, int T, int num_routed, int k, int renorm,
                         int weight_round, const int32_t* global_to_local, void* logits, void* y, const LayerWs& w, const BlockWs& b,
                         const uint16_t* token_gate, int token_gate_dtype, LaunchAfter after, cudaStream_t st) {
  const bool shared = d.sh_intermediate > 0;
  if (!L->vh_gate || !L->vh_up || !L->u_down || L->rank_out % 64 != 0 || (shared && d.sh_intermediate % 64 != 0)) return BM_ERR_UNSUPPORTED;
  auto h = [](const uint16_t* p) { return reinterpret_cast<const __half*>(p); };
  const size_t mat = shared ? align_up(static_cast<size_t>(T) * d.sh_intermediate * 2, 256) : 0;
  __half* z = static_cast<__half*>(b.dense_ws);
  float* gate = reinterpret_cast<float*>(static_cast<unsigned char*>(b.dense_ws) + 3 * mat);
  int rc;
  if (shared && d.sh_token_gate) {
    if ((rc = launch_row_gate(x, x_dtype, token_gate, token_gate_dtype, T, L->hidden, gate, after == AFTER_ALL ? AFTER_ALL : AFTER_BESIDE, st))) return rc;
    after = AFTER_READS;
  }
  GemmTmaArgs a{};
  a.X = x; a.x_dtype = x_dtype; a.M = T; a.K = L->hidden; a.status = L->status_dev;
  a.seg[0] = GemmSeg{h(d.gate_w), nullptr, logits, num_routed, x_dtype};
  a.seg[1] = GemmSeg{L->vh_gate, nullptr, w.h_gate, L->rank_in, BM_F16};
  a.seg[2] = GemmSeg{L->vh_up, nullptr, w.h_up, L->rank_in, BM_F16};
  if (shared) a.seg[3] = GemmSeg{h(d.sh_gate), h(d.sh_up), z, d.sh_intermediate, BM_F16};
  a.n_seg = shared ? 4 : 3;
  a.row_gate = shared && d.sh_token_gate ? gate : nullptr;
  a.after = after;
  a.zero = reinterpret_cast<float4*>(w.rank_accum); a.zero_n = static_cast<int64_t>(T) * L->rank_out / 4;      // (rank_out is a multiple of 64)
  if ((rc = launch_gemm_tma(a, st))) return rc;
  rc = route_tokens(logits, x_dtype, T, num_routed, k, renorm, weight_round, global_to_local, L->num_experts, TILE_ROWS, w.topk_idx, w.topk_w,
                    w.token_indices, w.expert_offsets, w.route_flat, nullptr, nullptr, w.route_ws, w.route_ws_bytes, AFTER_READS, /*beside_follows=*/false, st);
  if (rc) return rc;
  rc = experts_forward_impl(L, reinterpret_cast<const uint16_t*>(w.h_gate), reinterpret_cast<const uint16_t*>(w.h_up), w.token_indices,
                            w.expert_offsets, w.route_flat, T, T * k, expected_assign(L, T, k, num_routed), w.rank_accum, BM_PATH_AUTO, true, w.experts_ws, w.experts_ws_bytes, st);
  if (rc) return rc;
  GemmTmaArgs c{};
  c.X = w.rank_accum; c.x_dtype = BM_F32; c.M = T; c.K = L->rank_out; c.status = L->status_dev;
  c.seg[0] = GemmSeg{L->u_down, nullptr, y, L->hidden, x_dtype};
  c.n_seg = 1;
  c.after = AFTER_READS;
  if (shared) { c.X2 = z; c.W2 = h(d.sh_down); c.K2 = d.sh_intermediate; }
  rc = launch_gemm_tma(c, st);
  if (rc != BM_ERR_UNSUPPORTED) return rc;
  // y's rows do not suit tiled copies: the shared expert's product first, then the other one on top
  if (shared) {
    GemmTcArgs t{};
    t.X = z; t.W[0] = t.W[1] = h(d.sh_down); t.C[0] = t.C[1] = b.res; t.M = T; t.N = L->hidden; t.K = d.sh_intermediate;
    t.x_dtype = BM_F16; t.c_dtype = x_dtype; t.status = L->status_dev;
    if ((rc = launch_gemm_tc(t, 1, st))) return rc;
  }
  return bm_combine_down_basis(L, w.rank_accum, T, shared ? b.res : nullptr, y, x_dtype, st);
}

extern "C" size_t bm_block_workspace_bytes(const bm_layer_t* L, const bm_block_dense_t* d, int32_t num_routed, int32_t T, int32_t k) {
  if (!L || !d || T < 0 || k <= 0) return 0;
  return carve_layer_ws(L, nullptr, T, k).total + carve_block_ws(L, d, num_routed, nullptr, T).total;
}

extern "C" int bm_block_forward(const bm_layer_t* L, const bm_block_dense_t* dense, const void* x, int x_dtype, int32_t T, int32_t num_routed,
                                int32_t k, int32_t renorm, int32_t weight_round, const int32_t* global_to_local, void* logits, void* y,
                                void* workspace, size_t workspace_bytes, void* stream) {
  bm::NvtxRange nvtx_range("bm_block_forward");
  BM_REQUIRE(L != nullptr && dense != nullptr && dense->gate_w != nullptr, BM_ERR_INVALID_ARG, "block_forward: null layer or router");
  BM_REQUIRE(T >= 0 && k > 0 && num_routed > 0 && (x_dtype == BM_F16 || x_dtype == BM_BF16) &&
                 (dense->w_dtype == BM_F16 || dense->w_dtype == BM_BF16),
             BM_ERR_INVALID_ARG, "block_forward: bad arguments");
  bm_block_dense_t d = *dense;
  const bool shared = d.sh_intermediate > 0;
  BM_REQUIRE(!shared || (d.sh_gate && d.sh_up && d.sh_down && d.sh_intermediate % 2 == 0), BM_ERR_INVALID_ARG,
             "block_forward: incomplete shared expert");
  BM_REQUIRE(global_to_local != nullptr || num_routed == L->num_experts, BM_ERR_INVALID_ARG,
             "block_forward: %d routed experts but %d packed and no id map", num_routed, L->num_experts);
  if (T == 0) return BM_OK;
  BM_REQUIRE(x && logits && y, BM_ERR_INVALID_ARG, "block_forward: null pointer");
  const LayerWs w = carve_layer_ws(L, workspace, T, k);
  const BlockWs b = carve_block_ws(L, &d, num_routed, static_cast<unsigned char*>(workspace) + w.total, T);
  BM_REQUIRE(workspace && workspace_bytes >= w.total + b.total && (reinterpret_cast<uintptr_t>(workspace) & 255u) == 0, BM_ERR_WORKSPACE,
             "block_forward: workspace must be 256-byte aligned and hold %zu bytes (%zu given)", w.total + b.total, workspace_bytes);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (global_to_local == nullptr) {
    // z fp32 [T, intermediate] fits the g and u areas of the shared expert's workspace, the token gate behind it in z's
    float* z = static_cast<float*>(b.dense_ws);
    float* gate = shared ? z + align_up(static_cast<size_t>(T) * d.sh_intermediate, 64) : nullptr;
    const int rc = forward_small(L, &d, x, x_dtype, logits, x_dtype, T, k, renorm, weight_round, nullptr, y, BM_PATH_AUTO, w, z, gate, st);
    if (rc != BM_ERR_UNSUPPORTED) return rc;
  }
  if (d.w_dtype == BM_BF16) {
    const size_t H = static_cast<size_t>(L->hidden), I = shared ? d.sh_intermediate : 0;
    BM_REQUIRE(H % 8 == 0, BM_ERR_UNSUPPORTED, "block_forward: hidden=%d must be a multiple of 8 with bf16 weights", L->hidden);
    const uint16_t** src[5] = {&d.gate_w, &d.sh_gate, &d.sh_up, &d.sh_down, &d.sh_token_gate};
    const size_t n[5] = {static_cast<size_t>(num_routed) * H, I * H, I * H, I * H, H};
    CastArgs c{};
    for (int i = 0; i < 5; ++i) {
      if (!*src[i] || (i > 0 && !shared)) continue;
      BM_REQUIRE((reinterpret_cast<uintptr_t>(*src[i]) & 15u) == 0, BM_ERR_UNSUPPORTED, "block_forward: bf16 weights must be 16-byte aligned");
      c.src[i] = reinterpret_cast<const uint4*>(*src[i]);
      c.dst[i] = reinterpret_cast<uint4*>(b.w[i]);
      c.n[i] = static_cast<int>(n[i] / 8);
      *src[i] = b.w[i];
    }
    cast_weights_kernel<<<dim3(148, 5), 256, 0, st>>>(c);
    BM_LAUNCH_CHECK("cast_weights_kernel");
  }
  int rc = forward_large(L, d, x, x_dtype, T, num_routed, k, renorm, weight_round, global_to_local, logits, y, w, b, dense->sh_token_gate, d.w_dtype,
                         d.w_dtype == BM_BF16 ? AFTER_READS : AFTER_ALL, st);
  if (rc != BM_ERR_UNSUPPORTED) return rc;
  rc = bm_gate_logits(x, x_dtype, d.gate_w, T, num_routed, L->hidden, logits, x_dtype, stream);
  if (rc) return rc;
  if (shared) {
    rc = bm_dense_mlp_forward(x, x_dtype, d.sh_gate, d.sh_up, d.sh_down, d.sh_token_gate, T, L->hidden, d.sh_intermediate, nullptr, b.res,
                              x_dtype, b.dense_ws, b.dense_ws_bytes, stream);
    if (rc) return rc;
  }
  return bm_layer_forward(L, x, x_dtype, logits, x_dtype, T, num_routed, k, renorm, weight_round, global_to_local, b.res, y, BM_PATH_AUTO,
                          workspace, w.total, stream);
}
