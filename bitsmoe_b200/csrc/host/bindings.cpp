// Host side of the calls a serving loop makes per layer and step: argument checks, output allocation, workspace lookup
// and the call into the C ABI, as CPython functions.  A decode step launches a few kernels of some microseconds each, so
// the Python that used to stand here (ctypes argument conversion, device context managers, tensor methods: about 25 us a
// layer) cost as much as the GPU work; here it is about 3 us plus the launches.
//
// The semantics are those of bitsmoe_b200/layer.py, which calls these functions.
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "../../../include/bitsmoe_b200.h"

namespace {

// A Python exception is set; unwinds to the function's entry.
struct PyError {};

void check(int status) {
  if (status == BM_OK) return;
  PyObject* mod = PyImport_ImportModule("bitsmoe_b200.capi");
  PyObject* r = mod ? PyObject_CallMethod(mod, "check", "i", status) : nullptr;     // raises BitsMoEError
  Py_XDECREF(r);
  Py_XDECREF(mod);
  if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, bm_last_error());
  throw PyError();
}

[[noreturn]] void fail(PyObject* type, const std::string& msg) {
  PyErr_SetString(type, msg.c_str());
  throw PyError();
}

const at::Tensor& tensor(PyObject* o) {
  if (!THPVariable_Check(o)) fail(PyExc_TypeError, "expected a tensor");
  return THPVariable_Unpack(o);
}
at::Tensor opt_tensor(PyObject* o) { return o == Py_None ? at::Tensor() : tensor(o); }
long integer(PyObject* o) {
  const long v = PyLong_AsLong(o);
  if (v == -1 && PyErr_Occurred()) throw PyError();
  return v;
}

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kHalf: return BM_F16;
    case at::kBFloat16: return BM_BF16;
    case at::kFloat: return BM_F32;
    default: fail(PyExc_TypeError, std::string("unsupported activation dtype ") + at::toString(t));
  }
}

void* ptr(const at::Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
const uint16_t* wptr(const at::Tensor& t) { return static_cast<const uint16_t*>(ptr(t)); }

// What a PackedLayer keeps on this side: its C handle and the workspaces of the shapes it has met.
struct HostLayer {
  bm_layer_t* handle = nullptr;
  c10::Device device{c10::kCUDA, 0};
  int64_t hidden = 0, rank_in = 0, rank_out = 0, experts = 0;      // hidden 0: the layer has no basis matrices
  struct Ws { int64_t T, k, variant; at::Tensor buf; c10::cuda::CUDAStream stream; };
  std::vector<Ws> ws;

  // A buffer may be dropped here while calls of another stream than the one it was made on still use it: the allocator
  // learns of every such stream.  A captured call gets one of its own from the graph's pool: the graph uses it as long as it
  // lives, whatever is dropped here.
  at::Tensor workspace(int64_t T, int64_t k, int64_t variant, size_t need_if_new(const HostLayer&, int64_t, int64_t, const void*), const void* arg) {
    const c10::cuda::CUDAStream now = c10::cuda::getCurrentCUDAStream(device.index());
    const bool captured = c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None;
    for (Ws& w : ws)
      if (!captured && w.T == T && w.k == k && w.variant == variant) {
        if (w.stream != now) {
          w.buf.record_stream(now.unwrap());
          w.stream = now;
        }
        return w.buf;
      }
    const size_t need = need_if_new(*this, T, k, arg);
    at::Tensor buf = at::empty({static_cast<int64_t>(need < 256 ? 256 : need)}, at::TensorOptions().dtype(at::kByte).device(device));
    if (captured) return buf;
    if (ws.size() > 8) ws.clear();
    ws.push_back(Ws{T, k, variant, buf, now});
    return buf;
  }
};

constexpr const char* CAPSULE = "bitsmoe_b200.layer";
HostLayer* layer_of(PyObject* o) {
  auto* L = static_cast<HostLayer*>(PyCapsule_GetPointer(o, CAPSULE));
  if (!L) throw PyError();
  if (!L->handle) fail(PyExc_RuntimeError, "the packed layer is closed");
  return L;
}

at::Tensor contiguous(const at::Tensor& t) { return t.is_contiguous() ? t : t.contiguous(); }
void require_cuda(const at::Tensor& t, const char* what) {
  if (!t.is_cuda()) fail(PyExc_RuntimeError, std::string(what) + " requires CUDA tensors; there is no CPU path");
}
// The library takes pointers: what a tensor has to hold is checked here, where its size is known.
void require(bool ok, const char* msg) {
  if (!ok) fail(PyExc_RuntimeError, msg);
}
void require_matrix(const at::Tensor& t, int64_t rows, int64_t cols, const char* msg) {
  require(t.dim() == 2 && t.size(0) == rows && t.size(1) == cols, msg);
}
void require_residual(const at::Tensor& residual, const at::Tensor& x) {
  require(!residual.defined() || (residual.device() == x.device() && residual.numel() == x.numel()), "residual must have x's elements and device");
}
void require_map(const at::Tensor& g2l, int64_t num_routed, c10::Device device) {
  require(!g2l.defined() || (g2l.scalar_type() == at::kInt && g2l.is_contiguous() && g2l.device() == device && g2l.numel() >= num_routed),
          "global_to_local must be a contiguous int32 entry for every routed expert, on the layer's device");
}
void* stream_of(c10::Device d) { return c10::cuda::getCurrentCUDAStream(d.index()).stream(); }

template <typename F>
PyObject* guarded(F&& f) {
  try {
    return f();
  } catch (const PyError&) {
    return nullptr;
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

void need_args(Py_ssize_t got, Py_ssize_t want) {
  if (got != want) fail(PyExc_TypeError, "wrong number of arguments");
}

// ---- layers
PyObject* layer_new(PyObject*, PyObject* const* a, Py_ssize_t n) {      // (handle, device index, hidden, rank_in, rank_out, experts)
  return guarded([&] {
    need_args(n, 6);
    HostLayer made;
    made.handle = static_cast<bm_layer_t*>(PyLong_AsVoidPtr(a[0]));
    made.device = c10::Device(c10::kCUDA, static_cast<c10::DeviceIndex>(integer(a[1])));
    made.hidden = integer(a[2]); made.rank_in = integer(a[3]); made.rank_out = integer(a[4]); made.experts = integer(a[5]);
    auto* L = new HostLayer(std::move(made));
    return PyCapsule_New(L, CAPSULE, [](PyObject* o) { delete static_cast<HostLayer*>(PyCapsule_GetPointer(o, CAPSULE)); });
  });
}
PyObject* layer_close(PyObject*, PyObject* const* a, Py_ssize_t n) {    // (layer): the handle is gone, buffers are given back
  return guarded([&]() -> PyObject* {
    need_args(n, 1);
    auto* L = static_cast<HostLayer*>(PyCapsule_GetPointer(a[0], CAPSULE));
    if (!L) throw PyError();
    L->handle = nullptr;
    L->ws.clear();
    Py_RETURN_NONE;
  });
}
PyObject* layer_drop_workspaces(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need_args(n, 1);
    layer_of(a[0])->ws.clear();
    Py_RETURN_NONE;
  });
}
size_t layer_ws_need(const HostLayer& L, int64_t T, int64_t k, const void*) {
  return bm_layer_workspace_bytes(L.handle, static_cast<int32_t>(T), static_cast<int32_t>(k));
}
PyObject* layer_workspace(PyObject*, PyObject* const* a, Py_ssize_t n) {    // (layer, T, k)
  return guarded([&] {
    need_args(n, 3);
    HostLayer* L = layer_of(a[0]);
    return THPVariable_Wrap(L->workspace(integer(a[1]), integer(a[2]), 0, layer_ws_need, nullptr));
  });
}

// (layer, x, logits, top_k, renorm, round code, residual, global_to_local, path, out) -> y
PyObject* layer_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    need_args(n, 10);
    HostLayer* L = layer_of(a[0]);
    const at::Tensor x = contiguous(tensor(a[1])), logits = contiguous(tensor(a[2]));
    require_cuda(x, "forward");
    require_cuda(logits, "forward");
    require(x.device() == L->device && logits.device() == L->device, "forward: x and logits must be on the layer's device");
    require(x.dim() >= 1 && logits.dim() == 2 && logits.size(0) == x.size(0), "forward: x [T, H] and logits [T, E] must have the same tokens");
    const int32_t k = static_cast<int32_t>(integer(a[3]));
    const int64_t T = x.size(0);
    require(L->hidden == 0 || x.numel() == T * L->hidden, "forward: the rows of x do not have the layer's hidden size");
    const int xd = dtype_code(x.scalar_type()), ld = dtype_code(logits.scalar_type());
    at::Tensor residual = opt_tensor(a[6]);
    const at::Tensor g2l = opt_tensor(a[7]), out = opt_tensor(a[9]);
    require_residual(residual, x);
    require_map(g2l, logits.size(1), L->device);
    require(!out.defined() || (out.scalar_type() == x.scalar_type() && out.device() == x.device() && out.is_contiguous() && out.numel() == x.numel()),
            "forward: out must be contiguous, of x's type and device, and hold x's elements");
    const c10::cuda::CUDAGuard guard(L->device);
    const at::Tensor y = out.defined() ? out : at::empty_like(x);
    if (residual.defined()) residual = contiguous(residual.scalar_type() == x.scalar_type() ? residual : residual.to(x.scalar_type()));
    const at::Tensor ws = L->workspace(T, k, 0, layer_ws_need, nullptr);
    check(bm_layer_forward(L->handle, x.data_ptr(), xd, logits.data_ptr(), ld, static_cast<int32_t>(T), static_cast<int32_t>(logits.size(1)), k,
                           integer(a[4]) != 0, static_cast<int32_t>(integer(a[5])), static_cast<const int32_t*>(ptr(g2l)), ptr(residual),
                           y.data_ptr(), static_cast<int32_t>(integer(a[8])), ws.data_ptr(), ws.nbytes(), stream_of(L->device)));
    return THPVariable_Wrap(y);
  });
}

struct BlockNeed { const bm_block_dense_t* d; int32_t routed; };
size_t block_ws_need(const HostLayer& L, int64_t T, int64_t k, const void* p) {
  const auto* b = static_cast<const BlockNeed*>(p);
  return bm_block_workspace_bytes(L.handle, b->d, b->routed, static_cast<int32_t>(T), static_cast<int32_t>(k));
}

// Whether the block's dense weights can be handed to bm_block_forward as they are: one 16-bit type, contiguous, aligned.
bool block_weights_ok(const at::Tensor* w, int n, const at::Tensor& x) {
  const auto type = w[0].scalar_type();
  if (type != at::kHalf && type != at::kBFloat16) return false;
  for (int i = 0; i < n; ++i)
    if (w[i].defined() && (w[i].scalar_type() != type || !w[i].is_contiguous() || w[i].device() != x.device() ||
                           (reinterpret_cast<uintptr_t>(w[i].data_ptr()) & 15u)))
      return false;
  return true;
}

// (layer, x [..., H], gate, sh_gate, sh_up, sh_down, sh_token_gate, top_k, renorm, round code, global_to_local) -> (y, logits),
// or None when the weights do not suit the one-call forward
PyObject* block_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need_args(n, 11);
    HostLayer* L = layer_of(a[0]);
    const at::Tensor x = contiguous(tensor(a[1]));
    const at::Tensor w[5] = {tensor(a[2]), opt_tensor(a[3]), opt_tensor(a[4]), opt_tensor(a[5]), opt_tensor(a[6])};
    if ((x.scalar_type() != at::kHalf && x.scalar_type() != at::kBFloat16) || !x.is_cuda() || x.device() != L->device ||
        !block_weights_ok(w, 5, x) || x.dim() < 2 || w[0].dim() != 2 || x.size(-1) == 0 || x.size(-1) % 8 != 0)
      Py_RETURN_NONE;
    bm_block_dense_t d{};
    d.gate_w = wptr(w[0]);
    d.sh_gate = wptr(w[1]); d.sh_up = wptr(w[2]); d.sh_down = wptr(w[3]); d.sh_token_gate = wptr(w[4]);
    d.sh_intermediate = w[1].defined() ? static_cast<int32_t>(w[1].size(0)) : 0;
    d.w_dtype = dtype_code(w[0].scalar_type());
    const int64_t H = x.size(-1), T = x.numel() / H, E = w[0].size(0), I = d.sh_intermediate;
    require(L->hidden == 0 || H == L->hidden, "block_forward: the rows of x do not have the layer's hidden size");
    require_matrix(w[0], E, H, "block_forward: the router weight must be [experts, hidden]");
    if (w[1].defined()) require_matrix(w[1], I, H, "block_forward: the shared gate weight must be [intermediate, hidden]");
    if (w[2].defined()) require_matrix(w[2], I, H, "block_forward: the shared up weight must be [intermediate, hidden]");
    if (w[3].defined()) require_matrix(w[3], H, I, "block_forward: the shared down weight must be [hidden, intermediate]");
    require(!w[4].defined() || w[4].numel() == H, "block_forward: the token gate's weight must have hidden elements");
    const int32_t k = static_cast<int32_t>(integer(a[7]));
    const at::Tensor g2l = opt_tensor(a[10]);
    require_map(g2l, E, L->device);
    const c10::cuda::CUDAGuard guard(L->device);
    const at::Tensor y = at::empty_like(x), logits = at::empty({T, E}, x.options());
    const BlockNeed need{&d, static_cast<int32_t>(E)};
    const int64_t variant = 1 + 2 * d.sh_intermediate + (d.w_dtype == BM_BF16);
    const at::Tensor ws = L->workspace(T, k, variant, block_ws_need, &need);
    check(bm_block_forward(L->handle, &d, x.data_ptr(), dtype_code(x.scalar_type()), static_cast<int32_t>(T), static_cast<int32_t>(E), k,
                           integer(a[8]) != 0, static_cast<int32_t>(integer(a[9])), static_cast<const int32_t*>(ptr(g2l)), logits.data_ptr(),
                           y.data_ptr(), ws.data_ptr(), ws.nbytes(), stream_of(L->device)));
    PyObject* py = THPVariable_Wrap(y);
    PyObject* pl = THPVariable_Wrap(logits);
    PyObject* r = py && pl ? PyTuple_Pack(2, py, pl) : nullptr;
    Py_XDECREF(py);
    Py_XDECREF(pl);
    return r;
  });
}

// (x, w_gate, w_up, w_down, token_gate | None, residual | None) -> y; weights fp16, contiguous, on x's device
PyObject* dense_mlp(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    need_args(n, 6);
    const at::Tensor x = contiguous(tensor(a[0]));
    require_cuda(x, "dense_mlp");
    const c10::cuda::CUDAGuard guard(x.device());
    auto half = [&](const at::Tensor& t) {
      return t.scalar_type() == at::kHalf && t.device() == x.device() && t.is_contiguous() ? t : t.detach().to(x.device(), at::kHalf).contiguous();
    };
    const at::Tensor wg = half(tensor(a[1])), wu = half(tensor(a[2])), wd = half(tensor(a[3]));
    const at::Tensor tg = a[4] == Py_None ? at::Tensor() : half(tensor(a[4]));
    at::Tensor residual = opt_tensor(a[5]);
    require(x.dim() == 2 && wg.dim() == 2, "dense_mlp: x must be [T, H] and the gate weight [I, H]");
    const int32_t T = static_cast<int32_t>(x.size(0)), H = static_cast<int32_t>(x.size(1)), I = static_cast<int32_t>(wg.size(0));
    require_matrix(wg, I, H, "dense_mlp: the gate weight must be [intermediate, hidden]");
    require_matrix(wu, I, H, "dense_mlp: the up weight must be [intermediate, hidden]");
    require_matrix(wd, H, I, "dense_mlp: the down weight must be [hidden, intermediate]");
    require(!tg.defined() || tg.numel() == H, "dense_mlp: the token gate's weight must have hidden elements");
    require_residual(residual, x);
    const int xd = dtype_code(x.scalar_type());
    const at::Tensor y = at::empty_like(x);
    if (residual.defined()) residual = contiguous(residual.scalar_type() == x.scalar_type() ? residual : residual.to(x.scalar_type()));
    const size_t need = bm_dense_mlp_workspace_bytes(T, I);
    const at::Tensor ws = at::empty({static_cast<int64_t>(need < 256 ? 256 : need)}, at::TensorOptions().dtype(at::kByte).device(x.device()));
    check(bm_dense_mlp_forward(x.data_ptr(), xd, wptr(wg), wptr(wu), wptr(wd), wptr(tg), T, H, I, ptr(residual), y.data_ptr(), xd, ws.data_ptr(),
                               ws.nbytes(), stream_of(x.device())));
    return THPVariable_Wrap(y);
  });
}

at::Tensor run_experts(HostLayer* L, const at::Tensor& hg, const at::Tensor& hu, const at::Tensor& tok, const at::Tensor& off,
                       const at::Tensor& rw, int64_t rank_out, int32_t path) {
  // h_up may have fewer rows than h_gate: only the rows that token_indices names are read
  for (const at::Tensor* h : {&hg, &hu})
    require(h->device() == L->device && h->scalar_type() == at::kHalf && h->is_contiguous() && h->dim() == 2 && h->size(1) == L->rank_in,
            "experts_forward: h_gate and h_up must be contiguous float16 [tokens, rank] of the layer's rank and device");
  require(rank_out == L->rank_out, "experts_forward: rank_out is not the layer's");
  require(tok.device() == L->device && tok.scalar_type() == at::kInt && tok.is_contiguous() && off.device() == L->device &&
              off.scalar_type() == at::kInt && off.is_contiguous() && off.numel() == L->experts + 1 && rw.device() == L->device &&
              rw.scalar_type() == at::kFloat && rw.is_contiguous() && rw.numel() >= tok.numel(),
          "experts_forward: routing must be contiguous on the layer's device: int32 token_indices, int32 expert_offsets [experts + 1], float32 weights");
  const c10::cuda::CUDAGuard guard(L->device);
  const int32_t T = static_cast<int32_t>(hg.size(0)), A = static_cast<int32_t>(tok.numel());
  const at::Tensor out = at::empty({T, rank_out}, hg.options().dtype(at::kFloat));
  const size_t need = bm_experts_workspace_bytes(L->handle, T, A, path);
  at::Tensor ws;
  if (need) ws = at::empty({static_cast<int64_t>(need)}, hg.options().dtype(at::kByte));
  check(bm_experts_forward(L->handle, wptr(hg), wptr(hu), static_cast<const int32_t*>(tok.data_ptr()), static_cast<const int32_t*>(off.data_ptr()),
                           static_cast<const float*>(rw.data_ptr()), T, A, static_cast<float*>(out.data_ptr()), path, ptr(ws), need,
                           stream_of(L->device)));
  return out;
}

// (layer, h_gate, h_up, token_indices, expert_offsets, route_weights, rank_out, path) -> rank_accum
PyObject* experts_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    need_args(n, 8);
    return THPVariable_Wrap(run_experts(layer_of(a[0]), tensor(a[1]), tensor(a[2]), tensor(a[3]), tensor(a[4]), tensor(a[5]), integer(a[6]),
                                        static_cast<int32_t>(integer(a[7]))));
  });
}

// ---- moe_packed_forward: layers already prepared for a set of weight lists
// A layer is found by the address and length of every payload tensor of the three lists, as the Python cache that owns
// it keys it; the entry holds the layer alive, so an address in it cannot have been given to another tensor.
struct OpEntry {
  std::vector<std::pair<const void*, int64_t>> payloads;
  int64_t rank_out, intermediate, h_rank;
  int device;
  PyObject* owner;
  PyObject* capsule;
};
std::vector<OpEntry> op_entries;

bool collect_payloads(PyObject* const* lists, std::vector<std::pair<const void*, int64_t>>* out, const OpEntry* expect) {
  size_t pos = 0;
  for (int m = 0; m < 3; ++m) {
    PyObject* seq = lists[6 * m];
    if (!PyTuple_Check(seq) && !PyList_Check(seq)) return false;
    PyObject** items = PySequence_Fast_ITEMS(seq);
    const Py_ssize_t len = PySequence_Fast_GET_SIZE(seq);
    for (Py_ssize_t i = 0; i < len; ++i, ++pos) {
      if (!THPVariable_Check(items[i])) return false;
      const at::Tensor& t = THPVariable_Unpack(items[i]);
      if (expect) {
        if (pos >= expect->payloads.size() || expect->payloads[pos].first != t.data_ptr() || expect->payloads[pos].second != t.numel()) return false;
      } else {
        out->emplace_back(t.data_ptr(), t.numel());
      }
    }
  }
  return !expect || pos == expect->payloads.size();
}

// (h_gate, h_up, token_indices, expert_offsets, route_weights, 18 lists, rank_out, intermediate, act_type, path) ->
// rank_accum, or None when an argument needs the full checks or the lists have not been met yet
PyObject* op_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need_args(n, 27);
    for (int i = 0; i < 5; ++i)
      if (!THPVariable_Check(a[i])) Py_RETURN_NONE;
    const at::Tensor &hg = tensor(a[0]), &hu = tensor(a[1]), &tok = tensor(a[2]), &off = tensor(a[3]), &rw = tensor(a[4]);
    auto ok = [&](const at::Tensor& t, at::ScalarType type, int dim) {
      return t.is_cuda() && t.scalar_type() == type && t.dim() == dim && t.is_contiguous();
    };
    if (!ok(hg, at::kHalf, 2) || !ok(hu, at::kHalf, 2) || !ok(tok, at::kInt, 1) || !ok(off, at::kInt, 1) || !ok(rw, at::kFloat, 1) ||
        hg.sizes() != hu.sizes() || tok.numel() != rw.numel() || tok.numel() == 0 || off.numel() < 2)
      Py_RETURN_NONE;
    for (int i = 5; i < 23; ++i)
      if ((!PyTuple_Check(a[i]) && !PyList_Check(a[i])) || PySequence_Fast_GET_SIZE(a[i]) != off.numel() - 1) Py_RETURN_NONE;
    const int64_t rank_out = integer(a[23]), inter = integer(a[24]);
    if (integer(a[25]) != 0) Py_RETURN_NONE;
    for (const OpEntry& e : op_entries) {
      if (e.rank_out != rank_out || e.intermediate != inter || e.h_rank != hg.size(1) || e.device != hg.device().index()) continue;
      auto* L = static_cast<HostLayer*>(PyCapsule_GetPointer(e.capsule, CAPSULE));
      if (!L || !L->handle || !collect_payloads(a + 5, nullptr, &e)) continue;
      return THPVariable_Wrap(run_experts(L, hg, hu, tok, off, rw, rank_out, static_cast<int32_t>(integer(a[26]))));
    }
    Py_RETURN_NONE;
  });
}
// (18 lists, rank_out, intermediate, h_rank, device index, owner, layer)
PyObject* op_register(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need_args(n, 24);
    OpEntry e{};
    if (!collect_payloads(a, &e.payloads, nullptr)) Py_RETURN_NONE;
    e.rank_out = integer(a[18]); e.intermediate = integer(a[19]); e.h_rank = integer(a[20]);
    e.device = static_cast<int>(integer(a[21]));
    e.owner = a[22]; e.capsule = a[23];
    Py_INCREF(e.owner);
    Py_INCREF(e.capsule);
    op_entries.push_back(std::move(e));
    Py_RETURN_NONE;
  });
}
PyObject* op_clear(PyObject*, PyObject*) {
  std::vector<OpEntry> gone;
  gone.swap(op_entries);
  for (OpEntry& e : gone) {
    Py_DECREF(e.owner);
    Py_DECREF(e.capsule);
  }
  Py_RETURN_NONE;
}

// ---- packing one matrix
at::Tensor ints(const std::vector<int32_t>& v, int64_t cols) {
  const int64_t n = static_cast<int64_t>(v.size());
  const at::Tensor t = cols ? at::empty({n / cols, cols}, at::kInt) : at::empty({n}, at::kInt);
  if (n) memcpy(t.data_ptr(), v.data(), v.size() * 4);
  return t;
}

// (rank_major fp32 [rank, dim] CUDA, s fp32 [rank] on the same device, [(bits, [(start, end), ...]), ...], to_host) ->
// (payload, rank_idx, tile_meta, slab_meta, scale, s, segments, original indices, original rank): payload, scale and s on the factor's device, or with
// to_host fetched in one copy into host tensors of their own
PyObject* pack_matrix(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need_args(n, 4);
    const at::Tensor w = tensor(a[0]), s = tensor(a[1]);
    const bool to_host = PyObject_IsTrue(a[3]) == 1;
    constexpr int SLAB = 64, TILE = 128, MICROS = 4;
    const int64_t dim = w.size(1), tiles = (dim + TILE - 1) / TILE;
    std::vector<int32_t> rows, slabs, slab_meta, tile_meta, segments;
    int64_t words = 0, scales = 0;
    PyObject* buckets = a[2];
    for (Py_ssize_t b = 0; b < PyList_Size(buckets); ++b) {
      PyObject* bucket = PyList_GetItem(buckets, b);
      const int32_t bits = static_cast<int32_t>(integer(PyTuple_GetItem(bucket, 0)));
      const int32_t wpr = bits == 16 ? 16 : bits, first = static_cast<int32_t>(rows.size());
      PyObject* ranges = PyTuple_GetItem(bucket, 1);
      for (Py_ssize_t i = 0; i < PyList_Size(ranges); ++i) {
        PyObject* r = PyList_GetItem(ranges, i);
        const int32_t e = static_cast<int32_t>(integer(PyTuple_GetItem(r, 1)));
        for (int32_t x = static_cast<int32_t>(integer(PyTuple_GetItem(r, 0))); x < e; ++x) rows.push_back(x);
      }
      const int32_t end = static_cast<int32_t>(rows.size());
      segments.insert(segments.end(), {bits, first, end});
      for (int32_t r0 = first; r0 < end; r0 += SLAB) {
        const int32_t k = std::min(SLAB, end - r0);
        slabs.insert(slabs.end(), {bits, k});
        slab_meta.insert(slab_meta.end(), {bits, k, r0, static_cast<int32_t>(tile_meta.size() / 3)});
        const int64_t wpt = static_cast<int64_t>(k) * MICROS * wpr;
        for (int64_t t = 0; t < tiles; ++t, words += wpt, scales += k)
          tile_meta.insert(tile_meta.end(), {static_cast<int32_t>(words), static_cast<int32_t>(scales),
                                             static_cast<int32_t>(std::min<int64_t>(TILE, dim - t * TILE))});
      }
    }
    const int64_t stored = static_cast<int64_t>(rows.size());
    const c10::cuda::CUDAGuard guard(w.device());
    const auto dev = at::TensorOptions().device(w.device());
    at::Tensor payload, scale, s_out, tables[6];
    auto make_tables = [&] {
      tables[0] = ints(rows, 0);
      tables[1] = ints(tile_meta, 3);
      tables[2] = ints(slab_meta, 4);
      tables[3] = ints(segments, 3);
      tables[4] = ints(rows, 0);      // the original indices: a tensor of their own
      tables[5] = at::empty({}, at::kInt);
      *static_cast<int32_t*>(tables[5].data_ptr()) = static_cast<int32_t>(w.size(0));
    };
    if (to_host) {
      // one device buffer and one pinned one: a single copy, then plain memory copies
      auto up = [](int64_t v) { return (v + 255) & ~static_cast<int64_t>(255); };
      const int64_t o_scale = up(words * 4), o_s = o_scale + up(scales * 2), total = o_s + stored * 2;
      at::Tensor h;
      cudaStream_t stream = nullptr;
      if (total > 0) {
        const at::Tensor d = at::empty({total}, dev.dtype(at::kByte));
        h = at::empty({total}, at::TensorOptions().dtype(at::kByte).pinned_memory(true));
        char* base = static_cast<char*>(d.data_ptr());
        check(bm_quantize_pack_matrix(static_cast<const float*>(w.data_ptr()), w.stride(0), static_cast<const float*>(s.data_ptr()),
                                      static_cast<int32_t>(dim), rows.data(), slabs.data(), static_cast<int32_t>(slabs.size() / 2),
                                      reinterpret_cast<uint32_t*>(base), reinterpret_cast<uint16_t*>(base + o_scale),
                                      reinterpret_cast<uint16_t*>(base + o_s), stream_of(w.device())));
        stream = c10::cuda::getCurrentCUDAStream(w.device().index()).stream();
        const cudaError_t e = cudaMemcpyAsync(h.data_ptr(), base, total, cudaMemcpyDeviceToHost, stream);
        if (e != cudaSuccess) fail(PyExc_RuntimeError, cudaGetErrorString(e));
      }
      // everything that does not need the device's answer is made while it works
      payload = at::empty({words}, at::kUInt32);
      scale = at::empty({scales}, at::kHalf);
      s_out = at::empty({stored}, at::kHalf);
      make_tables();
      if (total > 0) {
        cudaError_t done;
        Py_BEGIN_ALLOW_THREADS
        done = cudaStreamSynchronize(stream);
        Py_END_ALLOW_THREADS
        if (done != cudaSuccess) fail(PyExc_RuntimeError, cudaGetErrorString(done));
        const char* hb = static_cast<const char*>(h.data_ptr());
        memcpy(payload.data_ptr(), hb, words * 4);
        memcpy(scale.data_ptr(), hb + o_scale, scales * 2);
        memcpy(s_out.data_ptr(), hb + o_s, stored * 2);
      }
    } else {
      payload = at::empty({words}, dev.dtype(at::kUInt32));
      scale = at::empty({scales}, dev.dtype(at::kHalf));
      s_out = at::empty({stored}, dev.dtype(at::kHalf));
      check(bm_quantize_pack_matrix(static_cast<const float*>(w.data_ptr()), w.stride(0), static_cast<const float*>(s.data_ptr()),
                                    static_cast<int32_t>(dim), rows.data(), slabs.data(), static_cast<int32_t>(slabs.size() / 2),
                                    static_cast<uint32_t*>(payload.data_ptr()), static_cast<uint16_t*>(scale.data_ptr()),
                                    static_cast<uint16_t*>(s_out.data_ptr()), stream_of(w.device())));
      make_tables();
    }
    const at::Tensor out[9] = {payload, tables[0], tables[1], tables[2], scale, s_out, tables[3], tables[4], tables[5]};
    PyObject* r = PyTuple_New(9);
    for (int i = 0; i < 9; ++i) PyTuple_SET_ITEM(r, i, THPVariable_Wrap(out[i]));
    return r;
  });
}

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FAST(layer_new), FAST(layer_close), FAST(layer_drop_workspaces), FAST(layer_workspace), FAST(layer_forward),
                         FAST(block_forward), FAST(dense_mlp), FAST(experts_forward), FAST(op_forward), FAST(op_register), FAST(pack_matrix),
                         {"op_clear", op_clear, METH_NOARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_bm_host", "Native host path of bitsmoe_b200.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__bm_host(void) { return PyModule_Create(&module); }
