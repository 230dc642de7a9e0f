// Native host path between torch and the C ABI: argument checks, allocation of the outputs, the autograd nodes and the
// launches, behind two Python-callable functions. A call spends its host time here instead of in Python: through
// ctypes, Python autograd functions and functorch's wrapping of them a small dual forward took 136 us and a training
// step 450 us (1100 us under torch.func.jvp), all of it host time beside 9 to 50 us of kernels.
//
// Operators of the library `jvpfa` (all of them reach the kernels through function pointers that Python hands over,
// see `bind`; nothing here links against the CUDA library):
//   attention       (q, k, v) -> o; a dual o when an input carries a forward-mode tangent
//   attention_dual  (q, k, v, tq, tk, tv) -> [o, to]
//   fwd, bwd        the kernels with autograd: `fwd` records a node whose backward calls `bwd`
// They are dispatcher operators, so torch.func transforms peel their levels off the arguments before the kernels see
// them, as they do for torch's own operators.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/utils/pybind.h>
#include <torch/library.h>
#include <torch/torch.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAStream.h>
#include <cmath>
#include <mutex>
#include <vector>
#include "../../include/jvpfa.h"

namespace {

using at::Tensor;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

// ------------------------------------------------------------------------------------------------ the C ABI
struct Api {
  size_t (*fwd_workspace_bytes)(const jvpfa_fwd_args*) = nullptr;
  size_t (*bwd_workspace_bytes)(const jvpfa_bwd_args*) = nullptr;
  size_t (*mask_summary_bytes)(int32_t, int32_t, int32_t) = nullptr;
  int (*mask_summary)(const jvpfa_mask*, int32_t, int32_t, int32_t, uint8_t*, void*) = nullptr;
  int (*mask_check_begin)(const jvpfa_mask*, int32_t, int32_t, int32_t, const uint8_t*, void*, void**) = nullptr;
  int (*mask_check_end)(void*, int32_t*) = nullptr;
  int (*fwd_status)(const jvpfa_fwd_args*, int32_t*, void*) = nullptr;
  int (*bwd_status)(const jvpfa_bwd_args*, int32_t*, void*) = nullptr;
  PyObject* get_workspace = nullptr;   // (device index, stream, bytes) -> (pointer, bytes, status pointer); raises on a timeout
  PyObject* raise_status = nullptr;    // (status) -> raises
  PyObject* raise_mask = nullptr;      // (verdict) -> raises
};
Api g_api;

// Calls a Python function that raises and carries its exception over to the caller (from any thread).
[[noreturn]] void raise_through(PyObject* fn, long value) {
  pybind11::gil_scoped_acquire gil;
  PyObject* r = PyObject_CallFunction(fn, "l", value);
  Py_XDECREF(r);
  if (r != nullptr) TORCH_CHECK(false, "jvpfa: unexpected status ", value);
  python_error e;
  e.persist();
  throw e;
}
void check_status(int rc) {
  if (rc != JVPFA_OK) raise_through(g_api.raise_status, rc);
}

// ------------------------------------------------------------------------------------------------ workspaces
// The workspaces belong to Python (one per device and stream, grown on demand, status word in pinned host memory); this
// is a look-aside list of their addresses, so that an ordinary call does not enter Python.
struct Workspace {
  int device;
  void* stream;
  void* ptr;
  size_t bytes;
  volatile int32_t* status;   // pinned host memory the kernels write to when a wait gives up
};
std::mutex g_ws_mutex;
std::vector<Workspace> g_ws;

Workspace workspace_for(int device, void* stream, size_t bytes) {
  {
    std::lock_guard<std::mutex> lock(g_ws_mutex);
    for (const Workspace& w : g_ws)
      if (w.device == device && w.stream == stream) {
        if (w.bytes >= bytes && *w.status == 0) return w;
        break;
      }
  }
  pybind11::gil_scoped_acquire gil;
  PyObject* r = PyObject_CallFunction(g_api.get_workspace, "iKK", device, reinterpret_cast<unsigned long long>(stream),
                                      static_cast<unsigned long long>(bytes));
  unsigned long long ptr = 0, size = 0, status = 0;
  const bool ok = r != nullptr && PyArg_ParseTuple(r, "KKK", &ptr, &size, &status);
  Py_XDECREF(r);
  if (!ok) {
    python_error e;
    e.persist();
    throw e;
  }
  Workspace w{device, stream, reinterpret_cast<void*>(ptr), static_cast<size_t>(size), reinterpret_cast<volatile int32_t*>(status)};
  std::lock_guard<std::mutex> lock(g_ws_mutex);
  for (Workspace& x : g_ws)
    if (x.device == device && x.stream == stream) {
      x = w;
      return w;
    }
  g_ws.push_back(w);
  return w;
}

// ------------------------------------------------------------------------------------------------ tensors -> C structs
int dtype_code(at::ScalarType t) {
  return t == at::kHalf ? JVPFA_F16 : t == at::kBFloat16 ? JVPFA_BF16 : t == at::kFloat ? JVPFA_F32 : -1;
}

// (dtype, head dimension) that the tensor-core kernels take; they read strided inputs in place
bool tensor_core_path(at::ScalarType t, int64_t D) {
  if (D < 8 || D % 8 != 0) return false;
  return t == at::kFloat ? D <= 64 : D <= 256;
}

// Readable in place: last axis contiguous, every other stride (of an axis longer than 1) positive and a multiple of 16 bytes,
// 16-byte aligned storage (a functorch wrapper has none: the plain tensor inside is looked at again below it).
bool readable_in_place(const Tensor& t) {
  if (t.stride(3) != 1 || !tensor_core_path(t.scalar_type(), t.size(3))) return false;
  if (t.has_storage() && (reinterpret_cast<uintptr_t>(t.const_data_ptr()) & 15) != 0) return false;
  const int64_t es = static_cast<int64_t>(t.element_size());
  for (int d = 0; d < 3; ++d) {
    const int64_t s = t.stride(d);
    if ((d == 2 || t.size(d) > 1) && (s <= 0 || (s * es) % 16 != 0)) return false;
  }
  return true;
}
Tensor as_input(const Tensor& t) { return (t.is_contiguous() || readable_in_place(t)) ? t : t.contiguous(); }

jvpfa_strides strides_of(const Tensor& t) {
  if (t.is_contiguous()) return jvpfa_strides{0, 0, 0};
  const int64_t B = t.size(0), H = t.size(1), N = t.size(2), D = t.size(3);
  // an axis of length 1 may carry any stride: give it the contiguous one
  return jvpfa_strides{B > 1 ? t.stride(0) : H * N * D, H > 1 ? t.stride(1) : N * D, N > 1 ? t.stride(2) : D};
}

jvpfa_mask mask_of(const OptTensor& mask, int64_t B, int64_t H, int64_t N) {
  jvpfa_mask m{};
  if (!mask.has_value() || !mask->defined()) return m;
  const Tensor view = mask->expand({B, H, N, N});
  m.ptr = view.const_data_ptr();
  m.kind = mask->scalar_type() == at::kBool ? JVPFA_MASK_BOOL : JVPFA_MASK_ADDITIVE;
  m.dtype = m.kind == JVPFA_MASK_BOOL ? 0 : dtype_code(mask->scalar_type());
  for (int i = 0; i < 4; ++i) m.stride[i] = view.stride(i);
  return m;
}

bool has(const OptTensor& t) { return t.has_value() && t->defined(); }
bool has_fw_grad(const Tensor& t) { return t.defined() && t._fw_grad(/*level=*/0).defined(); }
bool has_fw_grad(const OptTensor& t) { return has(t) && has_fw_grad(*t); }

// ------------------------------------------------------------------------------------------------ the kernels (CUDA)
// [o, to (dual), stats (lse2 and mu as one (2,B,H,N) tensor), mask summary (masked)]
std::vector<Tensor> fwd_cuda(const Tensor& q_, const Tensor& k_, const Tensor& v_, const OptTensor& tq_, const OptTensor& tk_,
                             const OptTensor& tv_, const OptTensor& mask, bool causal, double scale, double dropout_p,
                             int64_t dropout_seed, bool verify, bool /*tangents_taken*/) {
  const c10::DeviceGuard device_guard(q_.device());
  const bool dual = has(tq_);
  const Tensor q = as_input(q_), k = as_input(k_), v = as_input(v_);
  const Tensor tq = dual ? as_input(*tq_) : Tensor(), tk = dual ? as_input(*tk_) : Tensor(), tv = dual ? as_input(*tv_) : Tensor();
  const int64_t B = q.size(0), H = q.size(1), N = q.size(2), D = q.size(3);
  void* stream = c10::cuda::getCurrentCUDAStream(q.device().index()).stream();
  std::vector<Tensor> out;
  out.reserve(4);
  out.push_back(at::empty({B, H, N, D}, q.options()));
  if (dual) out.push_back(at::empty({B, H, N, D}, q.options()));
  const Tensor stats = at::empty({2, B, H, N}, q.options().dtype(at::kFloat));
  out.push_back(stats);
  jvpfa_fwd_args a{};
  a.B = static_cast<int32_t>(B); a.H = static_cast<int32_t>(H); a.N = static_cast<int32_t>(N); a.D = static_cast<int32_t>(D);
  a.dtype = dtype_code(q.scalar_type());
  a.causal = causal;
  a.sm_scale = static_cast<float>(scale);
  a.mask = mask_of(mask, B, H, N);
  a.q = q.const_data_ptr(); a.k = k.const_data_ptr(); a.v = v.const_data_ptr();
  a.q_strides = strides_of(q); a.k_strides = strides_of(k); a.v_strides = strides_of(v);
  a.o = out[0].data_ptr();
  if (dual) {
    a.tq = tq.const_data_ptr(); a.tk = tk.const_data_ptr(); a.tv = tv.const_data_ptr();
    a.tq_strides = strides_of(tq); a.tk_strides = strides_of(tk); a.tv_strides = strides_of(tv);
    a.to = out[1].data_ptr();
  }
  a.lse2 = static_cast<float*>(stats.data_ptr());
  a.mu = a.lse2 + B * H * N;
  a.dropout_p = static_cast<float>(dropout_p);
  a.dropout_seed = static_cast<uint64_t>(dropout_seed);
  const Workspace ws = workspace_for(q.device().index(), stream, g_api.fwd_workspace_bytes(&a));
  a.workspace = ws.ptr;
  a.workspace_bytes = ws.bytes;
  void* check = nullptr;
  if (a.mask.kind != JVPFA_MASK_NONE) {
    const int32_t Bm = a.mask.stride[0] == 0 ? 1 : a.B, Hm = a.mask.stride[1] == 0 ? 1 : a.H;
    Tensor summary = at::empty({static_cast<int64_t>(g_api.mask_summary_bytes(Bm, Hm, a.N))}, q.options().dtype(at::kByte));
    uint8_t* sp = static_cast<uint8_t*>(summary.data_ptr());
    check_status(g_api.mask_summary(&a.mask, a.B, a.H, a.N, sp, stream));
    // the verdict on the mask comes from the summary; it is read after the attention kernel has been launched, so that
    // the host's wait for it runs beside that kernel
    if (verify) check_status(g_api.mask_check_begin(&a.mask, a.B, a.H, a.N, sp, stream, &check));
    a.mask_summary = sp;
    out.push_back(std::move(summary));
  }
  const int rc = g_api.fwd_status(&a, const_cast<int32_t*>(ws.status), stream);
  if (check != nullptr) {
    int32_t verdict = 0;
    const int rc_check = g_api.mask_check_end(check, &verdict);
    check_status(rc_check);
    if (verdict != 0) raise_through(g_api.raise_mask, verdict);
  }
  check_status(rc);
  return out;
}

// [dq, dk, dv] (no gradient through a tangent output: gto undefined) or [dq, dk, dv, dtq, dtk, dtv]
std::vector<Tensor> bwd_cuda(const OptTensor& go_, const OptTensor& gto_, const Tensor& q_, const Tensor& k_, const Tensor& v_,
                             const OptTensor& tq_, const OptTensor& tk_, const OptTensor& tv_, const Tensor& o, const OptTensor& to,
                             const Tensor& stats, const OptTensor& mask, const OptTensor& summary, bool causal, double scale,
                             double dropout_p, int64_t dropout_seed) {
  const c10::DeviceGuard device_guard(q_.device());
  const bool dual = has(gto_);
  const Tensor q = as_input(q_), k = as_input(k_), v = as_input(v_);
  const int64_t B = q.size(0), H = q.size(1), N = q.size(2), D = q.size(3);
  const Tensor go = has(go_) ? as_input(*go_) : at::zeros({B, H, N, D}, q.options());
  Tensor tq, tk, tv, gto;
  if (dual) {
    tq = as_input(*tq_); tk = as_input(*tk_); tv = as_input(*tv_);
    gto = as_input(*gto_);
  }
  void* stream = c10::cuda::getCurrentCUDAStream(q.device().index()).stream();
  std::vector<Tensor> out;
  out.reserve(6);
  for (int i = 0; i < (dual ? 6 : 3); ++i) out.push_back(at::empty({B, H, N, D}, q.options()));
  jvpfa_bwd_args a{};
  a.B = static_cast<int32_t>(B); a.H = static_cast<int32_t>(H); a.N = static_cast<int32_t>(N); a.D = static_cast<int32_t>(D);
  a.dtype = dtype_code(q.scalar_type());
  a.causal = causal;
  a.sm_scale = static_cast<float>(scale);
  a.mask = mask_of(mask, B, H, N);
  a.mask_summary = has(summary) ? static_cast<const uint8_t*>(summary->const_data_ptr()) : nullptr;
  a.q = q.const_data_ptr(); a.k = k.const_data_ptr(); a.v = v.const_data_ptr();
  a.q_strides = strides_of(q); a.k_strides = strides_of(k); a.v_strides = strides_of(v);
  a.o = o.const_data_ptr();
  a.lse2 = static_cast<const float*>(stats.const_data_ptr());
  a.mu = a.lse2 + B * H * N;
  a.go = go.const_data_ptr();
  a.go_strides = strides_of(go);
  a.dq = out[0].data_ptr(); a.dk = out[1].data_ptr(); a.dv = out[2].data_ptr();
  if (dual) {
    a.tq = tq.const_data_ptr(); a.tk = tk.const_data_ptr(); a.tv = tv.const_data_ptr();
    a.tq_strides = strides_of(tq); a.tk_strides = strides_of(tk); a.tv_strides = strides_of(tv);
    a.to = to->const_data_ptr();
    a.gto = gto.const_data_ptr();
    a.gto_strides = strides_of(gto);
    a.dtq = out[3].data_ptr(); a.dtk = out[4].data_ptr(); a.dtv = out[5].data_ptr();
  }
  a.dropout_p = static_cast<float>(dropout_p);
  a.dropout_seed = static_cast<uint64_t>(dropout_seed);
  const Workspace ws = workspace_for(q.device().index(), stream, g_api.bwd_workspace_bytes(&a));
  a.workspace = ws.ptr;
  a.workspace_bytes = ws.bytes;
  check_status(g_api.bwd_status(&a, const_cast<int32_t*>(ws.status), stream));
  return out;
}

// ------------------------------------------------------------------------------------------------ calls through the dispatcher
using FwdFn = std::vector<Tensor>(const Tensor&, const Tensor&, const Tensor&, const OptTensor&, const OptTensor&, const OptTensor&,
                                  const OptTensor&, bool, double, double, int64_t, bool, bool);
using BwdFn = std::vector<Tensor>(const OptTensor&, const OptTensor&, const Tensor&, const Tensor&, const Tensor&, const OptTensor&,
                                  const OptTensor&, const OptTensor&, const Tensor&, const OptTensor&, const Tensor&, const OptTensor&,
                                  const OptTensor&, bool, double, double, int64_t);
using AttnFn = Tensor(const Tensor&, const Tensor&, const Tensor&, const OptTensor&, bool, double, double, int64_t, bool, bool);
using DualFn = std::vector<Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&,
                                   const OptTensor&, bool, double, double, int64_t, bool);

template <typename F>
const c10::TypedOperatorHandle<F>& op(const char* name) {
  static const c10::TypedOperatorHandle<F> h = c10::Dispatcher::singleton().findSchemaOrThrow(name, "").template typed<F>();
  return h;
}

// ------------------------------------------------------------------------------------------------ autograd
struct AttentionBackward : public torch::autograd::Node {
  SavedVariable q, k, v, tq, tk, tv, o, to, stats, summary;
  Tensor mask;   // the caller's, never differentiated: kept as it is
  bool dual = false, causal = false;
  double scale = 1.0, dropout_p = 0.0;
  int64_t dropout_seed = 0;

  std::string name() const override { return "JVPAttentionBackward"; }
  void release_variables() override {
    const std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable* s : {&q, &k, &v, &tq, &tk, &tv, &o, &to, &stats, &summary}) s->reset_data();
    mask.reset();
  }
  // An output that the loss does not use arrives as an undefined gradient. Without one for the tangent output the
  // primal-only kernels run and the tangent inputs get no gradient.
  variable_list apply(variable_list&& grads) override {
    const std::lock_guard<std::mutex> lock(mutex_);
    variable_list res(dual ? 6 : 3);
    const Tensor go = grads[0], gto = dual ? grads[1] : Tensor();
    bool wanted = false;
    for (size_t i = 0; i < res.size(); ++i) wanted |= task_should_compute_output(i);
    if (!wanted || (!go.defined() && !gto.defined())) return res;
    auto self = getptr();
    const bool both = gto.defined();
    const auto opt = [](const Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); };
    const std::vector<Tensor> g = op<BwdFn>("jvpfa::bwd").call(
        opt(go), opt(gto), q.unpack(), k.unpack(), v.unpack(), both ? opt(tq.unpack()) : OptTensor(),
        both ? opt(tk.unpack()) : OptTensor(), both ? opt(tv.unpack()) : OptTensor(), o.unpack(self),
        both ? opt(to.unpack(self)) : OptTensor(), stats.unpack(), opt(mask), opt(summary.unpack()), causal, scale, dropout_p, dropout_seed);
    for (size_t i = 0; i < g.size(); ++i)
      if (task_should_compute_output(i)) res[i] = g[i];
    return res;
  }
};

constexpr const char* kNoNesting =
    "JVP attention: forward-mode tangents of these inputs are not supported here (fwd_dual takes one level of tangents)";

std::vector<Tensor> fwd_autograd(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& tq, const OptTensor& tk,
                                 const OptTensor& tv, const OptTensor& mask, bool causal, double scale, double dropout_p,
                                 int64_t dropout_seed, bool verify, bool tangents_taken) {
  const bool dual = has(tq);
  // tangents_taken: the caller has read the tangents of q, k, v at this level and passes them as tq, tk, tv
  if ((!tangents_taken && (has_fw_grad(q) || has_fw_grad(k) || has_fw_grad(v))) || has_fw_grad(tq) || has_fw_grad(tk) || has_fw_grad(tv))
    TORCH_CHECK_NOT_IMPLEMENTED(false, kNoNesting);
  if (has_fw_grad(mask)) TORCH_CHECK_NOT_IMPLEMENTED(false, "JVP attention: a forward-mode tangent of the attention mask is not supported");
  const Tensor none;
  // (a mask that requires a gradient gets none, but the outputs can be differentiated)
  const bool record = torch::autograd::compute_requires_grad(q, k, v, dual ? *tq : none, dual ? *tk : none, dual ? *tv : none,
                                                             has(mask) ? *mask : none);
  std::vector<Tensor> out;
  {
    at::AutoDispatchBelowADInplaceOrView guard;
    out = op<FwdFn>("jvpfa::fwd").call(q, k, v, tq, tk, tv, mask, causal, scale, dropout_p, dropout_seed, verify, false);
  }
  if (!record) return out;
  std::shared_ptr<AttentionBackward> node(new AttentionBackward(), torch::autograd::deleteNode);
  if (dual) node->set_next_edges(torch::autograd::collect_next_edges(q, k, v, *tq, *tk, *tv));
  else node->set_next_edges(torch::autograd::collect_next_edges(q, k, v));
  const auto plain = [&](const Tensor& t) { return SavedVariable(tangents_taken && has_fw_grad(t) ? t.detach() : t, false); };
  node->q = plain(q); node->k = plain(k); node->v = plain(v);
  const size_t n_out = dual ? 2 : 1;
  if (dual) {
    node->tq = SavedVariable(*tq, false); node->tk = SavedVariable(*tk, false); node->tv = SavedVariable(*tv, false);
  }
  node->stats = SavedVariable(out[n_out], false);
  if (mask.has_value() && mask->defined()) {
    node->mask = *mask;
    node->summary = SavedVariable(out[n_out + 1], false);
  }
  node->dual = dual; node->causal = causal; node->scale = scale;
  node->dropout_p = dropout_p; node->dropout_seed = dropout_seed;
  for (size_t i = 0; i < n_out; ++i) torch::autograd::set_history(out[i], node);
  node->o = SavedVariable(out[0], true);
  if (dual) node->to = SavedVariable(out[1], true);
  return out;
}

std::vector<Tensor> bwd_autograd(const OptTensor& go_, const OptTensor& gto_, const Tensor& q, const Tensor& k, const Tensor& v,
                                 const OptTensor& tq, const OptTensor& tk, const OptTensor& tv, const Tensor& o, const OptTensor& to,
                                 const Tensor& stats, const OptTensor& mask, const OptTensor& summary, bool causal, double scale,
                                 double dropout_p, int64_t dropout_seed) {
  if (has_fw_grad(q) || has_fw_grad(k) || has_fw_grad(v) || has_fw_grad(tq) || has_fw_grad(tk) || has_fw_grad(tv))
    TORCH_CHECK_NOT_IMPLEMENTED(false, kNoNesting);
  // A backward inside fwAD.dual_level(): whatever nonlinear follows the attention gives upstream gradients that carry a tangent,
  // from the activations it saved. The gradients are those of the upstream gradients without it. Under torch.func.jvp the
  // tangent is what the caller asks for: refused (a functorch level is being worked on).
  const auto without_tangent = [](const OptTensor& t) -> OptTensor {
    if (!has_fw_grad(t)) return t;
    if (c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerBackMode))
      TORCH_CHECK_NOT_IMPLEMENTED(false, kNoNesting);
    return t->_fw_primal(/*level=*/0);
  };
  const OptTensor go = without_tangent(go_), gto = without_tangent(gto_);
  std::vector<Tensor> out;
  {
    at::AutoDispatchBelowADInplaceOrView guard;
    out = op<BwdFn>("jvpfa::bwd").call(go, gto, q, k, v, tq, tk, tv, o, to, stats, mask, summary, causal, scale, dropout_p, dropout_seed);
  }
  const Tensor none;
  const auto t = [&](const OptTensor& x) { return has(x) ? *x : none; };
  // (o: recorded whenever the gradients are of a recorded call; q, k, v of a call on dual tensors are saved without their graph)
  if (torch::autograd::compute_requires_grad(t(go), t(gto), q, k, v, t(tq), t(tk), t(tv), o)) {
    // the gradients come from kernels: differentiating them again raises instead of returning zeros
    std::shared_ptr<torch::autograd::Node> err(
        new torch::autograd::Error("trying to differentiate twice: the gradients of JVP attention are computed by kernels",
                                   torch::autograd::collect_next_edges(t(go), t(gto), q, k, v, t(tq), t(tk), t(tv), o)),
        torch::autograd::deleteNode);
    for (Tensor& g : out) torch::autograd::set_history(g, err);
  }
  return out;
}

// ------------------------------------------------------------------------------------------------ the public operators
Tensor attention(const Tensor& q_, const Tensor& k_, const Tensor& v_, const OptTensor& mask, bool causal, double scale,
                 double dropout_p, int64_t dropout_seed, bool verify, bool allow_dual) {
  const bool any = has_fw_grad(q_) || has_fw_grad(k_) || has_fw_grad(v_);
  if (any && !allow_dual) TORCH_CHECK_NOT_IMPLEMENTED(false, "JVP attention: fwd takes no forward-mode tangents, use fwd_dual");
  const Tensor q = as_input(q_), k = as_input(k_), v = as_input(v_);
  if (!any)
    return op<FwdFn>("jvpfa::fwd").call(q, k, v, OptTensor(), OptTensor(), OptTensor(), mask, causal, scale, dropout_p, dropout_seed, verify, false)[0];
  // an input without a tangent contributes a zero tangent
  const auto tangent = [](const Tensor& t) {
    return has_fw_grad(t) ? as_input(t._fw_grad(/*level=*/0)) : at::zeros(t.sizes(), t.options());
  };
  const std::vector<Tensor> out =
      op<FwdFn>("jvpfa::fwd").call(q, k, v, tangent(q), tangent(k), tangent(v), mask, causal, scale, dropout_p, dropout_seed, verify, true);
  out[0]._set_fw_grad(out[1], /*level=*/0, /*is_inplace_op=*/false);
  return out[0];
}

std::vector<Tensor> attention_dual(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& tq, const Tensor& tk,
                                   const Tensor& tv, const OptTensor& mask, bool causal, double scale, double dropout_p,
                                   int64_t dropout_seed, bool verify) {
  std::vector<Tensor> out = op<FwdFn>("jvpfa::fwd").call(as_input(q), as_input(k), as_input(v), as_input(tq),
                                                         as_input(tk), as_input(tv), mask, causal, scale, dropout_p,
                                                         dropout_seed, verify, false);
  out.resize(2);
  return out;
}

TORCH_LIBRARY(jvpfa, m) {
  m.def("fwd(Tensor q, Tensor k, Tensor v, Tensor? tq, Tensor? tk, Tensor? tv, Tensor? mask, bool causal, float scale, "
        "float dropout_p, int dropout_seed, bool verify, bool tangents_taken) -> Tensor[]");
  m.def("bwd(Tensor? go, Tensor? gto, Tensor q, Tensor k, Tensor v, Tensor? tq, Tensor? tk, Tensor? tv, Tensor o, Tensor? to, "
        "Tensor stats, Tensor? mask, Tensor? summary, bool causal, float scale, float dropout_p, int dropout_seed) -> Tensor[]");
  m.def("attention(Tensor q, Tensor k, Tensor v, Tensor? mask, bool causal, float scale, float dropout_p, int dropout_seed, "
        "bool verify, bool allow_dual) -> Tensor");
  m.def("attention_dual(Tensor q, Tensor k, Tensor v, Tensor tq, Tensor tk, Tensor tv, Tensor? mask, bool causal, float scale, "
        "float dropout_p, int dropout_seed, bool verify) -> Tensor[]");
}
TORCH_LIBRARY_IMPL(jvpfa, CUDA, m) {
  m.impl("fwd", fwd_cuda);
  m.impl("bwd", bwd_cuda);
}
TORCH_LIBRARY_IMPL(jvpfa, Autograd, m) {
  m.impl("fwd", fwd_autograd);
  m.impl("bwd", bwd_autograd);
}
TORCH_LIBRARY_IMPL(jvpfa, CompositeImplicitAutograd, m) {
  m.impl("attention", attention);
  m.impl("attention_dual", attention_dual);
}

// ------------------------------------------------------------------------------------------------ Python entry points
// The checks an ordinary call passes. False sends the call back to Python, whose checks raise the exception that belongs to
// the mistake (or convert a mask of an unusual type).
bool checks_pass(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& mask, bool causal) {
  if (q.dim() != 4 || !q.is_cuda() || dtype_code(q.scalar_type()) < 0) return false;
  for (const Tensor* t : {&k, &v})
    if (t->scalar_type() != q.scalar_type() || t->device() != q.device() || t->sizes() != q.sizes()) return false;
  if (mask.has_value()) {
    if (causal || mask->dim() != 4 || mask->device() != q.device()) return false;
    const int64_t full[4] = {q.size(0), q.size(1), q.size(2), q.size(2)};
    for (int i = 0; i < 4; ++i)
      if (mask->size(i) != 1 && mask->size(i) != full[i]) return false;
    const auto mt = mask->scalar_type();
    if (mt != at::kBool && dtype_code(mt) < 0) return false;
  }
  return true;
}

struct CallArgs {
  OptTensor mask;
  bool causal, verify;
  double scale, dropout_p;
  int64_t seed;
};
bool tensors_of(PyObject* const* args, int n, Tensor* out) {
  for (int i = 0; i < n; ++i) {
    if (!THPVariable_Check(args[i])) return false;
    out[i] = THPVariable_Unpack(args[i]);
  }
  return true;
}
// (mask or None, causal, scale or None, dropout_p, seed, verify)
bool parse_common(PyObject* const* args, int64_t head_dim, CallArgs* c) {
  if (args[0] != Py_None) {
    if (!THPVariable_Check(args[0])) return false;
    c->mask = THPVariable_Unpack(args[0]);
  }
  c->causal = PyObject_IsTrue(args[1]) == 1;
  c->scale = args[2] == Py_None ? std::pow(static_cast<double>(head_dim), -0.5) : PyFloat_AsDouble(args[2]);
  c->dropout_p = PyFloat_AsDouble(args[3]);
  c->seed = static_cast<int64_t>(PyLong_AsUnsignedLongLongMask(args[4]));
  c->verify = PyObject_IsTrue(args[5]) == 1;
  return !PyErr_Occurred();
}

// call(q, k, v, mask, causal, scale, dropout_p, seed, verify, allow_dual) -> o, or None if a check failed
PyObject* py_call(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Tensor t[3];
  CallArgs c;
  if (n != 10 || !tensors_of(args, 3, t)) Py_RETURN_NONE;
  if (t[0].dim() != 4 || !parse_common(args + 3, t[0].size(3), &c)) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
  }
  if (!checks_pass(t[0], t[1], t[2], c.mask, c.causal)) Py_RETURN_NONE;
  const bool allow_dual = PyObject_IsTrue(args[9]) == 1;
  Tensor o;
  {
    pybind11::gil_scoped_release no_gil;
    o = op<AttnFn>("jvpfa::attention").call(t[0], t[1], t[2], c.mask, c.causal, c.scale, c.dropout_p, c.seed, c.verify, allow_dual);
  }
  return THPVariable_Wrap(std::move(o));
  END_HANDLE_TH_ERRORS
}

// dual(q, k, v, tq, tk, tv, mask, causal, scale, dropout_p, seed, verify) -> (o, to), or None if a check failed
PyObject* py_dual(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Tensor t[6];
  CallArgs c;
  if (n != 12 || !tensors_of(args, 6, t)) Py_RETURN_NONE;
  if (t[0].dim() != 4 || !parse_common(args + 6, t[0].size(3), &c)) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
  }
  if (!checks_pass(t[0], t[1], t[2], c.mask, c.causal) || !checks_pass(t[3], t[4], t[5], OptTensor(), false) ||
      t[3].sizes() != t[0].sizes() || t[3].scalar_type() != t[0].scalar_type() || t[3].device() != t[0].device())
    Py_RETURN_NONE;
  std::vector<Tensor> o;
  {
    pybind11::gil_scoped_release no_gil;
    o = op<DualFn>("jvpfa::attention_dual").call(t[0], t[1], t[2], t[3], t[4], t[5], c.mask, c.causal, c.scale, c.dropout_p, c.seed, c.verify);
  }
  PyObject* a = THPVariable_Wrap(std::move(o[0]));
  PyObject* b = THPVariable_Wrap(std::move(o[1]));
  PyObject* r = (a != nullptr && b != nullptr) ? PyTuple_Pack(2, a, b) : nullptr;
  Py_XDECREF(a);
  Py_XDECREF(b);
  return r;
  END_HANDLE_TH_ERRORS
}

// bind(eight function addresses, get_workspace, raise_status, raise_mask)
PyObject* py_bind(PyObject*, PyObject* args) {
  unsigned long long f[8];
  PyObject *ws, *st, *mk;
  if (!PyArg_ParseTuple(args, "KKKKKKKKOOO", &f[0], &f[1], &f[2], &f[3], &f[4], &f[5], &f[6], &f[7], &ws, &st, &mk)) return nullptr;
  const auto set = [](auto& fn, unsigned long long address) { fn = reinterpret_cast<std::decay_t<decltype(fn)>>(address); };
  set(g_api.fwd_workspace_bytes, f[0]);
  set(g_api.bwd_workspace_bytes, f[1]);
  set(g_api.mask_summary_bytes, f[2]);
  set(g_api.mask_summary, f[3]);
  set(g_api.mask_check_begin, f[4]);
  set(g_api.mask_check_end, f[5]);
  set(g_api.fwd_status, f[6]);
  set(g_api.bwd_status, f[7]);
  Py_INCREF(ws); Py_INCREF(st); Py_INCREF(mk);
  g_api.get_workspace = ws;
  g_api.raise_status = st;
  g_api.raise_mask = mk;
  Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"call", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_call)), METH_FASTCALL, nullptr},
    {"dual", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_dual)), METH_FASTCALL, nullptr},
    {"bind", py_bind, METH_VARARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&kModule); }
