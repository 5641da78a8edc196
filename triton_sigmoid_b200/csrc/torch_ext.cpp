// Eager host path between torch tensors and the C ABI of include/sigattn_b200.h: argument checks, output and
// workspace allocation, parameter filling and the autograd node, all native.
//
// A call on short sequences is bound by the host, not by the kernels.  Measured on a B200 host with the same work in
// Python (ctypes, torch.autograd.Function): 20 us per forward call and 155 us per forward + backward pair, against
// kernels of about 10 and 35 us; the backward alone had to take the GIL on the autograd thread and fill a ctypes
// structure field by field.
//
// Python keeps the argument validation with its error texts, the unusual inputs (other index types, head dimensions
// that need padding) and the registered ops used under torch.compile: the entry points below return None whenever
// something is not plain, and the caller then takes the Python path, which ends in attention() here once the inputs
// are normalised.
#include <Python.h>

#include <ATen/TracerMode.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/grad_mode.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/Exceptions.h>

#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>

#include "../../include/sigattn_b200.h"

namespace {

using at::Tensor;

// The C ABI, bound once from the library that the ctypes binding has loaded (one instance per process).
struct Abi {
  int (*fwd)(const SigAttnParams*) = nullptr;
  int (*bwd)(const SigAttnParams*) = nullptr;
  const char* (*last_error)() = nullptr;
  int (*device_status)(int) = nullptr;
} g_abi;

// accurate_sigmoid(): -1 = follow the environment, 0 / 1 = forced.
std::atomic<int> g_accurate_override{-1};

bool env_true(const char* name) {
  const char* v = std::getenv(name);
  if (!v || !*v) return false;
  std::string s(v);
  for (char& c : s) c = (char)std::tolower((unsigned char)c);
  return s == "1" || s == "true" || s == "yes" || s == "on";
}
// The run-time switches, read when an op runs.  Only with the GIL: an assignment to os.environ in another Python thread,
// which holds it too, rewrites the array that getenv() searches.
struct Switches {
  bool accurate, split_backward, debug;
};
Switches read_switches() {
  const int o = g_accurate_override.load(std::memory_order_relaxed);
  return {o >= 0 ? o != 0 : env_true("TRITON_SIGMOID_ACCURATE"), env_true("SIGATTN_B200_BWD_SPLIT"), env_true("SIGATTN_B200_DEBUG")};
}
// On a thread that does not hold it (autograd's).
Switches read_switches_locked() {
  const PyGILState_STATE state = PyGILState_Ensure();
  const Switches s = read_switches();
  PyGILState_Release(state);
  return s;
}

bool dtype_code(at::ScalarType t, int* code) {
  switch (t) {
    case at::kHalf: *code = SIGATTN_FP16; return true;
    case at::kBFloat16: *code = SIGATTN_BF16; return true;
    case at::kFloat: *code = SIGATTN_FP32; return true;
    default: return false;
  }
}

// What a call is, apart from its tensors.
struct Call {
  float scale = 0.f, bias = 0.f;
  bool bias_neg_log_lk = false, causal = false;
  int64_t max_q = 0, max_k = 0;  // packed sequences only
};
// q, k, v: (B, T, H, D), or (total, H, D) with cu_q / cu_k.  The others may be undefined.
struct Tensors {
  Tensor q, k, v, score_mod, lens_q, lens_k, cu_q, cu_k;
};

// A tensor the kernels can read in place: unit stride in the head dimension, every other stride (of dimensions that
// have one) a positive multiple of 16 bytes, base on a 16-byte boundary.  Views of a fused projection qualify.
bool readable_in_place(const Tensor& t) {
  const int64_t per16 = 16 / (int64_t)t.element_size();
  const auto sz = t.sizes();
  const auto st = t.strides();
  const int64_t n = t.dim();
  if (sz[n - 1] > 1 && st[n - 1] != 1) return false;
  for (int64_t i = 0; i < n - 1; ++i)
    if (sz[i] > 1 && (st[i] <= 0 || st[i] % per16 != 0)) return false;
  return (reinterpret_cast<uintptr_t>(t.const_data_ptr()) & 15u) == 0;
}
Tensor in_place_or_copy(const Tensor& t) { return t.numel() == 0 || readable_in_place(t) ? t : t.clone(at::MemoryFormat::Contiguous); }

// {batch, token, head} strides; a dimension of extent 1 gets what a contiguous tensor would have.
void fill_strides(int64_t* out, const Tensor& t) {
  const auto sz = t.sizes();
  const auto st = t.strides();
  const int64_t n = t.dim();
  const int64_t D = sz[n - 1], H = sz[n - 2], T = sz[n - 3];
  out[2] = H > 1 ? st[n - 2] : D;
  out[1] = T > 1 ? st[n - 3] : H * D;
  out[0] = n == 4 ? (sz[0] > 1 ? st[0] : T * H * D) : 0;
}

Tensor new_like(const Tensor& t) { return at::detail::empty_cuda(t.sizes(), t.scalar_type(), t.device(), std::nullopt); }

// The kernels' head dimension for tensors of D columns (the missing columns read as zeros).
int kernel_head_dim(int64_t D) { return D <= 64 ? 64 : 128; }

void fill_common(SigAttnParams& p, const Tensors& t, const Call& c, const Switches& sw) {
  std::memset(&p, 0, sizeof(p));
  p.struct_bytes = sizeof(p);
  int dt = 0;
  dtype_code(t.q.scalar_type(), &dt);
  p.dtype = dt;
  const bool packed = t.cu_q.defined();
  const int64_t n = t.q.dim();
  p.H = (int32_t)t.q.size(n - 2);
  p.head_cols = (int32_t)t.q.size(n - 1);
  p.D = kernel_head_dim(p.head_cols);
  if (packed) {
    p.B = (int32_t)t.cu_q.numel() - 1;
    p.Tq = (int32_t)c.max_q;
    p.Tk = (int32_t)c.max_k;
    p.total_q = (int32_t)t.q.size(0);
    p.total_k = (int32_t)t.k.size(0);
    p.cu_seqlens_q = static_cast<const int32_t*>(t.cu_q.const_data_ptr());
    p.cu_seqlens_k = static_cast<const int32_t*>(t.cu_k.const_data_ptr());
  } else {
    p.B = (int32_t)t.q.size(0);
    p.Tq = (int32_t)t.q.size(1);
    p.Tk = (int32_t)t.k.size(1);
  }
  p.flags = (c.causal ? SIGATTN_CAUSAL : 0u) | (sw.accurate ? SIGATTN_ACCURATE : 0u) |
            (c.bias_neg_log_lk ? SIGATTN_BIAS_NEG_LOG_LK : 0u);
  // rows between or behind the sequences, and rows of a sequence beyond max_seqlen, are zero in every output
  if (packed) p.flags |= SIGATTN_ZERO_GAPS;
  p.scale = c.scale;
  p.bias_scalar = c.bias;
  p.device = t.q.get_device();
  p.q = t.q.const_data_ptr();
  p.k = t.k.const_data_ptr();
  p.v = t.v.const_data_ptr();
  fill_strides(p.q_strides, t.q);
  fill_strides(p.k_strides, t.k);
  fill_strides(p.v_strides, t.v);
  if (t.lens_q.defined()) p.seq_lens_q = static_cast<const int32_t*>(t.lens_q.const_data_ptr());
  if (t.lens_k.defined()) p.seq_lens_k = static_cast<const int32_t*>(t.lens_k.const_data_ptr());
  if (t.score_mod.defined()) p.score_mod = static_cast<const float*>(t.score_mod.const_data_ptr());
  p.stream = c10::cuda::getCurrentCUDAStream(p.device).stream();
}

// One C-ABI call.  debug: outputs are poison-filled beforehand so that unwritten rows show, and the device
// is synchronised and checked after the launch.
void launch(int (*fn)(const SigAttnParams*), const SigAttnParams& p, const char* what, bool debug,
            std::initializer_list<Tensor*> outs) {
  if (debug && (!p.cu_seqlens_q || (p.flags & SIGATTN_ZERO_GAPS)))  // (calls that write every row)
    for (Tensor* t : outs) t->fill_(std::nan(""));
  const int rc = fn(&p);
  TORCH_CHECK(rc == 0, what, " failed (code ", rc, "): ", g_abi.last_error());
  if (debug) {
    const int code = g_abi.device_status(p.device);
    char site[16];
    std::snprintf(site, sizeof(site), "0x%x", (unsigned)code);
    TORCH_CHECK(code == 0, what, ": a kernel gave up on a bounded wait (site ", site,
                "); its outputs are undefined.  The health word has been cleared, the library is usable again.");
  }
}

Tensor run_forward(const Tensors& t, const Call& c, const Switches& sw) {
  Tensor out = new_like(t.q);
  if (out.numel() == 0) return out;
  if (t.cu_q.defined() && t.cu_q.numel() == 1) return out.zero_();  // no sequence at all
  SigAttnParams p;
  fill_common(p, t, c, sw);
  p.o = out.mutable_data_ptr();
  fill_strides(p.o_strides, out);
  launch(g_abi.fwd, p, "sigattn_fwd", sw.debug, {&out});
  return out;
}

void run_backward(const Tensors& t, const Call& c, const Switches& sw, const Tensor& dout, Tensor& dq, Tensor& dk, Tensor& dv) {
  dq = new_like(t.q);
  dk = new_like(t.k);
  dv = new_like(t.v);
  if (dq.numel() == 0 && dk.numel() == 0) return;
  if (t.cu_q.defined() && (dq.numel() == 0 || dk.numel() == 0 || t.cu_q.numel() == 1)) {
    for (Tensor* g : {&dq, &dk, &dv}) g->zero_();
    return;
  }
  SigAttnParams p;
  fill_common(p, t, c, sw);
  p.dout = dout.const_data_ptr();
  fill_strides(p.do_strides, dout);
  p.dq = dq.mutable_data_ptr();
  p.dk = dk.mutable_data_ptr();
  p.dv = dv.mutable_data_ptr();
  fill_strides(p.dq_strides, dq);
  fill_strides(p.dk_strides, dk);
  fill_strides(p.dv_strides, dv);
  Tensor ws;  // the fused backward's fp32 dQ accumulator (kept alive until the launch is queued)
  if (sw.split_backward) {
    p.flags |= SIGATTN_BWD_SPLIT;
  } else if (p.dtype != SIGATTN_FP32) {
    const int64_t elems = std::max<int64_t>(dq.numel() / p.head_cols * p.D, 4);
    ws = at::detail::empty_cuda({elems}, at::kFloat, t.q.device(), std::nullopt);
    p.workspace = ws.mutable_data_ptr();
    p.workspace_bytes = (size_t)elems * sizeof(float);
  }
  launch(g_abi.bwd, p, "sigattn_bwd", sw.debug, {&dq, &dk, &dv});
}

// What autograd (the output's gradient) or a saved-tensor hook hands to the backward may have any strides, and from a
// hook any type, size and device: checked and laid out again before a kernel gets the pointer.
Tensor taken(const Tensor& given, const char* name, at::IntArrayRef sizes, const Tensor& like) {
  const Tensor t = given.resolve_neg();
  TORCH_CHECK(t.layout() == at::kStrided && t.device() == like.device() && t.scalar_type() == like.scalar_type() && t.sizes() == sizes,
              "sigmoid attention backward: ", name, " must be a ", like.scalar_type(), " tensor of shape ", sizes, " on ", like.device(),
              ", got ", t.scalar_type(), " ", t.sizes(), " on ", t.device());
  return in_place_or_copy(t);
}
// The same for the per-key term, lengths and offsets (vectors of n values, or undefined).
Tensor taken_vector(const Tensor& given, const char* name, int64_t n, at::ScalarType type, const Tensor& like) {
  if (!given.defined()) return given;
  TORCH_CHECK(given.numel() == n, "sigmoid attention backward: ", name, " must have ", n, " entries, got ", given.numel());
  return given.to(like.device(), type).contiguous();
}

struct SigmoidAttentionBackward : public torch::autograd::Node {
  torch::autograd::SavedVariable q, k, v, score_mod, lens_q, lens_k, cu_q, cu_k;
  Call call;
  at::DimVector q_sizes, k_sizes;
  int64_t n_offsets = 0;  // entries of cu_q, cu_k

  std::string name() const override { return "SigmoidAttentionBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (auto* s : {&q, &k, &v, &score_mod, &lens_q, &lens_k, &cu_q, &cu_k}) s->reset_data();
  }
  torch::autograd::variable_list apply(torch::autograd::variable_list&& grads) override {
    const Switches sw = read_switches_locked();  // (before the lock: nobody waits for the GIL while holding it)
    std::lock_guard<std::mutex> lock(mutex_);
    if (!grads[0].defined()) {  // (whoever used the output had no gradient for it: zeros, as for a torch.autograd.Function)
      const Tensor qs = q.unpack(), ks = k.unpack(), vs = v.unpack();
      return {at::zeros_like(qs), at::zeros_like(ks), at::zeros_like(vs)};
    }
    const Tensor& grad = grads[0];  // (the engine has checked its type and device)
    const bool packed = n_offsets > 0;
    Tensors t;
    t.q = taken(q.unpack(), "query", q_sizes, grad);
    t.k = taken(k.unpack(), "key", k_sizes, grad);
    t.v = taken(v.unpack(), "value", k_sizes, grad);
    t.score_mod = taken_vector(score_mod.unpack(), "score_mod", packed ? k_sizes[0] : k_sizes[0] * k_sizes[1], at::kFloat, grad);
    t.lens_q = taken_vector(lens_q.unpack(), "seq_lens_q", q_sizes[0], at::kInt, grad);
    t.lens_k = taken_vector(lens_k.unpack(), "seq_lens_k", q_sizes[0], at::kInt, grad);
    t.cu_q = taken_vector(cu_q.unpack(), "cu_seqlens_q", n_offsets, at::kInt, grad);
    t.cu_k = taken_vector(cu_k.unpack(), "cu_seqlens_k", n_offsets, at::kInt, grad);
    Tensor dq, dk, dv;
    run_backward(t, call, sw, taken(grad, "grad", q_sizes, grad), dq, dk, dv);
    torch::autograd::variable_list out{dq, dk, dv};
    if (!at::GradMode::is_enabled()) return out;
    // create_graph: the gradients depend on q, k, v and grad in ways that have no formula here.  Left without a history
    // they would count as constants, and a second derivative would lack their part without a word.
    for (Tensor& g : out) g.set_requires_grad(true);
    auto once = std::make_shared<torch::autograd::DelayedError>("trying to differentiate sigmoid attention twice: its backward has no derivative",
                                                                (int64_t)out.size());
    return (*once)(std::move(out));
  }
};

bool has_tangent(const Tensor& t) { return t.defined() && t._fw_grad(/*level=*/0).defined(); }

// Forward, with the autograd node attached when a gradient can be asked for.
Tensor attention(Tensors t, const Call& c, const Switches& sw) {
  const bool grad = at::GradMode::is_enabled() && (t.q.requires_grad() || t.k.requires_grad() || t.v.requires_grad());
  // There is no forward-mode formula, and the node below knows nothing of tangents: an output without one would read as
  // a derivative of zero.
  TORCH_CHECK_NOT_IMPLEMENTED(!has_tangent(t.q) && !has_tangent(t.k) && !has_tangent(t.v) && !(grad && has_tangent(t.score_mod)),
                              "sigmoid attention has no forward-mode derivative (jvp)");
  t.q = in_place_or_copy(t.q);
  t.k = in_place_or_copy(t.k);
  t.v = in_place_or_copy(t.v);
  if (!grad) return run_forward(t, c, sw);
  using torch::autograd::SavedVariable;
  std::shared_ptr<SigmoidAttentionBackward> node(new SigmoidAttentionBackward(), torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(t.q, t.k, t.v));
  node->q = SavedVariable(t.q, false);
  node->k = SavedVariable(t.k, false);
  node->v = SavedVariable(t.v, false);
  node->score_mod = SavedVariable(t.score_mod, false);
  node->lens_q = SavedVariable(t.lens_q, false);
  node->lens_k = SavedVariable(t.lens_k, false);
  node->cu_q = SavedVariable(t.cu_q, false);
  node->cu_k = SavedVariable(t.cu_k, false);
  node->call = c;
  node->q_sizes = t.q.sizes();
  node->k_sizes = t.k.sizes();
  node->n_offsets = t.cu_q.defined() ? t.cu_q.numel() : 0;
  Tensor out = run_forward(t, c, sw);
  torch::autograd::set_history(out, node);
  return out;
}

// ---------------------------------------------------------------- Python entry points
bool is_b200(int device) {
  static std::atomic<int> known[64];
  if (device < 0 || device >= 64) return false;
  int s = known[device].load(std::memory_order_relaxed);
  if (s == 0) {
    const auto* prop = at::cuda::getDeviceProperties((c10::DeviceIndex)device);
    s = prop->major == 10 && prop->minor == 0 ? 1 : 2;
    known[device].store(s, std::memory_order_relaxed);
  }
  return s == 1;
}

bool plain(const Tensor& t) {
  using c10::DispatchKey;
  return t.defined() && t.is_cuda() && t.layout() == at::kStrided && t.unsafeGetTensorImpl()->has_storage() &&
         !t.key_set().has_any(c10::DispatchKeySet({DispatchKey::Negative, DispatchKey::Python, DispatchKey::Functionalize}));
}

// A Python dispatch mode is active (fake tensors, make_fx, operator counters, selective checkpointing) or torch.jit.trace
// is recording: what happens here would escape them, the caller takes the registered ops.
bool observed() { return c10::impl::TorchDispatchModeTLS::any_modes_set() || at::tracer::impl::is_dispatch_enabled(); }

// Argument readers: false = not plain, the caller answers None.
bool get_tensor(PyObject* o, Tensor* t) {
  if (!THPVariable_CheckExact(o)) return false;
  *t = THPVariable_Unpack(o);
  return plain(*t);
}
// int32 vector of n entries on `dev`, or None
bool get_index(PyObject* o, int64_t n, const at::Device& dev, Tensor* t) {
  if (o == Py_None) return true;
  return get_tensor(o, t) && t->scalar_type() == at::kInt && t->dim() == 1 && t->size(0) == n && t->is_contiguous() && t->device() == dev;
}
bool get_score_mod(PyObject* o, at::IntArrayRef shape, const at::Device& dev, Tensor* t) {
  if (o == Py_None) return true;
  return get_tensor(o, t) && t->scalar_type() == at::kFloat && t->sizes() == shape && t->is_contiguous() && t->device() == dev;
}
bool get_number(PyObject* o, double* v, bool* given) {
  *given = o != Py_None;
  if (!*given) return true;
  if (!PyFloat_CheckExact(o) && !PyLong_CheckExact(o)) return false;
  *v = PyFloat_AsDouble(o);
  if (!PyErr_Occurred()) return true;
  PyErr_Clear();  // an integer beyond a double: not plain, the Python path raises what it is
  return false;
}
// Same device, one supported dtype, a head dimension whose rows are whole 16-byte pieces.
bool qkv_ok(const Tensors& t) {
  int code;
  const auto dt = t.q.scalar_type();
  const int64_t D = t.q.size(t.q.dim() - 1);
  return dtype_code(dt, &code) && t.k.scalar_type() == dt && t.v.scalar_type() == dt && D > 0 && D <= 128 &&
         D % (16 / (int64_t)t.q.element_size()) == 0 &&
         t.k.device() == t.q.device() && t.v.device() == t.q.device() && is_b200(t.q.get_device());
}

PyObject* wrap(const Tensors& t, const Call& c) {
  Tensor out;
  const Switches sw = read_switches();
  {
    // the launch and the allocations need no interpreter; other Python threads may run meanwhile
    PyThreadState* state = PyEval_SaveThread();
    try {
      out = attention(t, c, sw);
    } catch (...) {
      PyEval_RestoreThread(state);
      throw;
    }
    PyEval_RestoreThread(state);
  }
  return THPVariable_Wrap(std::move(out));
}

bool nargs_ok(Py_ssize_t n, Py_ssize_t want, const char* name) {
  if (n == want && g_abi.fwd) return true;
  if (n != want) PyErr_Format(PyExc_TypeError, "%s takes %zd positional arguments, got %zd", name, want, n);
  else PyErr_SetString(PyExc_RuntimeError, "the sigattn library is not bound");
  return false;
}

// dense(q, k, v, is_causal, scale, sigmoid_bias, score_mod) -> tensor, or None: take the Python path
PyObject* py_dense(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!nargs_ok(n, 7, "dense")) return nullptr;
  if (observed()) Py_RETURN_NONE;
  Tensors t;
  Call c;
  if (!get_tensor(a[0], &t.q) || !get_tensor(a[1], &t.k) || !get_tensor(a[2], &t.v)) Py_RETURN_NONE;
  if (t.q.dim() != 4 || t.k.sizes() != t.q.sizes() || t.v.sizes() != t.q.sizes() || !qkv_ok(t)) Py_RETURN_NONE;
  const int64_t B = t.q.size(0), T = t.q.size(1), D = t.q.size(3);
  double scale = 0, bias = 0;
  bool has_scale, has_bias;
  if (!get_number(a[4], &scale, &has_scale) || !get_number(a[5], &bias, &has_bias) ||
      !get_score_mod(a[6], {B, T}, t.q.device(), &t.score_mod))
    Py_RETURN_NONE;
  const int causal = PyObject_IsTrue(a[3]);
  if (causal < 0) return nullptr;
  c.causal = causal != 0;
  c.scale = (float)(has_scale ? scale : 1.0 / std::sqrt((double)D));
  c.bias = (float)(has_bias ? bias : (T > 0 ? -std::log((double)T) : 0.0));
  return wrap(t, c);
  END_HANDLE_TH_ERRORS
}

// padded(q, k, v, seq_lens_k, seq_lens_q, is_causal, scale, sigmoid_bias, score_mod) -> tensor or None
PyObject* py_padded(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!nargs_ok(n, 9, "padded")) return nullptr;
  if (observed()) Py_RETURN_NONE;
  Tensors t;
  Call c;
  if (!get_tensor(a[0], &t.q) || !get_tensor(a[1], &t.k) || !get_tensor(a[2], &t.v)) Py_RETURN_NONE;
  if (t.q.dim() != 4 || t.k.dim() != 4 || t.v.sizes() != t.k.sizes() || !qkv_ok(t)) Py_RETURN_NONE;
  const int64_t B = t.q.size(0), Tk = t.k.size(1), D = t.q.size(3);
  if (t.k.size(0) != B || t.k.size(2) != t.q.size(2) || t.k.size(3) != D) Py_RETURN_NONE;
  double scale = 0, bias = 0;
  bool has_scale, has_bias;
  if (!get_index(a[3], B, t.q.device(), &t.lens_k) || !get_index(a[4], B, t.q.device(), &t.lens_q) ||
      !get_number(a[6], &scale, &has_scale) || !get_number(a[7], &bias, &has_bias) ||
      !get_score_mod(a[8], {B, Tk}, t.q.device(), &t.score_mod))
    Py_RETURN_NONE;
  const int causal = PyObject_IsTrue(a[5]);
  if (causal < 0) return nullptr;
  c.causal = causal != 0;
  c.scale = (float)(has_scale ? scale : 1.0 / std::sqrt((double)D));
  if (has_bias) c.bias = (float)bias;
  else if (!t.lens_k.defined()) c.bias = Tk > 0 ? (float)-std::log((double)Tk) : INFINITY;
  else c.bias_neg_log_lk = true;  // -log(valid keys), computed by the kernels from the lengths they clamp anyway
  return wrap(t, c);
  END_HANDLE_TH_ERRORS
}

// varlen(q, k, v, cu_q, cu_k, max_q, max_k, is_causal, scale, sigmoid_bias, score_mod) -> tensor or None
PyObject* py_varlen(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!nargs_ok(n, 11, "varlen")) return nullptr;
  if (observed()) Py_RETURN_NONE;
  Tensors t;
  Call c;
  if (!get_tensor(a[0], &t.q) || !get_tensor(a[1], &t.k) || !get_tensor(a[2], &t.v) || !get_tensor(a[3], &t.cu_q)) Py_RETURN_NONE;
  if (t.q.dim() != 3 || t.k.dim() != 3 || t.v.sizes() != t.k.sizes() || !qkv_ok(t)) Py_RETURN_NONE;
  const int64_t D = t.q.size(2);
  if (t.k.size(1) != t.q.size(1) || t.k.size(2) != D || t.cu_q.dim() != 1 || t.cu_q.size(0) < 1) Py_RETURN_NONE;
  double scale = 0, bias = 0;
  bool has_scale, has_bias;
  const int64_t entries = t.cu_q.size(0);
  if (a[4] == Py_None || !get_index(a[3], entries, t.q.device(), &t.cu_q) || !get_index(a[4], entries, t.q.device(), &t.cu_k) ||
      !PyLong_CheckExact(a[5]) || !PyLong_CheckExact(a[6]) || !get_number(a[8], &scale, &has_scale) ||
      !get_number(a[9], &bias, &has_bias) || !get_score_mod(a[10], {t.k.size(0)}, t.q.device(), &t.score_mod))
    Py_RETURN_NONE;
  int over_q = 0, over_k = 0;
  c.max_q = PyLong_AsLongAndOverflow(a[5], &over_q);
  c.max_k = PyLong_AsLongAndOverflow(a[6], &over_k);
  if (over_q || over_k || c.max_q > INT32_MAX || c.max_k > INT32_MAX || c.max_q < INT32_MIN || c.max_k < INT32_MIN) Py_RETURN_NONE;
  const int causal = PyObject_IsTrue(a[7]);
  if (causal < 0) return nullptr;
  c.causal = causal != 0;
  c.scale = (float)(has_scale ? scale : 1.0 / std::sqrt((double)D));
  if (has_bias) c.bias = (float)bias;
  else c.bias_neg_log_lk = true;
  return wrap(t, c);
  END_HANDLE_TH_ERRORS
}

// attention(q, k, v, score_mod, lens_q, lens_k, cu_q, cu_k, max_q, max_k, bias, scale, is_causal): inputs already
// validated and normalised by the Python path; bias None = -log(valid keys)
PyObject* py_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!nargs_ok(n, 13, "attention")) return nullptr;
  Tensors t;
  Call c;
  Tensor* dst[8] = {&t.q, &t.k, &t.v, &t.score_mod, &t.lens_q, &t.lens_k, &t.cu_q, &t.cu_k};
  for (int i = 0; i < 8; ++i) {
    if (a[i] == Py_None && i >= 3) continue;
    TORCH_CHECK_TYPE(THPVariable_Check(a[i]), "argument ", i, " is not a tensor");
    *dst[i] = THPVariable_Unpack(a[i]).resolve_neg();
    TORCH_CHECK(dst[i]->is_cuda() && dst[i]->device() == t.q.device(), "q, k, v and their lengths must be on one CUDA device, got ",
                t.q.device(), " and ", dst[i]->device());
  }
  TORCH_CHECK(qkv_ok(t), "q, k, v are not what the kernels take");
  c.max_q = PyLong_AsLong(a[8]);
  c.max_k = PyLong_AsLong(a[9]);
  c.bias_neg_log_lk = a[10] == Py_None;
  if (!c.bias_neg_log_lk) c.bias = (float)PyFloat_AsDouble(a[10]);
  c.scale = (float)PyFloat_AsDouble(a[11]);
  const int causal = PyObject_IsTrue(a[12]);
  if (PyErr_Occurred() || causal < 0) return nullptr;
  c.causal = causal != 0;
  return wrap(t, c);
  END_HANDLE_TH_ERRORS
}

PyObject* py_set_accurate(PyObject*, PyObject* arg) {
  const long v = PyLong_AsLong(arg);
  if (v == -1 && PyErr_Occurred()) return nullptr;
  g_accurate_override.store((int)v, std::memory_order_relaxed);
  Py_RETURN_NONE;
}

// bind(fwd, bwd, last_error, device_status): addresses of the C-ABI functions
PyObject* py_bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 4) {
    PyErr_SetString(PyExc_TypeError, "bind takes 4 addresses");
    return nullptr;
  }
  void* f[4];
  for (int i = 0; i < 4; ++i) {
    f[i] = PyLong_AsVoidPtr(a[i]);
    if (PyErr_Occurred()) return nullptr;
  }
  g_abi.last_error = reinterpret_cast<const char* (*)()>(f[2]);
  g_abi.device_status = reinterpret_cast<int (*)(int)>(f[3]);
  g_abi.bwd = reinterpret_cast<int (*)(const SigAttnParams*)>(f[1]);
  g_abi.fwd = reinterpret_cast<int (*)(const SigAttnParams*)>(f[0]);
  Py_RETURN_NONE;
}

#define SIG_FAST(fn) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn))
PyMethodDef g_methods[] = {
    {"dense", SIG_FAST(py_dense), METH_FASTCALL, nullptr},
    {"padded", SIG_FAST(py_padded), METH_FASTCALL, nullptr},
    {"varlen", SIG_FAST(py_varlen), METH_FASTCALL, nullptr},
    {"attention", SIG_FAST(py_attention), METH_FASTCALL, nullptr},
    {"bind", SIG_FAST(py_bind), METH_FASTCALL, nullptr},
    {"set_accurate", py_set_accurate, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_sigattn_torch", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__sigattn_torch() { return PyModule_Create(&g_module); }
