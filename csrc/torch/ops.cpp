// Host side of the operators that a layer is made of: checks, allocation, launch and autograd nodes in C++, as a Python extension over
// libtorch.  The kernels are those of libllmctl_b200.so, through its C ABI.
//
// What it is for: a launch costs the driver 4.5 us, but an operator of the Python modules (ops/functional.py, ops/attention.py,
// ops/serving.py) cost 16-17 us without gradients and 22-60 us with them, so that a small model, a decoding step or a layer's backward waited
// for Python (12 layers of width 768: 2340 us for 760 us of kernels).  Every function here takes plain tensors in the layouts that its
// kernel reads and returns None for anything else (subclasses, dispatch or function modes, functorch, tracing, forward-mode gradients, other
// types, strides, addresses): the Python operator then goes its own way, as it does for CPU tensors.
//
// Reference: none (the reference has no native layer).
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/autocast_mode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/dynamo/compiled_autograd.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <array>
#include <atomic>
#include <cstdio>
#include <initializer_list>

#include "llmctl_b200.h"

namespace {

using at::Tensor;

// ---------------------------------------------------------------------------------------------------------------------------------
// the kernel library
// ---------------------------------------------------------------------------------------------------------------------------------
#define LLMCTL_ENTRIES(X)                                                                                                         \
  X(llmctl_rmsnorm_fwd) X(llmctl_rmsnorm_bwd_bf16w) X(llmctl_rope_inplace) X(llmctl_gemm_rope_bf16) X(llmctl_gemm_bf16) X(llmctl_gemm_swiglu_bf16)               \
  X(llmctl_gemm_swiglu_bwd_bf16) X(llmctl_swiglu_bwd) X(llmctl_gemm_skinny_bf16) X(llmctl_gemm_skinny_scratch_elems) X(llmctl_flash_attn_fwd) X(llmctl_flash_attn_bwd) X(llmctl_kv_append) \
  X(llmctl_paged_attn_decode) X(llmctl_paged_attn_scratch_elems) X(llmctl_latent_kv_write) X(llmctl_latent_decode)
struct Entries {
#define X(name) decltype(&::name) name = nullptr;
  LLMCTL_ENTRIES(X)
#undef X
  const volatile uint32_t* waits = nullptr;      // != 0: a bounded wait of a kernel ran out (csrc/common/wait_status.h)
  void* (*wait_word)() = nullptr;
} lib;                                           // entries that a partial build leaves out stay null

PyObject* native_error = nullptr;                // ops.native.NativeError
PyObject* check_waits = nullptr;                 // ops.native.check_waits
PyObject* buffered_wgrad = nullptr;              // ops.functional._wgrad
std::atomic<long long> launches{0};

// Whether an entry can be called: it is there and no wait has run out (the Python operator reports that one).
template <typename F>
bool ready(F* f) {
  if (f == nullptr) return false;
  if (lib.waits == nullptr) {
    if (lib.wait_word == nullptr) return false;
    lib.waits = static_cast<const volatile uint32_t*>(lib.wait_word());
  }
  return lib.waits != nullptr && *lib.waits == 0;
}

struct Failed {                                  // of a call into the kernel library, thrown without the GIL
  const char* name;
  int rc;
};
void done(const char* name, int rc, int kernels = 1) {
  launches.fetch_add(kernels, std::memory_order_relaxed);
  if (rc != 0) throw Failed{name, rc};
}
void set_failed(const Failed& f) { PyErr_Format(native_error, "%s failed with cudaError %d", f.name, f.rc); }

// Body of an autograd node's backward: errors become the Python exceptions that the Python operators raise.
template <typename Body>
torch::autograd::variable_list node_body(const char* name, bool there, Body&& body) {
  try {
    if (there) return body();
  } catch (const Failed& f) {
    pybind11::gil_scoped_acquire gil;
    set_failed(f);
    python_error e;
    e.persist();
    throw e;
  }
  pybind11::gil_scoped_acquire gil;
  PyObject* r = PyObject_CallFunction(check_waits, "s", name);
  if (r != nullptr) PyErr_Format(native_error, "%s is not in the library", name);
  Py_XDECREF(r);
  python_error e;
  e.persist();
  throw e;
}

// ---------------------------------------------------------------------------------------------------------------------------------
// what the functions take
// ---------------------------------------------------------------------------------------------------------------------------------
// Nothing wants to see or replace the operators: no mode, transform or trace is active.
bool quiet() {
  return c10::impl::TorchDispatchModeTLS::stack_len() == 0 && at::impl::PythonTorchFunctionTLS::stack_len() == 0 &&
         !c10::impl::tls_local_dispatch_key_set().included_.has_any(
             c10::DispatchKeySet({c10::DispatchKey::FuncTorchDynamicLayerFrontMode, c10::DispatchKey::FuncTorchDynamicLayerBackMode, c10::DispatchKey::Functionalize})) &&
         !torch::jit::tracer::isTracing();
}
bool is_plain(const Tensor& t) {
  return t.is_cuda() && t.layout() == at::kStrided && !t.is_nested() &&
         !t.key_set().has_any(c10::DispatchKeySet({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                                   c10::DispatchKey::Functionalize, c10::DispatchKey::ZeroTensor, c10::DispatchKey::Negative,
                                                   c10::DispatchKey::Conjugate})) &&
         !torch::autograd::isFwGradDefined(t);
}
bool bf16(const Tensor& t) { return t.scalar_type() == at::kBFloat16; }
bool unit16(const Tensor& t) { return reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0; }
// contiguous from a 16-byte boundary, as the kernels read it
Tensor whole_units(const Tensor& t) {
  const Tensor c = t.contiguous();
  return unit16(c) ? c : c.clone();
}
// an operand of the GEMMs: rows of whole 16-byte units
bool is_matrix(const Tensor& t) { return bf16(t) && t.dim() == 2 && t.stride(1) == 1 && t.stride(0) % 8 == 0 && unit16(t); }
bool recorded(std::initializer_list<const Tensor*> ts) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : ts)
    if (t->requires_grad()) return true;
  return false;
}
void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
Tensor empty_like_on(const Tensor& t, at::IntArrayRef size, at::ScalarType type) { return at::empty(size, t.options().dtype(type).requires_grad(false)); }
Tensor new_bf16(const Tensor& t, at::IntArrayRef size) { return empty_like_on(t, size, at::kBFloat16); }
Tensor new_f32(const Tensor& t, at::IntArrayRef size) { return empty_like_on(t, size, at::kFloat); }
void* data(const Tensor& t) { return t.data_ptr(); }
const void* cdata(const Tensor& t) { return t.const_data_ptr(); }

// Arguments of a call.  A tensor argument is a torch.Tensor or Parameter itself; `ok` turns false for anything else.
struct Args {
  PyObject* const* a;
  Py_ssize_t n;
  bool ok = true;
  Tensor tensor(int i) {
    if (!THPVariable_CheckExact(a[i])) {
      ok = false;
      return Tensor();
    }
    Tensor t = THPVariable_Unpack(a[i]);
    if (!is_plain(t)) ok = false;
    return t;
  }
  Tensor optional(int i) { return a[i] == Py_None ? Tensor() : tensor(i); }
  long long integer(int i) {
    const long long v = PyLong_AsLongLong(a[i]);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return v;
  }
  double number(int i) {
    const double v = PyFloat_AsDouble(a[i]);
    if (v == -1.0 && PyErr_Occurred()) throw python_error();
    return v;
  }
};

// Runs `body` without the GIL.
template <typename Body>
auto without_gil(Body&& body) {
  pybind11::gil_scoped_release released;
  return body();
}

template <typename Body>
PyObject* call(PyObject* const* a, Py_ssize_t n, Py_ssize_t want, Body&& body) {
  HANDLE_TH_ERRORS
  if (n != want) {
    PyErr_Format(PyExc_TypeError, "takes %zd arguments (%zd given)", want, n);
    return nullptr;
  }
  try {
    Args args{a, n};
    return body(args);
  } catch (const Failed& f) {
    set_failed(f);
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}
PyObject* none() { Py_RETURN_NONE; }
PyObject* pair(const Tensor& a, PyObject* b) {
  PyObject* x = THPVariable_Wrap(a);
  PyObject* r = x == nullptr || b == nullptr ? nullptr : PyTuple_Pack(2, x, b);
  Py_XDECREF(x);
  Py_XDECREF(b);
  return r;
}

// ---------------------------------------------------------------------------------------------------------------------------------
// RMS norm
// ---------------------------------------------------------------------------------------------------------------------------------
struct NormOut {
  Tensor y, h, rstd;
};
NormOut norm_fwd(const Tensor& x, const Tensor& residual, const Tensor& w, double eps, bool keep) {
  const int64_t cols = x.size(-1), rows = x.numel() / cols;
  NormOut r{new_bf16(x, x.sizes()), residual.defined() ? new_bf16(x, x.sizes()) : x, keep ? new_f32(x, {rows}) : Tensor()};
  done("llmctl_rmsnorm_fwd", lib.llmctl_rmsnorm_fwd(cdata(x), residual.defined() ? cdata(residual) : nullptr, cdata(w), residual.defined() ? data(r.h) : nullptr, data(r.y),
                                                    keep ? static_cast<float*>(data(r.rstd)) : nullptr, static_cast<int>(rows), static_cast<int>(cols),
                                                    static_cast<float>(eps), stream()));
  return r;
}

constexpr int kNormBwdCtas = 148 * 4;

// A hook on saved tensors may give back anything: what has another type, size or device than what was kept is refused before a kernel reads it as that.
void came_back(const char* node, const Tensor& t, at::ScalarType type, at::IntArrayRef sizes, const Tensor& grad) {
  TORCH_CHECK(t.scalar_type() == type && t.sizes() == sizes && t.device() == grad.device() && is_plain(t), node, ": a saved tensor came back as ", t.scalar_type(),
              " of sizes ", t.sizes(), " on ", t.device());
}

// y = rmsnorm(x + residual) * w, and h = x + residual where there is a residual.
struct RmsNorm : torch::autograd::Function<RmsNorm> {
  static torch::autograd::variable_list forward(torch::autograd::AutogradContext* ctx, const Tensor& x, const std::optional<Tensor>& residual, const Tensor& w,
                                               double eps) {
    NormOut r = norm_fwd(x, residual.value_or(Tensor()), w, eps, true);
    ctx->save_for_backward({r.h, w, r.rstd});
    ctx->saved_data["residual"] = residual.has_value();
    if (residual.has_value()) return {r.y, r.h};
    return {r.y};
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    return node_body("llmctl_rmsnorm_bwd_bf16w", ready(lib.llmctl_rmsnorm_bwd_bf16w), [&]() -> torch::autograd::variable_list {
      const auto saved = ctx->get_saved_variables();
      const int64_t cols = grads[0].size(-1), rows = grads[0].numel() / cols;
      came_back("RmsNormBackward", saved[0], at::kBFloat16, grads[0].sizes(), grads[0]);
      came_back("RmsNormBackward", saved[1], at::kBFloat16, {cols}, grads[0]);
      came_back("RmsNormBackward", saved[2], at::kFloat, {rows}, grads[0]);
      const Tensor h = whole_units(saved[0]), w = whole_units(saved[1]), rstd = whole_units(saved[2]);
      const bool residual = ctx->saved_data["residual"].toBool();
      const Tensor dy = whole_units(grads[0]), dres = residual ? whole_units(grads[1]) : Tensor();
      Tensor dx = new_bf16(h, h.sizes()), dw = new_bf16(w, {cols});
      const int ctas = static_cast<int>(rows < kNormBwdCtas ? rows : kNormBwdCtas);
      Tensor scratch = new_f32(h, {ctas * cols});
      done("llmctl_rmsnorm_bwd_bf16w", lib.llmctl_rmsnorm_bwd_bf16w(cdata(dy), cdata(h), cdata(w), static_cast<const float*>(cdata(rstd)), residual ? cdata(dres) : nullptr,
                                                                    data(dx), data(dw), static_cast<float*>(data(scratch)), ctas, static_cast<int>(rows),
                                                                    static_cast<int>(cols), stream()), 2);
      return {dx, residual ? dx : Tensor(), dw, Tensor()};
    });
  }
};

// rmsnorm(x, residual or None, w, eps) -> (y, h)
PyObject* py_rmsnorm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return call(a, n, 4, [&](Args& args) -> PyObject* {
    const Tensor x = args.tensor(0), residual = args.optional(1), w = args.tensor(2);
    const double eps = args.number(3);
    if (!args.ok || !quiet() || !ready(lib.llmctl_rmsnorm_fwd) || !bf16(x) || !bf16(w) || x.dim() < 1 || x.numel() == 0 || !x.is_contiguous() || w.dim() != 1 ||
        w.size(0) != x.size(-1) || !w.is_contiguous() || !unit16(x) || !unit16(w))
      return none();
    if (residual.defined() && (!bf16(residual) || !residual.is_contiguous() || residual.sizes() != x.sizes() || !unit16(residual))) return none();
    const bool grad = residual.defined() ? recorded({&x, &residual, &w}) : recorded({&x, &w});
    Tensor y, h;
    without_gil([&] {
      if (grad) {
        const auto out = RmsNorm::apply(x, residual.defined() ? std::optional<Tensor>(residual) : std::nullopt, w, eps);
        y = out[0];
        if (residual.defined()) h = out[1];
      } else {
        NormOut r = norm_fwd(x, residual, w, eps, false);
        y = r.y;
        h = r.h;
      }
    });
    if (residual.defined()) return pair(y, THPVariable_Wrap(h));
    Py_INCREF(a[0]);
    return pair(y, a[0]);
  });
}

// ---------------------------------------------------------------------------------------------------------------------------------
// GEMMs
// ---------------------------------------------------------------------------------------------------------------------------------
void gemm(const Tensor& a, const Tensor& b, const Tensor& c, bool a_mn, bool b_mn, bool accumulate, int tile_n, int max_ctas) {
  const int64_t M = c.size(0), N = c.size(1), K = a_mn ? a.size(0) : a.size(1);
  done("llmctl_gemm_bf16", lib.llmctl_gemm_bf16(cdata(a), cdata(b), data(c), static_cast<int>(M), static_cast<int>(N), static_cast<int>(K), a.stride(0), b.stride(0),
                                                c.stride(0), a_mn, b_mn, c.scalar_type() == at::kFloat, accumulate, tile_n, max_ctas, stream()));
}

// gemm(a, b, a_mn, b_mn, out or None, fp32, accumulate, tile_n, max_ctas) -> out
PyObject* py_gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return call(a, n, 9, [&](Args& args) -> PyObject* {
    const Tensor x = args.tensor(0), y = args.tensor(1);
    Tensor out = args.optional(4);
    const bool a_mn = args.integer(2), b_mn = args.integer(3), fp32 = args.integer(5), accumulate = args.integer(6);
    const int tile_n = static_cast<int>(args.integer(7)), max_ctas = static_cast<int>(args.integer(8));
    if (!args.ok || !quiet() || !ready(lib.llmctl_gemm_bf16) || !bf16(x) || !bf16(y) || x.dim() != 2 || y.dim() != 2 || x.stride(1) != 1 || y.stride(1) != 1) return none();
    const int64_t M = x.size(a_mn ? 1 : 0), N = y.size(b_mn ? 1 : 0);
    if (x.size(a_mn ? 0 : 1) != y.size(b_mn ? 0 : 1)) return none();
    if (out.defined() ? out.dim() != 2 || out.size(0) != M || out.size(1) != N || out.stride(1) != 1 || (out.scalar_type() != at::kFloat && !bf16(out)) : accumulate)
      return none();
    without_gil([&] {
      if (!out.defined()) out = empty_like_on(x, {M, N}, fp32 ? at::kFloat : at::kBFloat16);
      gemm(x, y, out, a_mn, b_mn, accumulate, tile_n, max_ctas);
    });
    return THPVariable_Wrap(out);
  });
}

// rows of the last dimension as a matrix for the GEMMs, or undefined
Tensor as_rows(const Tensor& x) {
  if (x.dim() == 2) return is_matrix(x) ? x : Tensor();
  if (x.dim() < 1 || !x.is_contiguous()) return Tensor();
  const Tensor r = x.view({-1, x.size(-1)});
  return is_matrix(r) ? r : Tensor();
}
Tensor as_shape_of(const Tensor& y, const Tensor& x) {
  if (x.dim() == 2) return y;
  auto size = x.sizes().vec();
  size.back() = y.size(1);
  return y.view(size);
}

// dyT x of a weight; where the weight has a buffer for its gradient (main_grad, looked up now: it may come and go between the passes) through the
// Python operator, which accumulates into it and tells its owner, and nothing is returned.  What the owner runs then is a program's own: no
// dispatch key may be left out around it.
Tensor wgrad(const Tensor& dy, const Tensor& x, const Tensor& w, int tile_n) {
  {
    pybind11::gil_scoped_acquire gil;
    PyObject *o = THPVariable_Wrap(w), *dict = PyObject_GenericGetDict(o, nullptr);
    PyObject* buffer = dict == nullptr ? nullptr : PyDict_GetItemString(dict, "main_grad");
    const bool buffered = buffer != nullptr && buffer != Py_None;
    PyErr_Clear();
    Py_XDECREF(dict);
    PyObject* r = nullptr;
    if (buffered) {
      PyObject *a = THPVariable_Wrap(dy), *b = THPVariable_Wrap(x);
      r = PyObject_CallFunctionObjArgs(buffered_wgrad, a, b, o, nullptr);
      Py_XDECREF(a);
      Py_XDECREF(b);
    }
    Py_DECREF(o);
    if (buffered) {
      if (r == nullptr) {
        python_error e;
        e.persist();
        throw e;
      }
      Tensor out = r == Py_None ? Tensor() : THPVariable_Unpack(r);
      Py_DECREF(r);
      return out;
    }
  }
  at::AutoDispatchBelowADInplaceOrView below;
  Tensor dw = new_bf16(w, w.sizes());
  gemm(dy, x, dw, true, true, false, tile_n, 0);
  return dw;
}
Tensor dgrad(const Tensor& dy, const Tensor& w, int tile_n) {
  at::AutoDispatchBelowADInplaceOrView below;
  Tensor dx = new_bf16(dy, {dy.size(0), w.size(1)});
  gemm(dy, w, dx, false, true, false, tile_n, 0);
  return dx;
}

// A recorded operator as a node of its own: torch::autograd::Function looks its arguments up by name, and wraps and checks them in ways that
// operators which return one new tensor have no use for (forward and backward of a small attention 72 us; the engine alone takes 29).  `T` says
// what its backward needs (kEntry, there()) and is
//   static variable_list gradients(const Numbers&, const Tensor& grad, Kept saved, unsigned wants)
// with a bit of `wants` for each gradient that is asked for, unless kAllAtOnce.  Nothing else may enter: compiled autograd calls it with tensors of its own, and
// for any call whose numbers and `wants` are the same.
namespace compiled = torch::dynamo::autograd;
using Kept = c10::ArrayRef<Tensor>;
constexpr unsigned kMostKept = 5;
template <typename T, typename Numbers>
struct Recorded : torch::autograd::Node {
  c10::SmallVector<torch::autograd::SavedVariable, kMostKept> saved;
  int output = -1;                                 // which of them is what the forward returned
  Numbers numbers;

  static std::shared_ptr<T> make(torch::autograd::edge_list&& next, Numbers numbers) {
    std::shared_ptr<T> node(new T(), torch::autograd::deleteNode);
    node->set_next_edges(std::move(next));
    node->numbers = std::move(numbers);
    return node;
  }
  c10::SmallVector<Tensor, kMostKept> kept() {
    c10::SmallVector<Tensor, kMostKept> ts;
    for (size_t i = 0; i < saved.size(); ++i) ts.push_back(static_cast<int>(i) == output ? saved[i].unpack(getptr()) : saved[i].unpack());
    return ts;
  }
  unsigned wants() const {
    unsigned bits = 0;
    if constexpr (!T::kAllAtOnce)
      for (uint32_t i = 0; i < num_outputs(); ++i) bits |= static_cast<unsigned>(task_should_compute_output(i)) << i;
    return bits;
  }
  static torch::autograd::variable_list run(const Numbers& numbers, const Tensor& grad, Kept kept, unsigned wants) {
    return node_body(T::kEntry, T::there(), [&] { return T::gradients(numbers, grad, kept, wants); });
  }

  torch::autograd::variable_list apply(torch::autograd::variable_list&& grads) override {
    if (!grads[0].defined()) return torch::autograd::variable_list(num_outputs());
    c10::SmallVector<Tensor, kMostKept> ts;
    {
      std::lock_guard<std::mutex> hold(mutex_);
      ts = kept();
    }
    return run(numbers, grads[0], ts, wants());
  }
  void release_variables() override {
    std::lock_guard<std::mutex> hold(mutex_);
    for (auto& t : saved) t.reset_data();
  }
  void compiled_args(compiled::CompiledNodeArgs& args) const override {
    for (size_t i = 0; i < saved.size(); ++i) args.collect(saved[i], static_cast<int>(i) == output);
    numbers.collect(args);
    args.collect(static_cast<int64_t>(wants()));
  }
  torch::autograd::variable_list apply_with_saved(const torch::autograd::variable_list& grads, compiled::SwapSavedVariables& swap) override {
    for (auto& t : saved) swap.before(t);
    compiled::PackedArgs packed;
    std::vector<at::TypePtr> schema;
    for (const Tensor& t : kept()) {
      packed.pack(t);
      schema.push_back(compiled::IValuePacker<Tensor>::packed_type());
    }
    const size_t outputs = num_outputs(), n = saved.size();
    auto later = [numbers = numbers, wants = wants(), outputs, n](const torch::autograd::variable_list& grads, const std::vector<c10::IValue>& stack) {
      compiled::PackedArgs packed(stack);
      c10::SmallVector<Tensor, kMostKept> kept;
      for (size_t i = 0; i < n; ++i) kept.push_back(packed.unpack<Tensor>());
      return grads[0].defined() ? run(numbers, grads[0], kept, wants) : torch::autograd::variable_list(outputs);
    };
    const auto& compiler = compiled::getPyCompilerInterface();
    const std::string id = compiler->bind_function(swap.get_py_compiler(), name(), later, schema, /*is_custom_function=*/true, /*is_traceable=*/false);
    const auto metadata = compiled::IValuePacker<std::vector<std::optional<torch::autograd::InputMetadata>>>::pack(compiled::get_input_metadata(next_edges()));
    auto out = compiler->call_function(swap.get_py_compiler(), "apply_functional", id, grads, packed.vec(), metadata);
    for (auto& t : saved) swap.after(t);
    return out;
  }
};

struct ProductNumbers {
  int tile_n = 0;
  std::vector<std::array<int64_t, 2>> sizes;       // of the saved matrices
  void collect(compiled::CompiledNodeArgs& args) const {
    args.collect(static_cast<int64_t>(tile_n));
    for (const auto& s : sizes) {
      args.collect(s[0]);
      args.collect(s[1]);
    }
  }
};
template <typename T>
struct Product : Recorded<T, ProductNumbers> {
  static constexpr bool kAllAtOnce = false;
  void keep(std::initializer_list<const Tensor*> ts) {
    for (const Tensor* t : ts) {
      this->saved.emplace_back(*t, false);
      this->numbers.sizes.push_back({t->size(0), t->size(1)});
    }
  }
  // a hook on saved tensors may give back anything: what the kernels cannot read is refused
  static void check(const ProductNumbers& numbers, Kept kept, const Tensor& grad) {
    for (size_t i = 0; i < kept.size(); ++i) {
      const Tensor& t = kept[i];
      TORCH_CHECK(t.device() == grad.device() && is_matrix(t) && t.size(0) == numbers.sizes[i][0] && t.size(1) == numbers.sizes[i][1], T::kName, ": a saved matrix came back as ",
                  t.scalar_type(), " of sizes ", t.sizes(), " on ", t.device());
    }
  }
  // the gradient as an operand
  static Tensor rows(const Tensor& g) {
    at::AutoDispatchBelowADInplaceOrView below;
    return is_matrix(g) ? g : whole_units(g);
  }
  std::string name() const override { return T::kName; }
};

struct LinearNode final : Product<LinearNode> {
  static constexpr const char *kName = "LinearBackward", *kEntry = "llmctl_gemm_bf16";
  static bool there() { return ready(lib.llmctl_gemm_bf16); }
  static Tensor record(const Tensor& x, const Tensor& w, int tile_n) {
    auto node = make(torch::autograd::collect_next_edges(x, w), {tile_n, {}});
    node->keep({&x, &w});
    Tensor y = new_bf16(x, {x.size(0), w.size(0)});
    gemm(x, w, y, false, false, false, tile_n, 0);
    torch::autograd::set_history(y, node);
    return y;
  }
  static torch::autograd::variable_list gradients(const ProductNumbers& z, const Tensor& grad, Kept kept, unsigned wants) {
    check(z, kept, grad);
    const Tensor &x = kept[0], &w = kept[1], dy = rows(grad);
    Tensor dx, dw;
    if (wants & 1) dx = dgrad(dy, w, z.tile_n);
    if (wants & 2) dw = wgrad(dy, x, w, z.tile_n);
    return {dx, dw};
  }
};

// act = swiglu(x @ w.T) and the product before
std::pair<Tensor, Tensor> up_and_activate(const Tensor& x, const Tensor& w, bool keep) {
  const int64_t M = x.size(0), F = w.size(0) / 2;
  Tensor act = new_bf16(x, {M, F}), gu = keep ? new_bf16(x, {M, 2 * F}) : Tensor();
  done("llmctl_gemm_swiglu_bf16", lib.llmctl_gemm_swiglu_bf16(cdata(x), cdata(w), keep ? data(gu) : nullptr, data(act), static_cast<int>(M), static_cast<int>(F),
                                                              static_cast<int>(x.size(1)), x.stride(0), w.stride(0), 2 * F, F, stream()));
  return {act, gu};
}

struct LinearSwigluNode final : Product<LinearSwigluNode> {
  static constexpr const char *kName = "LinearSwigluBackward", *kEntry = "llmctl_swiglu_bwd";
  static bool there() { return ready(lib.llmctl_swiglu_bwd) && lib.llmctl_gemm_bf16; }
  static Tensor record(const Tensor& x, const Tensor& w) {
    auto node = make(torch::autograd::collect_next_edges(x, w), {});
    const auto [act, gu] = up_and_activate(x, w, true);
    node->keep({&x, &w, &gu});
    torch::autograd::set_history(act, node);
    return act;
  }
  static torch::autograd::variable_list gradients(const ProductNumbers& z, const Tensor& grad, Kept kept, unsigned wants) {
    check(z, kept, grad);
    const Tensor &x = kept[0], &w = kept[1], dgu = [&] {
      at::AutoDispatchBelowADInplaceOrView below;
      const Tensor gu = whole_units(kept[2]), dact = whole_units(grad);         // the kernel's one row stride is that of gu and of its gradient
      Tensor d = new_bf16(gu, gu.sizes());
      done("llmctl_swiglu_bwd", lib.llmctl_swiglu_bwd(cdata(dact), cdata(gu), data(d), static_cast<int>(gu.size(0)), static_cast<int>(gu.size(1) / 2), gu.stride(0), ::stream()));
      return d;
    }();
    Tensor dx, dw;
    if (wants & 1) dx = dgrad(dgu, w, 0);
    if (wants & 2) dw = wgrad(dgu, x, w, 0);
    return {dx, dw};
  }
};

// swiglu(x @ up.T) @ down.T: the gradient of the product of the two halves goes straight into theirs
struct SwigluMlpNode final : Product<SwigluMlpNode> {
  static constexpr const char *kName = "SwigluMlpBackward", *kEntry = "llmctl_gemm_swiglu_bwd_bf16";
  static bool there() { return ready(lib.llmctl_gemm_swiglu_bwd_bf16) && lib.llmctl_gemm_bf16; }
  static Tensor record(const Tensor& x, const Tensor& up, const Tensor& down) {
    auto node = make(torch::autograd::collect_next_edges(x, up, down), {});
    const auto [act, gu] = up_and_activate(x, up, true);
    node->keep({&x, &up, &down, &gu, &act});
    Tensor y = new_bf16(x, {x.size(0), down.size(0)});
    gemm(act, down, y, false, false, false, 0, 0);
    torch::autograd::set_history(y, node);
    return y;
  }
  static torch::autograd::variable_list gradients(const ProductNumbers& z, const Tensor& grad, Kept kept, unsigned wants) {
    check(z, kept, grad);
    const Tensor &x = kept[0], &up = kept[1], &down = kept[2], &act = kept[4], dy = rows(grad);
    Tensor dgu, dx, d_up, d_down;
    if (wants & 3) {
      at::AutoDispatchBelowADInplaceOrView below;
      const Tensor gu = whole_units(kept[3]);                                   // the kernel's one row stride is that of gu and of its gradient
      dgu = new_bf16(gu, gu.sizes());
      done("llmctl_gemm_swiglu_bwd_bf16",
           lib.llmctl_gemm_swiglu_bwd_bf16(cdata(dy), cdata(down), cdata(gu), data(dgu), static_cast<int>(gu.size(0)), static_cast<int>(gu.size(1) / 2),
                                           static_cast<int>(dy.size(1)), dy.stride(0), down.stride(0), gu.stride(0), ::stream()));
    }
    if (wants & 4) d_down = wgrad(dy, act, down, 0);
    if (wants & 1) dx = dgrad(dgu, up, 0);
    if (wants & 2) d_up = wgrad(dgu, x, up, 0);
    return {dx, d_up, d_down};
  }
};

// linear(x, w, tile_n, workspace or None) -> x @ w.T; where no gradient is recorded few rows take the decode GEMM, whose partials and tickets
// workspace(x, floats of partials, stream) returns
PyObject* py_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return call(a, n, 4, [&](Args& args) -> PyObject* {
    const Tensor x = args.tensor(0), w = args.tensor(1);
    const int tile_n = static_cast<int>(args.integer(2));
    if (!args.ok || !quiet() || !is_matrix(w) || x.numel() == 0) return none();
    if (recorded({&x, &w})) {
      if (!ready(lib.llmctl_gemm_bf16) || !is_matrix(x) || x.size(1) != w.size(1) || w.size(0) % 8 || w.size(1) % 8) return none();
      return THPVariable_Wrap(without_gil([&] { return LinearNode::record(x, w, tile_n); }));
    }
    const Tensor rows = as_rows(x);
    if (!rows.defined() || rows.size(1) != w.size(1)) return none();
    const bool skinny = a[3] != Py_None;
    if (skinny ? !ready(lib.llmctl_gemm_skinny_bf16) || !lib.llmctl_gemm_skinny_scratch_elems : !ready(lib.llmctl_gemm_bf16) || w.size(0) % 8) return none();
    Tensor ws, counters;
    if (skinny) {
      PyObject* pair = PyObject_CallFunction(a[3], "OLN", a[0], lib.llmctl_gemm_skinny_scratch_elems(static_cast<int>(rows.size(0)), static_cast<int>(w.size(0)),
                                                                                                      static_cast<int>(w.size(1)), 0), PyLong_FromVoidPtr(stream()));
      if (pair == nullptr) throw python_error();
      ws = THPVariable_Unpack(PyTuple_GET_ITEM(pair, 0));
      counters = THPVariable_Unpack(PyTuple_GET_ITEM(pair, 1));
      Py_DECREF(pair);
    }
    Tensor y = without_gil([&] {
      Tensor out = new_bf16(x, {rows.size(0), w.size(0)});
      if (skinny)
        done("llmctl_gemm_skinny_bf16",
             lib.llmctl_gemm_skinny_bf16(cdata(rows), cdata(w), data(out), static_cast<int>(rows.size(0)), static_cast<int>(w.size(0)), static_cast<int>(w.size(1)),
                                         rows.stride(0), w.stride(0), out.stride(0), static_cast<float*>(data(ws)), ws.numel(),
                                         static_cast<unsigned int*>(data(counters)), static_cast<int>(counters.numel()), 0, stream()));
      else
        gemm(rows, w, out, false, false, false, tile_n, 0);
      return as_shape_of(out, x);
    });
    return THPVariable_Wrap(y);
  });
}

// gemm_swiglu(x, w, keep) -> (swiglu(x @ w.T), the product before or None)
PyObject* py_gemm_swiglu(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return call(a, n, 3, [&](Args& args) -> PyObject* {
    const Tensor x = args.tensor(0), w = args.tensor(1);
    const bool keep = args.integer(2);
    if (!args.ok || !quiet() || !ready(lib.llmctl_gemm_swiglu_bf16) || !is_matrix(x) || !is_matrix(w) || x.size(1) != w.size(1) || w.size(0) % 16) return none();
    Tensor act, gu;
    without_gil([&] { std::tie(act, gu) = up_and_activate(x, w, keep); });
    if (keep) return pair(act, THPVariable_Wrap(gu));
    Py_INCREF(Py_None);
    return pair(act, Py_None);
  });
}

// mlp(x, w_up, w_down, least, fused) -> swiglu(x @ w_up.T) @ w_down.T for more than `least` rows; where a gradient is recorded as one node if the
// down-projection has at least `fused` rows (and the product before it needs a gradient), else as two
PyObject* py_mlp(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return call(a, n, 5, [&](Args& args) -> PyObject* {
    const Tensor x = args.tensor(0), up = args.tensor(1), down = args.tensor(2);
    const int least = static_cast<int>(args.integer(3)), fused = static_cast<int>(args.integer(4));
    if (!args.ok || !quiet() || !ready(lib.llmctl_gemm_swiglu_bf16) || !ready(lib.llmctl_gemm_bf16) || !is_matrix(up) || !is_matrix(down) || x.numel() == 0 ||
        up.size(0) % 16 || down.size(0) % 8 || down.size(1) != up.size(0) / 2)
      return none();
    if (recorded({&x, &up, &down})) {
      if (!ready(lib.llmctl_gemm_swiglu_bwd_bf16) || !ready(lib.llmctl_swiglu_bwd) || !is_matrix(x) || x.size(1) != up.size(1) || x.size(0) <= least || up.size(1) % 8) return none();
      return THPVariable_Wrap(without_gil([&] {
        const bool first = x.requires_grad() || up.requires_grad();
        if (first && down.size(0) >= fused) return SwigluMlpNode::record(x, up, down);
        return LinearNode::record(first ? LinearSwigluNode::record(x, up) : up_and_activate(x, up, false).first, down, 0);
      }));
    }
    const Tensor rows = as_rows(x);
    if (!rows.defined() || rows.size(1) != up.size(1) || rows.size(0) <= least) return none();
    Tensor y = without_gil([&] {
      Tensor out = new_bf16(x, {rows.size(0), down.size(0)});
      gemm(up_and_activate(rows, up, false).first, down, out, false, false, false, 0, 0);
      return as_shape_of(out, x);
    });
    return THPVariable_Wrap(y);
  });
}

// ---------------------------------------------------------------------------------------------------------------------------------
// attention
// ---------------------------------------------------------------------------------------------------------------------------------
struct AttnOut {
  Tensor o, lse;
};
// q, k, v: [B, S, H, D] as attention_ok takes them
bool attention_ok(const Tensor& q, const Tensor& k, const Tensor& v, bool causal) {
  if (q.dim() != 4 || !bf16(q)) return false;
  const int64_t B = q.size(0), S = q.size(1), H = q.size(2), D = q.size(3);
  if ((D != 64 && D != 128) || B < 1 || S < 1 || H < 1 || (!causal && S % 128)) return false;
  for (const Tensor* t : {&q, &k, &v})
    if (t->dim() != 4 || !bf16(*t) || t->sizes() != q.sizes() || t->stride(3) != 1 || t->stride(2) != D || (B > 1 && t->stride(0) != S * t->stride(1)) ||
        t->stride(1) % 8 || !unit16(*t))
      return false;
  return true;
}
AttnOut attn_fwd(const Tensor& q, const Tensor& k, const Tensor& v, double scale, bool causal, bool keep) {
  const int64_t B = q.size(0), S = q.size(1), H = q.size(2), D = q.size(3);
  AttnOut r{new_bf16(q, {B, S, H, D}), keep ? new_f32(q, {B, H, S}) : Tensor()};
  done("llmctl_flash_attn_fwd", lib.llmctl_flash_attn_fwd(cdata(q), cdata(k), cdata(v), data(r.o), keep ? static_cast<float*>(data(r.lse)) : nullptr, static_cast<int>(B),
                                                          static_cast<int>(S), static_cast<int>(H), static_cast<int>(D), q.stride(1), k.stride(1), v.stride(1),
                                                          H * D, static_cast<float>(scale), causal, stream()));
  return r;
}
// dq | dk | dv, packed like the projection that made q | k | v, so that the weight gradient that follows sees one tensor
Tensor attn_bwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse, const Tensor& grad, double scale, bool causal) {
  const int64_t B = q.size(0), S = q.size(1), H = q.size(2), D = q.size(3);
  const Tensor d_o = whole_units(grad);
  Tensor d = new_bf16(q, {B, S, 3, H, D});
  Tensor scratch = new_f32(q, {2 * B * H * ((S + 127) / 128 * 128) + 2});
  char* at = static_cast<char*>(data(d));
  done("llmctl_flash_attn_bwd", lib.llmctl_flash_attn_bwd(cdata(q), cdata(k), cdata(v), cdata(o), cdata(d_o), static_cast<const float*>(cdata(lse)), at, at + 2 * H * D,
                                                          at + 4 * H * D, static_cast<float*>(data(scratch)), static_cast<int>(B), static_cast<int>(S),
                                                          static_cast<int>(H), static_cast<int>(D), q.stride(1), k.stride(1), v.stride(1), H * D, 3 * H * D,
                                                          static_cast<float>(scale), causal, stream()), 2);
  return d;
}

struct AttentionNumbers {
  double scale = 0;
  bool causal = true;
  void collect(compiled::CompiledNodeArgs& args) const {
    args.collect(scale);
    args.collect(causal);
  }
};
struct FlashAttention final : Recorded<FlashAttention, AttentionNumbers> {
  static constexpr const char* kEntry = "llmctl_flash_attn_bwd";
  static constexpr bool kAllAtOnce = true;
  static bool there() { return ready(lib.llmctl_flash_attn_bwd); }
  static Tensor record(const Tensor& q, const Tensor& k, const Tensor& v, double scale, bool causal) {
    auto node = make(torch::autograd::collect_next_edges(q, k, v), {scale, causal});
    for (const Tensor* t : {&q, &k, &v}) node->saved.emplace_back(*t, false);
    AttnOut r = attn_fwd(q, k, v, scale, causal, true);
    torch::autograd::set_history(r.o, node);
    node->output = 3;
    node->saved.emplace_back(r.o, true);
    node->saved.emplace_back(r.lse, false);
    return r.o;
  }
  static torch::autograd::variable_list gradients(const AttentionNumbers& z, const Tensor& grad, Kept kept, unsigned) {
    const Tensor &q = kept[0], &k = kept[1], &v = kept[2], &o = kept[3], &lse = kept[4];
    const auto here = grad.device();
    TORCH_CHECK(q.device() == here && k.device() == here && v.device() == here && o.device() == here && attention_ok(q, k, v, z.causal) && bf16(o) &&
                    o.is_contiguous() && unit16(o) && o.sizes() == q.sizes() && lse.device() == here && lse.scalar_type() == at::kFloat && lse.is_contiguous() &&
                    lse.numel() == q.size(0) * q.size(1) * q.size(2) && grad.sizes() == q.sizes(),
                "FlashAttentionBackward: saved tensors came back in other forms");
    at::AutoDispatchBelowADInplaceOrView below;
    const Tensor d = attn_bwd(q, k, v, o, lse, grad, z.scale, z.causal);
    return {d.select(2, 0), d.select(2, 1), d.select(2, 2)};
  }
  std::string name() const override { return "FlashAttentionBackward"; }
};

// attention(q, k, v, scale, causal) -> [B, S, H, D]
PyObject* py_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return call(a, n, 5, [&](Args& args) -> PyObject* {
    const Tensor q = args.tensor(0), k = args.tensor(1), v = args.tensor(2);
    const double scale = args.number(3);
    const bool causal = args.integer(4);
    if (!args.ok || !quiet() || !ready(lib.llmctl_flash_attn_fwd) || !lib.llmctl_flash_attn_bwd || !attention_ok(q, k, v, causal)) return none();
    const bool grad = recorded({&q, &k, &v});
    Tensor o = without_gil([&] { return grad ? FlashAttention::record(q, k, v, scale, causal) : attn_fwd(q, k, v, scale, causal, false).o; });
    return THPVariable_Wrap(o);
  });
}

// The first 2 H heads of packed rows q | k | v, rotated in place.
void rope(const Tensor& x, const Tensor& cos, const Tensor& sin, const Tensor& positions, int64_t S, int64_t heads, int64_t D, float sign) {
  done("llmctl_rope_inplace", lib.llmctl_rope_inplace(data(x), x.stride(0), static_cast<int>(x.size(0)), static_cast<int>(heads), static_cast<int>(D),
                                                      static_cast<const float*>(cdata(cos)), static_cast<const float*>(cdata(sin)),
                                                      positions.defined() ? static_cast<const int*>(cdata(positions)) : nullptr, static_cast<int>(S), sign, stream()));
}
struct Packed {
  Tensor q, k, v;
};
Packed unpack(const Tensor& qkv, int64_t B, int64_t S, int64_t H, int64_t D) {
  const Tensor v5 = qkv.detach().view({B, S, 3, H, D});
  return {v5.select(2, 0), v5.select(2, 1), v5.select(2, 2)};
}

struct RopeAttention : torch::autograd::Function<RopeAttention> {
  // rotates qkv in place: the product that made it keeps no copy of its output
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& qkv, const Tensor& cos, const Tensor& sin, const std::optional<Tensor>& positions,
                        int64_t B, int64_t S, int64_t H, int64_t D, double scale) {
    rope(qkv, cos, sin, positions.value_or(Tensor()), S, 2 * H, D, 1.f);
    const Packed p = unpack(qkv, B, S, H, D);
    AttnOut r = attn_fwd(p.q, p.k, p.v, scale, true, true);
    ctx->save_for_backward({qkv.detach(), r.o, r.lse, cos, sin, positions.value_or(Tensor())});
    ctx->saved_data["sizes"] = std::vector<int64_t>{B, S, H, D};
    ctx->saved_data["tables"] = std::vector<int64_t>{cos.numel(), sin.numel()};
    ctx->saved_data["scale"] = scale;
    return r.o.view({B * S, H * D});
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    return node_body("llmctl_flash_attn_bwd", ready(lib.llmctl_flash_attn_bwd), [&]() -> torch::autograd::variable_list {
      const auto s = ctx->get_saved_variables();
      const auto z = ctx->saved_data["sizes"].toIntVector();
      const int64_t B = z[0], S = z[1], H = z[2], D = z[3];
      const char* node = "RopeAttentionBackward";
      came_back(node, s[0], at::kBFloat16, {B * S, 3 * H * D}, grads[0]);
      came_back(node, s[1], at::kBFloat16, {B, S, H, D}, grads[0]);
      came_back(node, s[2], at::kFloat, {B, H, S}, grads[0]);
      const auto tables = ctx->saved_data["tables"].toIntVector();
      for (int i = 0; i < 2; ++i) {
        came_back(node, s[3 + i], at::kFloat, s[3 + i].sizes(), grads[0]);
        TORCH_CHECK(s[3 + i].numel() == tables[i], node, ": a table came back with ", s[3 + i].numel(), " numbers");
      }
      if (s[5].defined()) {
        came_back(node, s[5], at::kInt, s[5].sizes(), grads[0]);
        TORCH_CHECK(s[5].numel() == B * S, node, ": ", s[5].numel(), " positions came back");
      }
      const Packed p = unpack(whole_units(s[0]), B, S, H, D);
      const Tensor d = attn_bwd(p.q, p.k, p.v, whole_units(s[1]), whole_units(s[2]), grads[0].reshape({B, S, H, D}), ctx->saved_data["scale"].toDouble(), true).view({B * S, 3 * H * D});
      rope(d, whole_units(s[3]), whole_units(s[4]), s[5].defined() ? whole_units(s[5]) : s[5], S, 2 * H, D, -1.f);
      return {d, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    });
  }
};

// rope_attention(qkv, cos, sin, positions or None, B, S, H, D, scale) -> [B * S, H * D]
PyObject* py_rope_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return call(a, n, 9, [&](Args& args) -> PyObject* {
    const Tensor qkv = args.tensor(0), cos = args.tensor(1), sin = args.tensor(2), positions = args.optional(3);
    const int64_t B = args.integer(4), S = args.integer(5), H = args.integer(6), D = args.integer(7);
    const double scale = args.number(8);
    if (!args.ok || !quiet() || !ready(lib.llmctl_rope_inplace) || !ready(lib.llmctl_flash_attn_fwd) || !lib.llmctl_flash_attn_bwd || !bf16(qkv) || qkv.dim() != 2 ||
        !qkv.is_contiguous() || B < 1 || S < 1 || H < 1 || (D != 64 && D != 128) || qkv.size(0) != B * S || qkv.size(1) != 3 * H * D || !unit16(qkv) ||
        cos.scalar_type() != at::kFloat || sin.scalar_type() != at::kFloat || !cos.is_contiguous() || !sin.is_contiguous() || cos.requires_grad() || sin.requires_grad())
      return none();
    if (positions.defined() && (positions.scalar_type() != at::kInt || !positions.is_contiguous() || positions.numel() != B * S)) return none();
    if (qkv.is_leaf() && qkv.requires_grad()) return none();
    const bool grad = recorded({&qkv});
    Tensor o = without_gil([&] {
      if (grad) return RopeAttention::apply(qkv, cos, sin, positions.defined() ? std::optional<Tensor>(positions) : std::nullopt, B, S, H, D, scale);
      if (!qkv.is_inference()) qkv.unsafeGetTensorImpl()->bump_version();
      rope(qkv, cos, sin, positions, S, 2 * H, D, 1.f);
      const Packed p = unpack(qkv, B, S, H, D);
      return attn_fwd(p.q, p.k, p.v, scale, true, false).o.view({B * S, H * D});
    });
    return THPVariable_Wrap(o);
  });
}

// block(x, residual or None, norm1, qkv, out, norm2, up, down, cos, sin, positions or None, B, S, H, D, eps, scale, tile_n, least) -> (y, residual): a
// decoder layer (RMS norms, packed projection, rotation, causal attention, gated MLP) where no gradient is recorded, as one call.  Layer by
// layer from Python 12 of them cost 62 us each, as long as their kernels at 777 tokens of width 768.
PyObject* py_block(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return call(a, n, 19, [&](Args& args) -> PyObject* {
    const Tensor x = args.tensor(0), residual = args.optional(1), n1 = args.tensor(2), qkv = args.tensor(3), out = args.tensor(4), n2 = args.tensor(5), up = args.tensor(6),
                 down = args.tensor(7), cos = args.tensor(8), sin = args.tensor(9), positions = args.optional(10);
    const int64_t B = args.integer(11), S = args.integer(12), H = args.integer(13), D = args.integer(14);
    const double eps = args.number(15), scale = args.number(16);
    const int tile_n = static_cast<int>(args.integer(17)), least = static_cast<int>(args.integer(18));
    if (!args.ok || at::GradMode::is_enabled() || !quiet() || !ready(lib.llmctl_rmsnorm_fwd) || !ready(lib.llmctl_gemm_bf16) || !ready(lib.llmctl_rope_inplace) ||
        !ready(lib.llmctl_flash_attn_fwd) || !ready(lib.llmctl_gemm_swiglu_bf16))
      return none();
    if (!bf16(x) || x.dim() != 2 || !x.is_contiguous() || !unit16(x) || B < 1 || S < 1 || H < 1 || (D != 64 && D != 128) || x.size(0) != B * S || x.size(0) <= least) return none();
    const int64_t T = x.size(0), W = x.size(1), F = down.dim() == 2 ? down.size(1) : 0;
    auto weight = [&](const Tensor& w, int64_t rows, int64_t cols) { return is_matrix(w) && w.size(0) == rows && w.size(1) == cols && rows % 8 == 0; };
    auto norm = [&](const Tensor& w) { return bf16(w) && w.dim() == 1 && w.size(0) == W && w.is_contiguous() && unit16(w); };
    if (F < 8 || F % 8 || W % 8 || !norm(n1) || !norm(n2) || !weight(qkv, 3 * H * D, W) || !weight(out, W, H * D) || !weight(up, 2 * F, W) || !weight(down, W, F)) return none();
    if (residual.defined() && (!bf16(residual) || !residual.is_contiguous() || residual.sizes() != x.sizes() || !unit16(residual))) return none();
    if (cos.scalar_type() != at::kFloat || sin.scalar_type() != at::kFloat || !cos.is_contiguous() || !sin.is_contiguous()) return none();
    if (positions.defined() && (positions.scalar_type() != at::kInt || !positions.is_contiguous() || positions.numel() != T)) return none();
    Tensor y, r;
    without_gil([&] {
      auto linear = [&](const Tensor& in, const Tensor& w) {
        Tensor to = new_bf16(in, {T, w.size(0)});
        gemm(in, w, to, false, false, false, tile_n, 0);
        return to;
      };
      // what the layer's operators would have given back by then is given back: a projection is three rows wide
      NormOut first = norm_fwd(x, residual, n1, eps, false);
      Tensor o = [&] {
        Tensor p;
        if (D == 64 && lib.llmctl_gemm_rope_bf16 && unit16(cos) && unit16(sin)) {
          p = new_bf16(x, {T, 3 * H * D});
          done("llmctl_gemm_rope_bf16",
               lib.llmctl_gemm_rope_bf16(cdata(first.y), cdata(qkv), data(p), static_cast<int>(T), static_cast<int>(3 * H * D), static_cast<int>(W), W, qkv.stride(0), 3 * H * D,
                                         static_cast<const float*>(cdata(cos)), static_cast<const float*>(cdata(sin)),
                                         positions.defined() ? static_cast<const int*>(cdata(positions)) : nullptr, static_cast<int>(S), static_cast<int>(2 * H * D), stream()));
        } else {
          p = linear(first.y, qkv);
          rope(p, cos, sin, positions, S, 2 * H, D, 1.f);
        }
        first.y.reset();
        const Packed z = unpack(p, B, S, H, D);
        return attn_fwd(z.q, z.k, z.v, scale, true, false).o.view({T, H * D});
      }();
      Tensor a = linear(o, out);
      o.reset();
      const NormOut second = norm_fwd(a, first.h, n2, eps, false);
      a.reset();
      first.h.reset();
      y = linear(up_and_activate(second.y, up, false).first, down);
      r = second.h;
    });
    return pair(y, THPVariable_Wrap(r));
  });
}

// ---------------------------------------------------------------------------------------------------------------------------------
// paged cache
// ---------------------------------------------------------------------------------------------------------------------------------
// a cache of whole rows of heads x head_dim
bool is_cache(const Tensor& t, int64_t row) { return bf16(t) && t.is_contiguous() && unit16(t) && t.numel() % row == 0; }

// kv_append(qkv, k_cache, v_cache, slots, heads, head_dim) -> True
PyObject* py_kv_append(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return call(a, n, 6, [&](Args& args) -> PyObject* {
    const Tensor qkv = args.tensor(0), k = args.tensor(1), v = args.tensor(2), slots = args.tensor(3);
    const int64_t H = args.integer(4), D = args.integer(5), hd = H * D;
    if (!args.ok || !quiet() || !ready(lib.llmctl_kv_append) || H < 1 || D < 1 || hd % 8 || !is_matrix(qkv) || qkv.size(1) < 3 * hd || !is_cache(k, hd) || !is_cache(v, hd) ||
        slots.scalar_type() != at::kLong || !slots.is_contiguous() || slots.numel() < qkv.size(0))
      return none();
    without_gil([&] {
      done("llmctl_kv_append", lib.llmctl_kv_append(cdata(qkv), qkv.stride(0), static_cast<int>(hd), static_cast<int>(2 * hd), data(k), data(v),
                                                    static_cast<const long long*>(cdata(slots)), static_cast<int>(qkv.size(0)), static_cast<int>(H), static_cast<int>(D), stream()));
    });
    Py_RETURN_TRUE;
  });
}

// paged_decode(q, k_cache, v_cache, tables, lens, max_context, splits, scale) -> out
PyObject* py_paged_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return call(a, n, 8, [&](Args& args) -> PyObject* {
    const Tensor q = args.tensor(0), k = args.tensor(1), v = args.tensor(2), tables = args.tensor(3), lens = args.tensor(4);
    const int context = static_cast<int>(args.integer(5)), splits = static_cast<int>(args.integer(6));
    const double scale = args.number(7);
    if (!args.ok || !quiet() || !ready(lib.llmctl_paged_attn_decode) || !lib.llmctl_paged_attn_scratch_elems || !bf16(q) || q.dim() != 3 || q.numel() == 0 || q.stride(2) != 1 ||
        q.stride(1) != q.size(2) || !unit16(q))
      return none();
    const int64_t row = q.size(1) * q.size(2);
    if (k.dim() != 4 || k.size(2) != q.size(1) || k.size(3) != q.size(2) || v.sizes() != k.sizes() || !is_cache(k, row) || !is_cache(v, row)) return none();
    if (tables.dim() != 2 || tables.scalar_type() != at::kInt || !tables.is_contiguous() || tables.size(0) < q.size(0) || lens.scalar_type() != at::kInt || !lens.is_contiguous() ||
        lens.numel() < q.size(0))
      return none();
    Tensor o = without_gil([&] {
      const int B = static_cast<int>(q.size(0)), H = static_cast<int>(q.size(1)), D = static_cast<int>(q.size(2));
      const long long need = lib.llmctl_paged_attn_scratch_elems(B, H, D, splits);
      Tensor scratch = need ? new_f32(q, {need}) : Tensor(), out = new_bf16(q, q.sizes());
      done("llmctl_paged_attn_decode", lib.llmctl_paged_attn_decode(cdata(q), q.stride(0), cdata(k), cdata(v), static_cast<const int*>(cdata(tables)), static_cast<int>(tables.size(1)),
                                                                    static_cast<const int*>(cdata(lens)), data(out), out.stride(0), need ? static_cast<float*>(data(scratch)) : nullptr, B, H, D,
                                                                    static_cast<int>(k.size(1)), context, splits, static_cast<float>(scale), stream()), need ? 2 : 1);
      return out;
    });
    return THPVariable_Wrap(o);
  });
}

// ---------------------------------------------------------------------------------------------------------------------------------
// latent attention
// ---------------------------------------------------------------------------------------------------------------------------------
bool is_indices(const Tensor& t, at::ScalarType type, int64_t least) { return t.scalar_type() == type && t.is_contiguous() && t.numel() >= least; }

// latent_kv_write(d, Q, R, dr, wq or None, wkv or None, cache or None, slots, positions, freq, mult, eps) -> the normed query latent, or True without one
PyObject* py_latent_kv_write(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return call(a, n, 12, [&](Args& args) -> PyObject* {
    const Tensor d = args.tensor(0), wq = args.optional(4), wkv = args.optional(5), cache = args.optional(6), slots = args.tensor(7), positions = args.tensor(8),
                 freq = args.tensor(9);
    const int64_t Q = args.integer(1), R = args.integer(2), dr = args.integer(3);
    const double mult = args.number(10), eps = args.number(11);
    if (!args.ok || !quiet() || !ready(lib.llmctl_latent_kv_write) || !bf16(d) || d.dim() != 2 || d.numel() == 0 || d.stride(1) != 1 || Q < 0 || R < 0 || dr < 0 || Q + R < 1 ||
        d.size(1) < Q + R + dr || recorded({&d}))
      return none();
    auto norm = [&](const Tensor& w, int64_t size) { return size == 0 || (w.defined() && bf16(w) && w.dim() == 1 && w.size(0) == size && w.is_contiguous()); };
    if (!norm(wq, Q) || !norm(wkv, R) || (R > 0 && (!cache.defined() || !bf16(cache) || !cache.is_contiguous() || cache.dim() != 3 || cache.size(2) != R + dr)) ||
        !is_indices(slots, at::kLong, d.size(0)) || !is_indices(positions, at::kInt, d.size(0)) || !is_indices(freq, at::kFloat, dr / 2))
      return none();
    auto at = [](const Tensor& t) { return t.defined() ? cdata(t) : nullptr; };
    Tensor cq;
    without_gil([&] {
      if (Q > 0) cq = new_bf16(d, {d.size(0), Q});
      done("llmctl_latent_kv_write", lib.llmctl_latent_kv_write(cdata(d), d.stride(0), static_cast<int>(Q), static_cast<int>(R), static_cast<int>(dr), at(wq), at(wkv),
                                                                Q > 0 ? data(cq) : nullptr, R > 0 ? data(cache) : nullptr, static_cast<const long long*>(cdata(slots)),
                                                                static_cast<const int*>(cdata(positions)), static_cast<const float*>(cdata(freq)), static_cast<float>(mult),
                                                                static_cast<float>(eps), static_cast<int>(d.size(0)), 0, stream()));
    });
    if (Q == 0) Py_RETURN_TRUE;
    return THPVariable_Wrap(cq);
  });
}

// latent_decode(q, dn, w_uk, w_uv, cache, tables, tiles, positions, freq, mult, scale, heads_per_tile, splits, keys_per_split, sinks or None, window,
// gate or None) -> [T, heads * dv]: absorbed queries, attention over the cache, values, for tokens whose kernel is llmctl_latent_decode
PyObject* py_latent_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return call(a, n, 17, [&](Args& args) -> PyObject* {
    const Tensor q = args.tensor(0), uk = args.tensor(2), uv = args.tensor(3), cache = args.tensor(4), tables = args.tensor(5), tiles = args.tensor(6),
                 positions = args.tensor(7), freq = args.tensor(8), sinks = args.optional(14), gate = args.optional(16);
    const int64_t dn = args.integer(1), splits = args.integer(12), per = args.integer(13);
    const double mult = args.number(9), scale = args.number(10);
    const int hpt = static_cast<int>(args.integer(11)), window = static_cast<int>(args.integer(15));
    if (!args.ok || !quiet() || !ready(lib.llmctl_latent_decode) || !bf16(q) || q.dim() != 2 || q.numel() == 0 || q.stride(1) != 1 || !bf16(uk) || !bf16(uv) || uk.dim() != 3 ||
        uv.dim() != 3 || recorded({&q, &uk, &uv}) || at::autocast::is_autocast_enabled(at::kCUDA) || !bf16(cache) || cache.dim() != 3 || !cache.is_contiguous() || !unit16(cache))
      return none();
    const int64_t T = q.size(0), H = uk.size(0), R = uk.size(2), D = cache.size(2), dr = D - R, dv = uv.size(1);
    if (dr < 0 || uk.size(1) != dn || q.size(1) < H * (dn + dr) || uv.size(0) != H || uv.size(2) != R || hpt < 1 || hpt > 32 || splits < 1 || tables.dim() != 2 ||
        !is_indices(tables, at::kInt, 1) || !is_indices(tiles, at::kInt, 4) || !is_indices(positions, at::kInt, T) || !is_indices(freq, at::kFloat, dr / 2))
      return none();
    if (sinks.defined() && !is_indices(sinks, at::kFloat, H)) return none();
    if (gate.defined() && (!bf16(gate) || gate.dim() != 2 || gate.size(0) != T || gate.size(1) != H || gate.stride(1) != 1)) return none();
    Tensor o = without_gil([&] {
      at::AutoDispatchBelowADInplaceOrView below;
      const Tensor ql = at::bmm(q.as_strided({H, T, dn}, {dn + dr, q.stride(0), 1}), uk);            // [H, T, R]
      Tensor ol = new_bf16(q, {T, H, R}), out = new_bf16(q, {T, H * dv});
      Tensor partial = splits > 1 ? new_f32(q, {T * H * splits * (R + 2)}) : Tensor();
      done("llmctl_latent_decode",
           lib.llmctl_latent_decode(cdata(ql), ql.stride(1), ql.stride(0), cdata(q), q.stride(0), static_cast<int>(dn), cdata(cache), cache.size(0) * cache.size(1),
                                    static_cast<const int*>(cdata(tables)), static_cast<int>(tables.size(1)), static_cast<int>(cache.size(1)), static_cast<const int*>(cdata(tiles)),
                                    static_cast<int>(tiles.size(0)), static_cast<int>(T), static_cast<const int*>(cdata(positions)), static_cast<const float*>(cdata(freq)),
                                    static_cast<float>(mult), static_cast<float>(scale), static_cast<int>(H), static_cast<int>(R), static_cast<int>(dr), hpt, static_cast<int>(splits),
                                    static_cast<int>(per), data(ol), splits > 1 ? static_cast<float*>(data(partial)) : nullptr,
                                    sinks.defined() ? static_cast<const float*>(cdata(sinks)) : nullptr, window, gate.defined() ? cdata(gate) : nullptr,
                                    gate.defined() ? gate.stride(0) : 0, stream()), splits > 1 ? 2 : 1);
      Tensor by_head = out.as_strided({H, T, dv}, {dv, H * dv, 1});                                   // the product lands head by head in place
      at::bmm_out(by_head, ol.transpose(0, 1), uv.transpose(1, 2));
      return out;
    });
    return THPVariable_Wrap(o);
  });
}

// ---------------------------------------------------------------------------------------------------------------------------------
// the module
// ---------------------------------------------------------------------------------------------------------------------------------
// bind(path of the loaded kernel library, NativeError, check_waits, gradient of a weight with a buffer for it)
PyObject* py_bind(PyObject*, PyObject* args) {
  const char* path;
  PyObject *error, *waits, *wgrad;
  if (!PyArg_ParseTuple(args, "sOOO", &path, &error, &waits, &wgrad)) return nullptr;
  void* so = dlopen(path, RTLD_NOW | RTLD_NOLOAD);
  if (so == nullptr) {
    PyErr_Format(PyExc_RuntimeError, "%s is not loaded", path);
    return nullptr;
  }
#define X(name) lib.name = reinterpret_cast<decltype(lib.name)>(dlsym(so, #name));
  LLMCTL_ENTRIES(X)
#undef X
  lib.wait_word = reinterpret_cast<void* (*)()>(dlsym(so, "llmctl_wait_status_word"));
  Py_INCREF(error);
  Py_INCREF(waits);
  Py_INCREF(wgrad);
  native_error = error;
  check_waits = waits;
  buffered_wgrad = wgrad;
  Py_RETURN_NONE;
}
PyObject* py_launches(PyObject*, PyObject*) { return PyLong_FromLongLong(launches.load(std::memory_order_relaxed)); }

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&py_##name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {{"bind", py_bind, METH_VARARGS, nullptr}, {"launches", py_launches, METH_NOARGS, nullptr}, FAST(rmsnorm), FAST(gemm), FAST(linear), FAST(gemm_swiglu),
                         FAST(mlp), FAST(attention), FAST(rope_attention), FAST(block), FAST(kv_append), FAST(paged_decode), FAST(latent_kv_write), FAST(latent_decode), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "llmctl_ops", "Host side of the operators (csrc/torch/ops.cpp)", -1, methods};

}  // namespace

// Under another PyTorch or Python than it was built for it might misread every tensor: it refuses to be imported there.
PyMODINIT_FUNC PyInit_llmctl_ops() {
  PyObject* torch = PyImport_ImportModule("torch");
  PyObject* version = torch == nullptr ? nullptr : PyObject_GetAttrString(torch, "__version__");
  Py_XDECREF(torch);
  if (version == nullptr) return nullptr;
  int major = 0, minor = 0;
  sscanf(Py_GetVersion(), "%d.%d", &major, &minor);
  const bool same = PyUnicode_Check(version) && PyUnicode_CompareWithASCIIString(version, LLMCTL_TORCH_VERSION) == 0 && major == PY_MAJOR_VERSION &&
                    minor == PY_MINOR_VERSION;
  if (!same) PyErr_Format(PyExc_ImportError, "built for PyTorch %s and Python %d.%d, this is PyTorch %S and Python %d.%d", LLMCTL_TORCH_VERSION, PY_MAJOR_VERSION,
                          PY_MINOR_VERSION, version, major, minor);
  Py_DECREF(version);
  return same ? PyModule_Create(&module) : nullptr;
}
