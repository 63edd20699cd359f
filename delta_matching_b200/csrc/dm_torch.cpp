// The eager route of dm_attn_func / dm_attn_func_bhnd in C++: contract checks, allocation, the two whole-pass calls of the C
// ABI (dm_attn_fwd, dm_attn_bwd) and the autograd node between them.  The reference has an op library of this kind under
// its Python autograd function (csrc/delta_matching_api.cpp:105-391, 683-715; delta_matching/attn.py:37-118).
//
// Why it exists: the kernels of a short sequence take about 50 us in all, and the Python route around them (a Python
// autograd.Function, three transposes with their graph nodes, five ctypes calls of 15 - 27 arguments, some twenty torch.empty)
// took 430 us of host time per forward + backward.  Here a pass is one C call with its tensors carved out of few
// allocations: the codes, scales and LSE that the backward needs share one buffer, as do the temporaries of each pass.
//
// The module does not link against the kernel library: bind() receives the addresses of the entry points from the
// ctypes handle, so that DM_SO decides for both which library runs.  attn() returns None whenever a call is not one it
// serves as it stands (a violated constraint, a tensor subclass, a functorch or dispatch-mode wrapper, a trace); the caller then
// takes the Python route, which raises the contract's exceptions or serves the call.
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/dynamo/compiled_autograd.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/utils/pybind.h>
#include <ATen/core/PythonFallbackKernel.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <atomic>
#include <cmath>
#include <cstdlib>
#include <mutex>

#include "../../include/dm_b200.h"

namespace {

using at::Tensor;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

struct Lib {
  decltype(&dm_attn_fwd) fwd = nullptr;
  decltype(&dm_attn_bwd) bwd = nullptr;
  decltype(&dm_last_error) last_error = nullptr;
  decltype(&dm_attn_bwd_workspace_bytes) bwd_workspace_bytes = nullptr;
  decltype(&dm_quant_qkv_workspace_bytes) quant_workspace_bytes = nullptr;
} g_lib;

constexpr int kMaxDevices = 64;
std::atomic<int*> g_status[kMaxDevices] = {};  // pinned status words (ops.status_word), one per device that has been used
PyObject* g_status_word = nullptr;        // ops: device index -> address of its status word
PyObject* g_raise_if_set = nullptr;       // ops._raise_if_set
PyObject* g_split_bwd = nullptr;          // ops.bwd_fp8: the backward under a workspace bound
int64_t g_small_ws = 0, g_max_tiles = 0;  // ops._SMALL_WS, ops._MAX_WS_TILES

void check(int rc) {
  if (rc == 0) return;
  char buf[1024] = "";
  g_lib.last_error(buf, sizeof(buf));
  throw std::runtime_error(buf[0] ? buf : "delta_matching_b200: library call failed");
}

enum Flags : int64_t { kCausal = 1, kMatched = 2, kDs32 = 4, kNorm = 8, kHeadMajor = 16 };

struct Shape {
  int B, N, H, Hk, D;
  int64_t rows_q() const { return static_cast<int64_t>(B) * H * N; }
  int64_t rows_k() const { return static_cast<int64_t>(B) * Hk * N; }
};

// Element strides of a (B, N, H, D) or (B, H, N, D) tensor as (batch, head, token).
struct Strides {
  int64_t b, h, n;
  Strides(const Tensor& t, bool head_major)
      : b(t.stride(0)), h(t.stride(head_major ? 1 : 2)), n(t.stride(head_major ? 2 : 1)) {}
};

// The kernels read rows of head_dim elements at 16-byte aligned addresses; anything else is copied (ops._rows).
Tensor rows(const Tensor& t) {
  if (t.stride(3) != 1 || t.stride(0) % 8 || t.stride(1) % 8 || t.stride(2) % 8 ||
      reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16)
    return t.contiguous();
  return t;
}

// A saved tensor as the kernels read it, in order and aligned.  Unpack hooks may hand over anything (torch checks what hooks make
// of a gradient, but not this): another layout is copied, another type, shape or device is refused.
Tensor unpacked(const Tensor& t, const char* name, at::ScalarType type, at::IntArrayRef sizes, const at::Device& dev) {
  TORCH_CHECK(t.defined() && t.layout() == at::kStrided && t.scalar_type() == type && t.sizes() == sizes && t.device() == dev,
              "delta_matching: ", name, " must come back from saved-tensor hooks as a ", type, " tensor of shape ", sizes, " on ", dev);
  const bool in_place = t.is_contiguous() && reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0;
  return in_place ? t : t.clone(at::MemoryFormat::Contiguous);
}

// Sub-buffers of one allocation, each 256-byte aligned.
class Carve {
 public:
  int64_t take(int64_t bytes) {
    const int64_t at = size_;
    size_ += (bytes + 255) & ~int64_t(255);
    return at;
  }
  int64_t size() const { return size_; }

 private:
  int64_t size_ = 0;
};

Tensor bytes_on(int64_t n, const at::Device& dev) {
  return Tensor(at::detail::empty_cuda({n}, at::kByte, dev, std::nullopt));
}
Tensor bf16_on(at::IntArrayRef size, const at::Device& dev) {
  return Tensor(at::detail::empty_cuda(size, at::kBFloat16, dev, std::nullopt));
}

// What the backward reads: codes and scales of q, k, v and the LSE; and the scratch of the K mean, which is small (a sixteenth
// of K's codes) and not worth an allocation of its own.
struct Saved {
  Carve c;
  int64_t q8, k8, v8, qs, ks, vs, lse, mean, part;
  explicit Saved(const Shape& s) {
    q8 = c.take(s.rows_q() * s.D);
    k8 = c.take(s.rows_k() * s.D);
    v8 = c.take(s.rows_k() * s.D);
    qs = c.take(s.rows_q() / 8);
    ks = c.take(s.rows_k() / 8);
    vs = c.take(s.rows_k() / 8);
    lse = c.take(s.rows_q() * 4);
    mean = c.take(static_cast<int64_t>(s.B) * s.Hk * s.D * 4);
    part = c.take(static_cast<int64_t>(g_lib.quant_workspace_bytes(s.B, s.N, s.Hk, s.D)));
  }
};

// The word is read without a synchronisation, as every op does (ops._enter); a kernel that gave up makes this call raise.
int* status_of(int dev) {
  int* w = g_status[dev].load(std::memory_order_acquire);
  if (w == nullptr) {
    pybind11::gil_scoped_acquire gil;
    pybind11::object addr = pybind11::reinterpret_borrow<pybind11::object>(g_status_word)(dev);
    w = reinterpret_cast<int*>(addr.cast<uintptr_t>());
    g_status[dev].store(w, std::memory_order_release);
  }
  if (*static_cast<volatile int*>(w) != 0) {
    std::string msg;
    {
      pybind11::gil_scoped_acquire gil;
      try {
        pybind11::reinterpret_borrow<pybind11::object>(g_raise_if_set)(dev);
      } catch (pybind11::error_already_set& e) {
        msg = pybind11::str(e.value()).cast<std::string>();
      }
    }
    if (!msg.empty()) throw std::runtime_error(msg);
  }
  return w;
}

// Producers and forward; `saved` is filled and kept by the caller.
Tensor run_forward(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const Shape& s, int64_t flags, Tensor* saved_out) {
  const at::Device dev = q_in.device();
  const c10::cuda::CUDAGuard guard(dev);
  int* status = status_of(dev.index());
  const Tensor q = rows(q_in), k = rows(k_in), v = rows(v_in);
  const bool hm = (flags & kHeadMajor) != 0;
  const Strides sq(q, hm), sk(k, hm), sv(v, hm);
  const Saved L(s);
  Tensor saved = bytes_on(L.c.size(), dev);
  uint8_t* p = static_cast<uint8_t*>(saved.mutable_data_ptr());
  Tensor o = bf16_on({s.B, s.N, s.H, s.D}, dev);
  check(g_lib.fwd(q.const_data_ptr(), sq.b, sq.h, sq.n, k.const_data_ptr(), sk.b, sk.h, sk.n, v.const_data_ptr(), sv.b, sv.h, sv.n,
                  s.B, s.N, s.H, s.Hk, s.D, (flags & kCausal) ? 1 : 0, p + L.q8, p + L.k8, p + L.v8,
                  reinterpret_cast<float*>(p + L.qs), reinterpret_cast<float*>(p + L.ks), reinterpret_cast<float*>(p + L.vs),
                  reinterpret_cast<float*>(p + L.mean), p + L.part, o.mutable_data_ptr(), reinterpret_cast<float*>(p + L.lse), status,
                  c10::cuda::getCurrentCUDAStream(dev.index()).stream()));
  if (saved_out) *saved_out = std::move(saved);
  return o;
}

// dQ, dK, dV token-major.  `o`: the forward's output (stale delta), undefined for the matched delta.
variable_list run_backward(const Tensor& d_o_in, const Tensor& saved_in, const Tensor& o_in, const Shape& s, int64_t flags, const at::Device& dev) {
  const c10::cuda::CUDAGuard guard(dev);
  int* status = status_of(dev.index());
  const Saved L(s);
  const Tensor d_o = rows(d_o_in), saved = unpacked(saved_in, "the saved codes", at::kByte, {L.c.size()}, dev);
  const Tensor o = o_in.defined() ? unpacked(o_in, "the saved O", at::kBFloat16, {s.B, s.N, s.H, s.D}, dev) : o_in;
  const Strides sd(d_o, false);
  uint8_t* p = static_cast<uint8_t*>(saved.mutable_data_ptr());      // only read
  // The dS workspace of the whole call, as long as no bound is set and it is no larger than what ops takes without asking the
  // device how much memory is free; otherwise ops.bwd_fp8 plans the ranges.
  const int64_t ws_bytes = g_lib.bwd_workspace_bytes(s.B, s.N, s.H, s.Hk, s.D, (flags & kCausal) ? 1 : 0);
  const int64_t n_t = s.N / 128;
  const bool whole = ws_bytes <= g_small_ws && n_t * n_t * s.H * s.B <= g_max_tiles && std::getenv("DM_BWD_WORKSPACE_MB") == nullptr &&
                     std::getenv("DM_BWD_WS_LIMIT_GB") == nullptr;
  Carve c;
  const int64_t do8 = c.take(s.rows_q() * s.D), dos = c.take(s.rows_q() / 8), delta = c.take(s.rows_q() * 4);
  const int64_t ws = whole ? c.take(ws_bytes) : 0;
  Tensor tmp = bytes_on(c.size(), dev);
  uint8_t* t = static_cast<uint8_t*>(tmp.mutable_data_ptr());
  Tensor dq, dk, dv;
  if (whole) {
    dq = bf16_on({s.B, s.N, s.H, s.D}, dev);
    dk = bf16_on({s.B, s.N, s.Hk, s.D}, dev);
    dv = bf16_on({s.B, s.N, s.Hk, s.D}, dev);
  }
  const int call_flags = ((flags & kDs32) ? DM_DS_BLOCK32 : 0) | ((flags & kNorm) ? 0 : DM_ATTN_DELTA_SUM) | (whole ? 0 : DM_ATTN_DELTA_ONLY);
  check(g_lib.bwd(d_o.const_data_ptr(), sd.b, sd.h, sd.n, o.defined() ? o.const_data_ptr() : nullptr, p + L.q8, p + L.k8, p + L.v8,
                  reinterpret_cast<float*>(p + L.qs), reinterpret_cast<float*>(p + L.ks), reinterpret_cast<float*>(p + L.vs),
                  reinterpret_cast<float*>(p + L.lse), t + do8, reinterpret_cast<float*>(t + dos), reinterpret_cast<float*>(t + delta),
                  s.B, s.N, s.H, s.Hk, s.D, (flags & kCausal) ? 1 : 0, whole ? dq.mutable_data_ptr() : nullptr,
                  whole ? dk.mutable_data_ptr() : nullptr, whole ? dv.mutable_data_ptr() : nullptr, whole ? t + ws : nullptr, ws_bytes,
                  call_flags, status, c10::cuda::getCurrentCUDAStream(dev.index()).stream()));
  if (!whole) {
    auto codes = [&](const Tensor& from, int64_t at, int h) {
      return from.narrow(0, at, static_cast<int64_t>(s.B) * h * s.N * s.D).view(at::kFloat8_e4m3fn).view({s.B, h, s.N, s.D});
    };
    auto floats = [&](const Tensor& from, int64_t at, int h, int64_t n) {
      return from.narrow(0, at, static_cast<int64_t>(s.B) * h * n * 4).view(at::kFloat).view({s.B, h, n});
    };
    const at::AutoDispatchBelowADInplaceOrView below;
    pybind11::gil_scoped_acquire gil;
    pybind11::object f = pybind11::reinterpret_borrow<pybind11::object>(g_split_bwd);
    pybind11::tuple r = f(codes(saved, L.q8, s.H), codes(saved, L.k8, s.Hk), codes(saved, L.v8, s.Hk), codes(tmp, do8, s.H),
                          floats(saved, L.qs, s.H, s.N / 32), floats(saved, L.ks, s.Hk, s.N / 32), floats(saved, L.vs, s.Hk, s.N / 32),
                          floats(tmp, dos, s.H, s.N / 32), floats(saved, L.lse, s.H, s.N), floats(tmp, delta, s.H, s.N),
                          (flags & kCausal) != 0, (flags & kDs32) != 0);
    dq = r[0].cast<Tensor>();
    dk = r[1].cast<Tensor>();
    dv = r[2].cast<Tensor>();
  }
  return {dq, dk, dv};
}

Shape shape_of(const Tensor& q, const Tensor& k, int64_t flags) {
  const bool hm = (flags & kHeadMajor) != 0;
  return {static_cast<int>(q.size(0)), static_cast<int>(q.size(hm ? 2 : 1)), static_cast<int>(q.size(hm ? 1 : 2)),
          static_cast<int>(k.size(hm ? 1 : 2)), static_cast<int>(q.size(3))};
}

// dQ, dK, dV in the layout of the inputs; an undefined dO is a zero one.
variable_list gradients(const Tensor& grad, const Tensor& saved, const Tensor& o, const Shape& s, int64_t flags, const at::Device& dev) {
  const at::AutoGradMode no_grad(false);
  const Tensor d_o = grad.defined() ? grad : at::zeros({s.B, s.N, s.H, s.D}, at::TensorOptions(dev).dtype(at::kBFloat16));
  variable_list g = run_backward(d_o, saved, o, s, flags, dev);
  if (flags & kHeadMajor)
    for (Tensor& t : g) t = t.permute({0, 2, 1, 3});
  return g;
}

// The autograd node.  (torch::autograd::Function would do, at some 4 us more per forward + backward for its context, the map of
// saved values and the generic wrapping of inputs and outputs.)
struct AttnBackward : public torch::autograd::Node {
  SavedVariable saved, o;       // o: stale delta only, the matched delta never reads O
  Shape s;
  int64_t flags = 0;

  variable_list apply(variable_list&& grads) override {
    const std::lock_guard<std::mutex> lock(mutex_);
    const bool twice = at::GradMode::is_enabled() && grads[0].defined() && grads[0].requires_grad();
    variable_list g;
    {
      const at::AutoGradMode no_grad(false);      // for the unpack hooks
      g = gradients(grads[0], saved.unpack(), (flags & kMatched) ? Tensor() : o.unpack(shared_from_this()), s, flags, input_metadata(0).device());
    }
    if (twice) {      // what torch.autograd.function.once_differentiable does: a second derivative raises when it is taken
      for (Tensor& t : g) t = t.detach().requires_grad_();
      g = torch::autograd::DelayedError("trying to differentiate twice a function that was marked with @once_differentiable", 3)
              .apply(std::move(g));
    }
    return g;
  }
  // Compiled autograd: what the pass depends on, and the pass as a function of it that the recorded graph calls (opaque: the
  // kernels take addresses, there is nothing to trace through).
  void compiled_args(torch::dynamo::autograd::CompiledNodeArgs& args) const override {
    args.collect(saved, false);
    args.collect(o, true);
    for (const int64_t x : {int64_t(s.B), int64_t(s.N), int64_t(s.H), int64_t(s.Hk), int64_t(s.D), flags}) args.collect(x);
  }
  variable_list apply_with_saved(const variable_list& grads, torch::dynamo::autograd::SwapSavedVariables& swap) override {
    using torch::dynamo::autograd::IValuePacker;
    swap.before(saved);
    swap.before(o);
    torch::dynamo::autograd::PackedArgs packed;
    std::vector<at::TypePtr> schema;
    auto pack = [&](const auto& x) {
      packed.pack(x);
      schema.push_back(IValuePacker<std::decay_t<decltype(x)>>::packed_type());
    };
    for (const int64_t x : {flags, int64_t(s.B), int64_t(s.N), int64_t(s.H), int64_t(s.Hk), int64_t(s.D)}) pack(x);
    pack(saved.unpack());
    if (!(flags & kMatched)) pack(o.unpack(shared_from_this()));
    const auto& compiler = torch::dynamo::autograd::getPyCompilerInterface();
    const std::string fn = compiler->bind_function(swap.get_py_compiler(), name(), &AttnBackward::apply_recorded, std::move(schema),
                                                   /*is_custom_function=*/true, /*is_traceable=*/false);
    variable_list g = compiler->call_function(
        swap.get_py_compiler(), "apply_functional", fn, grads, packed.vec(),
        IValuePacker<std::vector<std::optional<torch::autograd::InputMetadata>>>::pack(torch::dynamo::autograd::get_input_metadata(next_edges())));
    swap.after(saved);
    swap.after(o);
    return g;
  }
  static variable_list apply_recorded(const variable_list& grads, const std::vector<c10::IValue>& args) {
    torch::dynamo::autograd::PackedArgs packed(args);
    auto i = [&] { return static_cast<int>(packed.unpack<int64_t>()); };
    const int64_t flags = packed.unpack<int64_t>();
    Shape s;
    s.B = i(); s.N = i(); s.H = i(); s.Hk = i(); s.D = i();
    const Tensor buffer = packed.unpack<Tensor>();
    return gradients(grads[0], buffer, (flags & kMatched) ? Tensor() : packed.unpack<Tensor>(), s, flags, buffer.device());
  }
  void release_variables() override {
    const std::lock_guard<std::mutex> lock(mutex_);
    saved.reset_data();
    o.reset_data();
  }
  std::string name() const override { return "DeltaMatchingAttnBackward"; }
};

Tensor with_graph(const Tensor& q, const Tensor& k, const Tensor& v, int64_t flags) {
  const Shape s = shape_of(q, k, flags);
  Tensor buffer, o;
  {
    const at::AutoDispatchBelowADInplaceOrView below;
    o = run_forward(q, k, v, s, flags, &buffer);
  }
  std::shared_ptr<AttnBackward> node(new AttnBackward(), torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(q, k, v));
  node->s = s;
  node->flags = flags;
  torch::autograd::set_history(o, node);
  node->saved = SavedVariable(buffer, false);
  if (!(flags & kMatched)) node->o = SavedVariable(o, true);
  return o;
}

// (ds32, norm) of a numerics arm, or -1 for a name that is none at this head_dim (ops.NUMERICS, attn._numerics).
int64_t numerics_flags(PyObject* name, int64_t D) {
  if (!PyUnicode_Check(name)) return -1;
  auto is = [&](const char* s) { return PyUnicode_CompareWithASCIIString(name, s) == 0; };
  if (is("sm100-mx") || (D == 256 && is("sm100-mx-d256"))) return kNorm;
  if (is("sm100-mx-ds32") || (D == 256 && is("sm100-mx-d256-ds32"))) return kNorm | kDs32;
  if (is("sm100-mx-nonorm")) return 0;
  return -1;
}

bool plain_cuda_bf16(PyObject* o, const Tensor*& t) {
  if (!THPVariable_CheckExact(o)) return false;
  t = &THPVariable_Unpack(o);
  constexpr c10::DispatchKeySet kWrapped({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::Functionalize,
                                          c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Conjugate, c10::DispatchKey::Negative});
  return t->dim() == 4 && t->is_cuda() && t->scalar_type() == at::kBFloat16 && t->layout() == at::kStrided &&
         !t->unsafeGetTensorImpl()->key_set().has_any(kWrapped) && !t->_fw_grad(0).defined();
}

// attn(q, k, v, softmax_scale, causal, mode, numerics, head_major) -> o, or None for the Python route
PyObject* attn(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Tensor *qp = nullptr, *kp = nullptr, *vp = nullptr;
  if (n != 8 || !plain_cuda_bf16(args[0], qp) || !plain_cuda_bf16(args[1], kp) || !plain_cuda_bf16(args[2], vp)) Py_RETURN_NONE;
  if (c10::impl::TorchDispatchModeTLS::any_modes_set() || !PyUnicode_Check(args[5])) Py_RETURN_NONE;
  // torch.jit.trace records the Python route's autograd function; from here it would see a tensor from nowhere, a constant
  if (torch::jit::tracer::isTracing()) Py_RETURN_NONE;
  const Tensor &q = *qp, &k = *kp, &v = *vp;
  const bool hm = args[7] == Py_True;
  const int causal = PyObject_IsTrue(args[4]);
  if (causal < 0) return nullptr;
  const bool matched = PyUnicode_CompareWithASCIIString(args[5], "matched") == 0;
  if (!matched && PyUnicode_CompareWithASCIIString(args[5], "stale") != 0) Py_RETURN_NONE;
  const int64_t B = q.size(0), N = q.size(hm ? 2 : 1), H = q.size(hm ? 1 : 2), D = q.size(3), Hk = k.size(hm ? 1 : 2);
  const int64_t num = numerics_flags(args[6], D);
  const bool fine = num >= 0 && (causal || !matched) && q.device() == k.device() && q.device() == v.device() && k.sizes() == v.sizes() &&
                    k.size(0) == B && k.size(3) == D && k.size(hm ? 2 : 1) == N && Hk > 0 && H % Hk == 0 && (D == 128 || D == 256) &&
                    N > 0 && N % (D == 128 ? 256 : 128) == 0 && N < (int64_t(1) << 31) && B > 0 && H > 0 && B * H <= 65535 &&
                    q.device().index() < kMaxDevices;
  if (!fine) Py_RETURN_NONE;
  if (args[3] != Py_None) {
    const double scale = PyFloat_AsDouble(args[3]);
    if (scale == -1.0 && PyErr_Occurred()) {
      PyErr_Clear();
      Py_RETURN_NONE;
    }
    if (!(std::fabs(scale - 1.0 / std::sqrt(static_cast<double>(D))) <= 1e-12)) Py_RETURN_NONE;
  }
  if (at::cuda::getDeviceProperties(q.device().index())->major != 10) Py_RETURN_NONE;
  const int64_t flags = (causal ? kCausal : 0) | (matched ? kMatched : 0) | num | (hm ? kHeadMajor : 0);
  Tensor o;
  {
    pybind11::gil_scoped_release no_gil;
    if (at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad())) {
      o = with_graph(q, k, v, flags);
    } else {
      const at::AutoDispatchBelowADInplaceOrView below;
      o = run_forward(q, k, v, shape_of(q, k, flags), flags, nullptr);
    }
  }
  return THPVariable_Wrap(std::move(o));
  END_HANDLE_TH_ERRORS
}

// bind(fwd, bwd, last_error, bwd_workspace_bytes, quant_workspace_bytes, status_word, raise_if_set, split_bwd, small_ws, max_tiles)
PyObject* bind(PyObject*, PyObject* args) {
  unsigned long long a[5];
  PyObject *sw, *ris, *sb;
  long long small_ws, max_tiles;
  if (!PyArg_ParseTuple(args, "KKKKKOOOLL", &a[0], &a[1], &a[2], &a[3], &a[4], &sw, &ris, &sb, &small_ws, &max_tiles)) return nullptr;
  g_lib.fwd = reinterpret_cast<decltype(&dm_attn_fwd)>(a[0]);
  g_lib.bwd = reinterpret_cast<decltype(&dm_attn_bwd)>(a[1]);
  g_lib.last_error = reinterpret_cast<decltype(&dm_last_error)>(a[2]);
  g_lib.bwd_workspace_bytes = reinterpret_cast<decltype(&dm_attn_bwd_workspace_bytes)>(a[3]);
  g_lib.quant_workspace_bytes = reinterpret_cast<decltype(&dm_quant_qkv_workspace_bytes)>(a[4]);
  Py_INCREF(sw);
  Py_INCREF(ris);
  Py_INCREF(sb);
  g_status_word = sw;
  g_raise_if_set = ris;
  g_split_bwd = sb;
  g_small_ws = small_ws;
  g_max_tiles = max_tiles;
  Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"attn", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&attn)), METH_FASTCALL, "attention on CUDA tensors, or None"},
    {"bind", bind, METH_VARARGS, "addresses of the kernel library's entry points and the op layer's callbacks"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_dm_native", "native eager route", -1, kMethods};

}  // namespace

PyMODINIT_FUNC PyInit__dm_native(void) { return PyModule_Create(&kModule); }
