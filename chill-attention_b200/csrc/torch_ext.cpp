// Eager-mode call path of chill_attention() as native code: argument checks, output allocation, the C-ABI calls and the
// autograd node.  A Python autograd.Function around the same calls (two interpreter round trips through the autograd
// engine, five tensor allocations and ~40 struct fields set from Python) takes 17 us per forward call of (8, 4, 128, 128)
// and 138 us per training step of (1, 2, 128, 64), this file 8 and 78 us; the GPU needs 6 and 25 us of that.
//
// Nothing is cached between calls: the structs are rebuilt from the tensors each time (well under a microsecond), so the
// path is safe for any number of threads, streams and devices.
#include <ATen/Context.h>
#include <ATen/core/grad_mode.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/zeros_like.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/utils/pybind.h>

#include <atomic>
#include <memory>
#include <string>
#include <utility>
#include <vector>

#include "chill_b200.h"

namespace py = pybind11;
using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

namespace {

// One kernel library (the built-in one or a custom-mask build): its entry points, resolved by the Python loader.
struct Library {
  decltype(&chill_fwd) fwd;
  decltype(&chill_bwd_delta) delta;
  decltype(&chill_bwd) bwd;
  decltype(&chill_bwd_uses_tensor_cores) bwd_uses_tc;
  decltype(&chill_bwd_dq_accum_bytes) accum_bytes;
  decltype(&chill_status_string) status_string;
  decltype(&chill_last_cuda_error) cuda_error;
  int32_t functor_id;
};

std::atomic<bool> g_deterministic{false};
std::atomic<long long> g_bwd_tc{0}, g_bwd_generic{0};

// Raised as chill_attention._cabi.ChillLibraryError in Python: torch asks such an exception for its type wherever it crosses
// over, be it out of a call of this module or out of a backward that the autograd engine runs.
struct ChillError : torch::PyTorchError {
  using torch::PyTorchError::PyTorchError;
  PyObject* python_type() override { return py::module_::import("chill_attention._cabi").attr("ChillLibraryError").ptr(); }
};

struct Call : torch::CustomClassHolder {
  std::shared_ptr<const Library> lib;
  chill_mask_desc mask;
  double sm_scale;
  uint32_t flags;
};

void check(const Library& lib, int status, const char* what) {
  if (status == CHILL_OK) return;
  std::string msg = std::string(what) + " failed: " + lib.status_string(status) + " (status " + std::to_string(status) + ")";
  if (status == CHILL_E_CUDA) msg += std::string(" ") + lib.cuda_error();
  throw ChillError(msg);
}

// What the tensor-core kernels need of an operand: contiguous channels, no broadcast dimension, 16-byte aligned base and
// batch / head / row strides.
bool tma_compatible(const Tensor& t) {
  const int64_t es = (int64_t)t.element_size();
  if (t.stride(3) != 1 || reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 != 0) return false;
  for (int d = 0; d < 3; ++d)
    if (t.size(d) > 1 && (t.stride(d) <= 0 || (t.stride(d) * es) % 16 != 0)) return false;
  return true;
}

// 16-bit operands TMA cannot describe are packed once: the copy costs far less than the CUDA-core kernels that would
// otherwise take the call.
Tensor packed(const Tensor& t) { return t.scalar_type() == at::kFloat || tma_compatible(t) ? t : t.contiguous(); }

void set_strides(int64_t* dst, const Tensor& t) {
  for (int64_t d = 0; d < t.dim(); ++d) dst[d] = t.stride(d);
}

chill_shape make_shape(const Tensor& q, const Tensor& k, const std::optional<Tensor>& lens, const Call& c) {
  chill_shape s{};
  s.B = (int32_t)q.size(0); s.H = (int32_t)q.size(1); s.H_kv = (int32_t)k.size(1);
  s.Lq = (int32_t)q.size(2); s.Lk = (int32_t)k.size(2); s.D = (int32_t)q.size(3);
  s.dtype = q.scalar_type() == at::kFloat ? CHILL_F32 : (q.scalar_type() == at::kHalf ? CHILL_F16 : CHILL_BF16);
  s.seq_len = s.Lq;
  s.sm_scale = (float)c.sm_scale;
  s.flags = c.flags;
  s.lens = lens.has_value() ? lens->const_data_ptr<int32_t>() : nullptr;
  s.mask = c.mask;
  return s;
}

void* current_stream(const Tensor& t) { return (void*)c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

std::pair<Tensor, Tensor> forward(const Tensor& q, const Tensor& k, const Tensor& v, const std::optional<Tensor>& lens,
                                  const Call& c, bool want_lse) {
  Tensor o = at::empty(q.sizes(), q.options()), lse;
  if (want_lse) lse = at::empty(q.sizes().slice(0, 3), q.options().dtype(at::kFloat));
  chill_fwd_args a{};
  a.s = make_shape(q, k, lens, c);
  a.q = q.const_data_ptr(); a.k = k.const_data_ptr(); a.v = v.const_data_ptr(); a.o = o.mutable_data_ptr();
  set_strides(a.q_strides, q); set_strides(a.k_strides, k); set_strides(a.v_strides, v); set_strides(a.o_strides, o);
  if (want_lse) {
    a.lse = lse.mutable_data_ptr<float>();
    set_strides(a.lse_strides, lse);
  }
  const int st = c.lib->fwd(&a, current_stream(q));
  check(*c.lib, st, "chill_fwd");
  return {o, lse};
}

struct AttentionFn : torch::autograd::Function<AttentionFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q_in, const Tensor& k_in, const Tensor& v_in,
                               const std::optional<Tensor>& lens, c10::intrusive_ptr<Call> call, bool return_lse) {
    const Tensor q = packed(q_in), k = packed(k_in), v = packed(v_in);  // the backward reads the packed copies again
    auto [o, lse] = ::forward(q, k, v, lens, *call, true);
    ctx->save_for_backward({q, k, v, o, lse, lens.has_value() ? *lens : Tensor()});
    ctx->saved_data["call"] = c10::IValue::make_capsule(std::move(call));
    ctx->set_materialize_grads(false);
    if (!return_lse) ctx->mark_non_differentiable({lse});
    return {o, lse};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &q = saved[0], &k = saved[1], &v = saved[2], &o = saved[3], &lse = saved[4];
    const std::optional<Tensor> lens = saved[5].defined() ? std::optional<Tensor>(saved[5]) : std::nullopt;
    const auto holder = ctx->saved_data["call"].toCapsule();
    const Call& c = *static_cast<const Call*>(holder.get());
    c10::cuda::CUDAGuard guard(q.device());
    Tensor d_o = grads[0].defined() ? grads[0] : at::zeros_like(o);
    // Autograd often hands over an expanded tensor (all strides 0 after o.sum().backward()) or a transposed view
    if (!tma_compatible(d_o)) d_o = d_o.contiguous();
    Tensor d_lse = grads[1].defined() ? grads[1].to(at::kFloat) : Tensor();  // gradient through a returned LSE
    Tensor dq = at::empty(q.sizes(), q.options()), dk = at::empty(k.sizes(), k.options()), dv = at::empty(v.sizes(), v.options());
    chill_bwd_args a{};
    a.s = make_shape(q, k, lens, c);
    a.q = q.const_data_ptr(); a.k = k.const_data_ptr(); a.v = v.const_data_ptr(); a.o = o.const_data_ptr();
    a.d_o = d_o.const_data_ptr();
    a.lse = lse.const_data_ptr<float>();
    a.dq = dq.mutable_data_ptr(); a.dk = dk.mutable_data_ptr(); a.dv = dv.mutable_data_ptr();
    set_strides(a.q_strides, q); set_strides(a.k_strides, k); set_strides(a.v_strides, v); set_strides(a.o_strides, o);
    set_strides(a.do_strides, d_o); set_strides(a.dq_strides, dq); set_strides(a.dk_strides, dk); set_strides(a.dv_strides, dv);
    set_strides(a.lse_strides, lse);
    if (d_lse.defined()) {
      a.d_lse = d_lse.const_data_ptr<float>();
      set_strides(a.dlse_strides, d_lse);
    }
    // delta and the fp32 dQ sums share one allocation (the sums need 16-byte alignment)
    const int64_t rows = ((int64_t)a.s.B * a.s.H * a.s.Lq + 3) / 4 * 4;
    a.delta = reinterpret_cast<float*>(16);  // any non-null value: the query below only looks at geometry and pointers
    const bool tc = c.lib->bwd_uses_tc(&a) == 1;
    const bool sums = tc && !g_deterministic.load() && !at::globalContext().deterministicAlgorithms();
    const int64_t n_sums = sums ? (int64_t)(c.lib->accum_bytes(&a.s) / sizeof(float)) : 0;
    Tensor work = at::empty({rows + n_sums}, q.options().dtype(at::kFloat));
    a.delta = work.mutable_data_ptr<float>();
    a.dq_accum = n_sums > 0 ? a.delta + rows : nullptr;
    (tc ? g_bwd_tc : g_bwd_generic) += 1;
    void* stream = current_stream(q);
    int st = c.lib->delta(&a, stream);
    if (st == CHILL_OK) st = c.lib->bwd(&a, stream);
    check(*c.lib, st, "chill_bwd");
    return {dq, dk, dv, Tensor(), Tensor(), Tensor()};
  }
};

// The argument checks of chill_attention(); the caller repeats them in Python for the message.
bool arguments_ok(const Tensor& q, const Tensor& k, const Tensor& v, const std::optional<Tensor>& lens) {
  if (q.dim() != 4 || k.dim() != 4 || v.dim() != 4) return false;
  const int64_t B = q.size(0), T = q.size(2), D = q.size(3);
  if (D != 16 && D != 32 && D != 64 && D != 128 && D != 256) return false;
  if (k.size(1) == 0 || q.size(1) % k.size(1) != 0 || k.sizes() != v.sizes()) return false;
  if (k.size(0) != B || k.size(2) != T || k.size(3) != D) return false;
  const auto dt = q.scalar_type();
  if (k.scalar_type() != dt || v.scalar_type() != dt || (dt != at::kFloat && dt != at::kHalf && dt != at::kBFloat16)) return false;
  if (!q.is_cuda() || k.device() != q.device() || v.device() != q.device()) return false;
  if (lens.has_value() && (lens->scalar_type() != at::kInt || lens->dim() != 1 || lens->size(0) != B || lens->device() != q.device()))
    return false;
  return true;
}

// Mask constants as both members of the descriptor.  The whole number is what Python's int() makes of the constant, which
// refuses NaN and infinity; what 64 bits do not hold is saturated (the library clamps further).
void set_mask_constants(chill_mask_desc& desc, const py::tuple& mask_args) {
  if (mask_args.size() > CHILL_MAX_MASK_ARGS) throw py::value_error("a mask takes at most 8 constants");
  desc.n_args = (int32_t)mask_args.size();
  for (size_t n = 0; n < mask_args.size(); ++n) {
    const py::object x = mask_args[n];
    const py::object whole = py::reinterpret_steal<py::object>(PyNumber_Long(x.ptr()));
    if (!whole) throw py::error_already_set();
    int overflow = 0;
    const long long i = PyLong_AsLongLongAndOverflow(whole.ptr(), &overflow);
    desc.i[n] = overflow == 0 ? i : (overflow > 0 ? INT64_MAX : INT64_MIN);
    desc.f[n] = PyFloat_AsDouble(x.ptr());
    if (PyErr_Occurred()) throw py::error_already_set();
  }
}

// O, (O, LSE) when return_lse, or None when the arguments do not pass the checks.
py::object attention(std::shared_ptr<Library> lib, const Tensor& q, const Tensor& k, const Tensor& v, std::optional<Tensor> lens,
                     const py::tuple& mask_args, double sm_scale, bool return_lse, uint32_t flags) {
  if (!arguments_ok(q, k, v, lens)) return py::none();
  auto call = c10::make_intrusive<Call>();
  call->mask = chill_mask_desc{};
  call->mask.id = lib->functor_id;
  call->lib = std::move(lib);
  set_mask_constants(call->mask, mask_args);
  call->sm_scale = sm_scale;
  call->flags = flags;
  c10::cuda::CUDAGuard guard(q.device());
  if (lens.has_value() && !lens->is_contiguous()) lens = lens->contiguous();
  Tensor o, lse;
  {
    py::gil_scoped_release no_gil;
    if (at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad())) {
      variable_list out = AttentionFn::apply(q, k, v, lens, call, return_lse);
      o = out[0];
      lse = out[1];
    } else {
      std::tie(o, lse) = forward(packed(q), packed(k), packed(v), lens, *call, return_lse);
    }
  }
  if (!return_lse) return py::cast(o);
  return py::make_tuple(o, lse);
}

template <class F>
F pointer(uint64_t address) {
  return reinterpret_cast<F>(static_cast<uintptr_t>(address));
}

}  // namespace

PYBIND11_MODULE(_chill_torch, m) {
  py::class_<Library, std::shared_ptr<Library>>(m, "Library")
      .def(py::init([](const std::vector<uint64_t>& fn, int32_t functor_id) {
        if (fn.size() != 7) throw py::value_error("seven entry points");
        return std::make_shared<Library>(Library{pointer<decltype(&chill_fwd)>(fn[0]), pointer<decltype(&chill_bwd_delta)>(fn[1]),
                       pointer<decltype(&chill_bwd)>(fn[2]), pointer<decltype(&chill_bwd_uses_tensor_cores)>(fn[3]),
                       pointer<decltype(&chill_bwd_dq_accum_bytes)>(fn[4]), pointer<decltype(&chill_status_string)>(fn[5]),
                       pointer<decltype(&chill_last_cuda_error)>(fn[6]), functor_id});
      }));
  m.def("attention", &attention);
  m.def("mask_constants", [](const py::tuple& mask_args) {  // what attention() hands to the library
    chill_mask_desc desc{};
    set_mask_constants(desc, mask_args);
    std::vector<std::pair<int64_t, double>> out;
    for (int n = 0; n < desc.n_args; ++n) out.emplace_back(desc.i[n], desc.f[n]);
    return out;
  });
  m.def("set_deterministic", [](bool flag) { g_deterministic = flag; });
  m.def("backward_counts", [] { return std::make_pair(g_bwd_tc.load(), g_bwd_generic.load()); });
  m.attr("abi_version") = CHILL_ABI_VERSION;
}
