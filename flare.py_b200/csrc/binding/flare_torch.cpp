// The torch side of the library in native code: argument checks, layout folding, buffer allocation, autograd and the
// C-ABI call of every public operation.
//
// The small calls of this library are bound by the host: a forward pass of a thousand tokens is ten microseconds of
// device work, and the same steps in Python (torch.library.custom_op, ctypes, a dozen tensor constructors) took sixty.
// Here a call is one vector-call into this module, one dispatcher hop for the operators that torch.compile and fake
// tensors must see (flare_b200::mixer_fwd, ...), and the launches.
//
// The operators are defined here (CUDA and Autograd kernels); their fake kernels are registered from mixer.py.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>
#include <torch/library.h>

#include "flare_b200.h"

namespace {

using at::Tensor;
using std::optional;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

PyObject* g_flare_error = nullptr;   // _cabi.FlareError

[[noreturn]] void raise_py(PyObject* type, const std::string& msg) {
  {
    pybind11::gil_scoped_acquire gil;
    PyErr_SetString(type, msg.c_str());
    python_error e;
    e.persist();
    throw e;
  }
}

void check_rc(int rc, const char* what) {
  if (rc == FLARE_OK) return;
  raise_py(g_flare_error ? g_flare_error : PyExc_RuntimeError,
           std::string(what) + " failed (code " + std::to_string(rc) + "): " + flare_last_error());
}

void need_cuda(const Tensor& t) {
  if (!t.is_cuda()) raise_py(PyExc_RuntimeError, "flare_b200 runs on CUDA tensors only (sm_100a); got a CPU tensor");
}

int dtype_code(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return FLARE_F32;
    case at::kHalf: return FLARE_F16;
    case at::kBFloat16: return FLARE_BF16;
    default: raise_py(PyExc_TypeError, std::string("unsupported dtype ") + at::toString(t.scalar_type()));
  }
}

void same_dtype(const char* msg, std::initializer_list<const Tensor*> ts) {
  for (const Tensor* t : ts)
    if (t->scalar_type() != (*ts.begin())->scalar_type()) raise_py(PyExc_TypeError, msg);
}

// Whether the kernels can address t in place: unit stride on the last dimension, 16-byte aligned rows, no broadcast
// (stride 0) dimension -- a TMA tensor map cannot describe one.
bool addressable(const Tensor& t) {
  const auto st = t.strides();
  const auto sz = t.sizes();
  const int64_t e = t.element_size(), nd = t.dim();
  if (nd == 0) raise_py(PyExc_IndexError, "expected a tensor of four dimensions, got a scalar");
  if (st[nd - 1] != 1 || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16) return false;
  for (int64_t i = 0; i + 1 < nd; ++i)
    if ((st[i] * e) % 16 || (st[i] == 0 && sz[i] != 1)) return false;
  return true;
}
Tensor tok(const Tensor& t) { return addressable(t) ? t : t.contiguous(); }

// q as [H,M,D] (latents shared by the batch) or [B,H,M,D]; an expand()-ed batch is folded back.
Tensor latents(const Tensor& q) {
  if (q.dim() != 3 && q.dim() != 4) {
    raise_py(PyExc_ValueError, "q must be [H,M,D] or [B,H,M,D]");
  }
  if (q.dim() == 4 && q.stride(0) == 0) return tok(q.select(0, 0));
  return tok(q);
}

// What the kernels write a [B,H,N,D] result into: k's strides when its last dimension is dense, else row-major.
Tensor like_tokens(const Tensor& k) {
  if (k.is_non_overlapping_and_dense() && k.stride(-1) == 1)
    return at::detail::empty_strided_cuda(k.sizes(), k.strides(), k.options());
  Tensor y = at::empty_like(k);
  return y.stride(-1) == 1 ? y : at::detail::empty_cuda(k.sizes(), k.options());
}

Tensor f32(at::IntArrayRef sizes, const Tensor& like) {
  return at::detail::empty_cuda(sizes, like.options().dtype(at::kFloat));
}
Tensor scratch(size_t bytes, const Tensor& like) {
  return at::detail::empty_cuda({(int64_t)bytes}, like.options().dtype(at::kByte));
}

void set_stride(int64_t (&dst)[3], const Tensor& t) {
  if (t.dim() < 3) raise_py(PyExc_ValueError, "expected a tensor of four dimensions, got " + std::to_string(t.dim()));
  const auto s = t.strides();
  for (int i = 0; i < 3; ++i) dst[i] = s[i];
}

FlareProblem problem(const Tensor& q, const Tensor& k, double scale) {
  FlareProblem p{};
  const auto ks = k.sizes();
  if (k.dim() != 4) raise_py(PyExc_ValueError, "k must be [B,H,N,D]");
  const auto qs = q.sizes();
  const auto qst = q.strides();
  const int o = q.dim() == 4 ? 1 : 0;
  if (o && qs[0] != ks[0]) raise_py(PyExc_ValueError, "q batch does not match k");
  if (qs[o] != ks[1] || qs[o + 2] != ks[3]) raise_py(PyExc_ValueError, "q does not match k in heads or head dimension");
  p.B = (int32_t)ks[0]; p.H = (int32_t)ks[1]; p.N = (int32_t)ks[2]; p.M = (int32_t)qs[o + 1]; p.D = (int32_t)ks[3];
  p.dtype = dtype_code(k);
  p.scale = (float)scale;
  p.q_stride[0] = o ? qst[0] : 0; p.q_stride[1] = qst[o]; p.q_stride[2] = qst[o + 1];
  set_stride(p.k_stride, k);
  return p;
}

// The key mask as one byte per token, non-zero = keep.  torch.bool already is that.
struct Mask {
  Tensor hold;
  const uint8_t* ptr = nullptr;
  Mask(const optional<Tensor>& m, const FlareProblem& p, const Tensor& k) {
    if (!m.has_value() || !m->defined()) return;
    if (m->dim() != 2 || m->size(0) != p.B || m->size(1) != p.N) raise_py(PyExc_ValueError, "key_mask must be [B,N]");
    hold = *m;
    if (hold.device() != k.device() || (hold.scalar_type() != at::kBool && hold.scalar_type() != at::kByte))
      hold = hold.to(k.device(), at::kByte);
    hold = hold.contiguous();
    ptr = static_cast<const uint8_t*>(hold.data_ptr());
  }
};

float* fp(const Tensor& t) { return static_cast<float*>(t.data_ptr()); }
flare_stream_t stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// ------------------------------------------------------------------------------------------------
// the mixer
// ------------------------------------------------------------------------------------------------
using Four = std::tuple<Tensor, Tensor, Tensor, Tensor>;
using Three = std::tuple<Tensor, Tensor, Tensor>;
using Two = std::tuple<Tensor, Tensor>;

Four mixer_fwd(const Tensor& q_, const Tensor& k_, const Tensor& v_, double scale, const optional<Tensor>& key_mask,
               double dropout_p, int64_t dropout_seed) {
  same_dtype("q, k, v must share a dtype", {&q_, &k_, &v_});
  c10::cuda::CUDAGuard guard(k_.device());
  const Tensor q = latents(q_), k = tok(k_), v = tok(v_);
  FlareProblem p = problem(q, k, scale);
  const Mask mask(key_mask, p, k);
  Tensor y = like_tokens(k);
  Tensor z32 = f32({p.B, p.H, p.M, p.D}, k), lse_m = f32({p.B, p.H, p.M}, k), lse_n = f32({p.B, p.H, p.N}, k);
  set_stride(p.v_stride, v);
  set_stride(p.y_stride, y);
  p.dropout_p = (float)dropout_p;
  p.dropout_seed = (uint64_t)dropout_seed;
  const size_t bytes = flare_fwd_workspace_bytes(&p);
  const Tensor ws = scratch(bytes, k);
  check_rc(flare_mixer_fwd(&p, q.data_ptr(), k.data_ptr(), v.data_ptr(), mask.ptr, y.data_ptr(), fp(z32), fp(lse_m),
                           fp(lse_n), ws.data_ptr(), bytes, stream_of(k)), "flare_mixer_fwd");
  return {y, z32, lse_m, lse_n};
}

Three mixer_bwd(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& dy_, const Tensor& y_,
                const Tensor& z32, const Tensor& lse_m, const Tensor& lse_n, double scale,
                const optional<Tensor>& key_mask, double dropout_p, int64_t dropout_seed) {
  c10::cuda::CUDAGuard guard(k_.device());
  const Tensor q = latents(q_), k = tok(k_), v = tok(v_), dy = tok(dy_), y = tok(y_);
  FlareProblem p = problem(q, k, scale);
  const Mask mask(key_mask, p, k);
  Tensor dk = like_tokens(k), dv = like_tokens(v);
  Tensor dq = f32(q.sizes(), k);
  set_stride(p.v_stride, v);
  set_stride(p.y_stride, y);
  set_stride(p.dy_stride, dy);
  set_stride(p.dk_stride, dk);
  set_stride(p.dv_stride, dv);
  p.dropout_p = (float)dropout_p;
  p.dropout_seed = (uint64_t)dropout_seed;
  const size_t bytes = flare_bwd_workspace_bytes(&p);
  const Tensor ws = scratch(bytes, k);
  check_rc(flare_mixer_bwd(&p, q.data_ptr(), k.data_ptr(), v.data_ptr(), dy.data_ptr(), y.data_ptr(), mask.ptr, fp(z32),
                           fp(lse_m), fp(lse_n), fp(dq), dk.data_ptr(), dv.data_ptr(), ws.data_ptr(), bytes,
                           stream_of(k)), "flare_mixer_bwd");
  return {dq, dk, dv};
}

// ------------------------------------------------------------------------------------------------
// gather and scatter on their own
// ------------------------------------------------------------------------------------------------
// the range sums of dq of every batch entry; a batch that shares its latents adds up over the batch too
Tensor sum_dq(const FlareProblem& p, const Tensor& part, const Tensor& q, flare_stream_t st) {
  Tensor dq = f32(q.sizes(), part);
  const bool batched = q.dim() == 4;
  check_rc(flare_reduce_sum(fp(part), batched ? p.n_splits : p.n_splits * p.B,
                            (int64_t)(batched ? p.B : 1) * p.H * p.M, p.D, fp(dq), st), "flare_reduce_sum");
  return dq;
}

Three gather_fwd(const Tensor& q_, const Tensor& k_, const Tensor& v_, double scale, const optional<Tensor>& key_mask) {
  c10::cuda::CUDAGuard guard(k_.device());
  const Tensor q = latents(q_), k = tok(k_), v = tok(v_);
  FlareProblem p = problem(q, k, scale);
  const Mask mask(key_mask, p, k);
  Tensor z32 = f32({p.B, p.H, p.M, p.D}, k), lse_m = f32({p.B, p.H, p.M}, k);
  Tensor z = at::detail::empty_cuda({p.B, p.H, p.M, p.D}, k.options());
  set_stride(p.v_stride, v);
  p.n_splits = flare_pick_splits(&p);
  const Tensor rec = f32({p.n_splits, p.B, p.H, p.M, p.D + 2}, k);
  const flare_stream_t st = stream_of(k);
  check_rc(flare_gather_partial(&p, q.data_ptr(), k.data_ptr(), v.data_ptr(), mask.ptr, fp(rec), st), "flare_gather_partial");
  check_rc(flare_combine(&p, fp(rec), p.n_splits, fp(z32), z.data_ptr(), fp(lse_m), nullptr, st), "flare_combine");
  return {z, z32, lse_m};
}

Three gather_bwd(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& dz, const Tensor& z32,
                 const Tensor& lse_m, double scale, const optional<Tensor>& key_mask) {
  c10::cuda::CUDAGuard guard(k_.device());
  const Tensor q = latents(q_), k = tok(k_), v = tok(v_);
  FlareProblem p = problem(q, k, scale);
  const Mask mask(key_mask, p, k);
  const Tensor dz32 = dz.to(at::kFloat).contiguous();
  Tensor dk = at::detail::empty_cuda(k.sizes(), k.options()), dv = at::detail::empty_cuda(v.sizes(), v.options());
  set_stride(p.v_stride, v);
  set_stride(p.dk_stride, dk);
  set_stride(p.dv_stride, dv);
  p.n_splits = flare_pick_splits(&p);
  const flare_stream_t st = stream_of(k);
  const Tensor part = f32({p.n_splits, p.B, p.H, p.M, p.D}, k);
  check_rc(flare_bwd_main(&p, FLARE_TERM_GATHER, q.data_ptr(), k.data_ptr(), v.data_ptr(), nullptr, nullptr, mask.ptr,
                          fp(z32), fp(dz32), fp(lse_m), nullptr, dk.data_ptr(), dv.data_ptr(), nullptr, fp(part), st),
           "flare_bwd_main");
  return {sum_dq(p, part, q, st), dk, dv};
}

Two scatter_fwd(const Tensor& q_, const Tensor& k_, const Tensor& z, double scale, const optional<Tensor>& key_mask) {
  c10::cuda::CUDAGuard guard(k_.device());
  const Tensor q = latents(q_), k = tok(k_);
  FlareProblem p = problem(q, k, scale);
  const Mask mask(key_mask, p, k);
  const Tensor z32 = z.to(at::kFloat).contiguous();
  Tensor y = like_tokens(k), lse_n = f32({p.B, p.H, p.N}, k);
  set_stride(p.y_stride, y);
  check_rc(flare_scatter(&p, q.data_ptr(), k.data_ptr(), fp(z32), mask.ptr, y.data_ptr(), fp(lse_n), stream_of(k)),
           "flare_scatter");
  return {y, lse_n};
}

Three scatter_bwd(const Tensor& q_, const Tensor& k_, const Tensor& z, const Tensor& dy_, const Tensor& y_,
                  const Tensor& lse_n, double scale, const optional<Tensor>& key_mask) {
  c10::cuda::CUDAGuard guard(k_.device());
  const Tensor q = latents(q_), k = tok(k_), dy = tok(dy_), y = tok(y_);
  FlareProblem p = problem(q, k, scale);
  const Mask mask(key_mask, p, k);
  const Tensor z32 = z.to(at::kFloat).contiguous();
  Tensor dk = at::detail::empty_cuda(k.sizes(), k.options());
  set_stride(p.y_stride, y);
  set_stride(p.dy_stride, dy);
  set_stride(p.dk_stride, dk);
  p.n_splits = flare_pick_splits(&p);
  const flare_stream_t st = stream_of(k);
  const Tensor part = f32({p.n_splits, p.B, p.H, p.M, p.D}, k);
  Tensor dz32 = f32({p.B, p.H, p.M, p.D}, k);
  const Tensor delta = f32({p.B, p.H, p.N}, k);
  check_rc(flare_bwd_dz_partial(&p, q.data_ptr(), k.data_ptr(), dy.data_ptr(), mask.ptr, fp(lse_n), fp(part), st),
           "flare_bwd_dz_partial");
  check_rc(flare_reduce_sum(fp(part), p.n_splits, (int64_t)p.B * p.H * p.M, p.D, fp(dz32), st), "flare_reduce_sum");
  check_rc(flare_bwd_main(&p, FLARE_TERM_SCATTER, q.data_ptr(), k.data_ptr(), nullptr, dy.data_ptr(), y.data_ptr(),
                          mask.ptr, fp(z32), nullptr, nullptr, fp(lse_n), dk.data_ptr(), nullptr, fp(delta), fp(part), st),
           "flare_bwd_main");
  return {sum_dq(p, part, q, st), dk, dz32};
}

// ------------------------------------------------------------------------------------------------
// operators and autograd
// ------------------------------------------------------------------------------------------------
#define FLARE_OP(name)                                                                                        \
  struct Op_##name {                                                                                          \
    static const auto& get() {                                                                                \
      static const auto h =                                                                                   \
          c10::Dispatcher::singleton().findSchemaOrThrow("flare_b200::" #name, "").typed<decltype(name)>();   \
      return h;                                                                                               \
    }                                                                                                         \
  };
FLARE_OP(mixer_fwd)
FLARE_OP(mixer_bwd)
FLARE_OP(gather_fwd)
FLARE_OP(gather_bwd)
FLARE_OP(scatter_fwd)
FLARE_OP(scatter_bwd)

// In torch.autocast the latents stay the module's fp32 parameter and meet 16-bit projections here: rounding them
// inside the operator keeps the cast and its backward out of the autograd graph, and dq is returned in q's own dtype
// without passing through 16 bits.
Tensor as_dtype(const Tensor& t, at::ScalarType dt) { return t.scalar_type() == dt ? t : t.to(dt); }
optional<Tensor> maybe(const Tensor& t) { return t.defined() ? optional<Tensor>(t) : std::nullopt; }

// The autograd functions of the operators return the result alone; z32 and the log-sum-exps, the backward's operands and not
// results anyone differentiates, reach the caller through `rest`.  As outputs they would have to be marked as
// non-differentiable, which compiled autograd refuses, or be wrapped and saved as differentiable ones (6 us a step).
class MixerFn : public torch::autograd::Function<MixerFn> {
 public:
  static constexpr bool is_traceable = true;       // compiled autograd may trace the backward: it calls operators only
  static Tensor forward(AutogradContext* ctx, const Tensor& q_, const Tensor& k, const Tensor& v, double scale,
                        const optional<Tensor>& key_mask, double dropout_p, int64_t dropout_seed, Three* rest) {
    at::AutoDispatchBelowADInplaceOrView below;
    const Tensor q = as_dtype(q_, k.scalar_type());
    auto [y, z32, lse_m, lse_n] = Op_mixer_fwd::get().call(q, k, v, scale, key_mask, dropout_p, dropout_seed);
    ctx->save_for_backward({q, k, v, y, z32, lse_m, lse_n, key_mask.value_or(Tensor())});
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["p"] = dropout_p;
    ctx->saved_data["seed"] = dropout_seed;
    ctx->saved_data["qdt"] = (int64_t)q_.scalar_type();
    ctx->set_materialize_grads(false);
    *rest = {z32, lse_m, lse_n};
    return y;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    if (!g[0].defined()) return variable_list(8);
    const auto s = ctx->get_saved_variables();
    auto [dq, dk, dv] = Op_mixer_bwd::get().call(s[0], s[1], s[2], g[0], s[3], s[4], s[5], s[6], ctx->saved_data["scale"].toDouble(),
                                                 maybe(s[7]), ctx->saved_data["p"].toDouble(), ctx->saved_data["seed"].toInt());
    return {as_dtype(dq, (at::ScalarType)ctx->saved_data["qdt"].toInt()), dk, dv, Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

class GatherFn : public torch::autograd::Function<GatherFn> {
 public:
  static constexpr bool is_traceable = true;       // compiled autograd may trace the backward: it calls operators only
  static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, double scale,
                        const optional<Tensor>& key_mask, Two* rest) {
    at::AutoDispatchBelowADInplaceOrView below;
    auto [z, z32, lse_m] = Op_gather_fwd::get().call(q, k, v, scale, key_mask);
    ctx->save_for_backward({q, k, v, z32, lse_m, key_mask.value_or(Tensor())});
    ctx->saved_data["scale"] = scale;
    ctx->set_materialize_grads(false);
    *rest = {z32, lse_m};
    return z;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    if (!g[0].defined()) return variable_list(6);
    const auto s = ctx->get_saved_variables();
    auto [dq, dk, dv] = Op_gather_bwd::get().call(s[0], s[1], s[2], g[0], s[3], s[4], ctx->saved_data["scale"].toDouble(), maybe(s[5]));
    return {as_dtype(dq, s[0].scalar_type()), dk, dv, Tensor(), Tensor(), Tensor()};
  }
};

class ScatterFn : public torch::autograd::Function<ScatterFn> {
 public:
  static constexpr bool is_traceable = true;       // compiled autograd may trace the backward: it calls operators only
  static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& z, double scale,
                        const optional<Tensor>& key_mask, Tensor* rest) {
    at::AutoDispatchBelowADInplaceOrView below;
    auto [y, lse_n] = Op_scatter_fwd::get().call(q, k, z, scale, key_mask);
    ctx->save_for_backward({q, k, z, y, lse_n, key_mask.value_or(Tensor())});
    ctx->saved_data["scale"] = scale;
    ctx->set_materialize_grads(false);
    *rest = lse_n;
    return y;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    if (!g[0].defined()) return variable_list(6);
    const auto s = ctx->get_saved_variables();
    auto [dq, dk, dz] = Op_scatter_bwd::get().call(s[0], s[1], s[2], g[0], s[3], s[4], ctx->saved_data["scale"].toDouble(), maybe(s[5]));
    return {as_dtype(dq, s[0].scalar_type()), dk, as_dtype(dz, s[2].scalar_type()), Tensor(), Tensor(), Tensor()};
  }
};

Four mixer_fwd_autograd(const Tensor& q, const Tensor& k, const Tensor& v, double scale, const optional<Tensor>& key_mask,
                        double dropout_p, int64_t dropout_seed) {
  if (!torch::autograd::compute_requires_grad(q, k, v)) {
    at::AutoDispatchBelowADInplaceOrView below;
    return Op_mixer_fwd::get().call(q, k, v, scale, key_mask, dropout_p, dropout_seed);
  }
  Three rest;
  const Tensor y = MixerFn::apply(q, k, v, scale, key_mask, dropout_p, dropout_seed, &rest);
  return {y, std::get<0>(rest), std::get<1>(rest), std::get<2>(rest)};
}
// The backward operators have no derivative of their own: where a graph of them is recorded (create_graph), differentiating
// their results raises instead of leaving their share out.
template <typename... In>
Three no_second_derivative(const char* name, Three r, const In&... in) {
  if (torch::autograd::compute_requires_grad(in...)) {
    const std::shared_ptr<torch::autograd::Node> node(
        new torch::autograd::NotImplemented(name, torch::autograd::collect_next_edges(in...)), torch::autograd::deleteNode);
    for (const Tensor& t : {std::get<0>(r), std::get<1>(r), std::get<2>(r)}) torch::autograd::set_history(t, node);
  }
  return r;
}
Three mixer_bwd_autograd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& dy, const Tensor& y,
                         const Tensor& z32, const Tensor& lse_m, const Tensor& lse_n, double scale,
                         const optional<Tensor>& key_mask, double dropout_p, int64_t dropout_seed) {
  Three r;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    r = Op_mixer_bwd::get().call(q, k, v, dy, y, z32, lse_m, lse_n, scale, key_mask, dropout_p, dropout_seed);
  }
  return no_second_derivative("flare_b200::mixer_bwd", std::move(r), q, k, v, dy, y, z32, lse_m, lse_n);
}
Three gather_bwd_autograd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& dz, const Tensor& z32,
                          const Tensor& lse_m, double scale, const optional<Tensor>& key_mask) {
  Three r;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    r = Op_gather_bwd::get().call(q, k, v, dz, z32, lse_m, scale, key_mask);
  }
  return no_second_derivative("flare_b200::gather_bwd", std::move(r), q, k, v, dz, z32, lse_m);
}
Three scatter_bwd_autograd(const Tensor& q, const Tensor& k, const Tensor& z, const Tensor& dy, const Tensor& y,
                           const Tensor& lse_n, double scale, const optional<Tensor>& key_mask) {
  Three r;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    r = Op_scatter_bwd::get().call(q, k, z, dy, y, lse_n, scale, key_mask);
  }
  return no_second_derivative("flare_b200::scatter_bwd", std::move(r), q, k, z, dy, y, lse_n);
}
Three gather_fwd_autograd(const Tensor& q, const Tensor& k, const Tensor& v, double scale, const optional<Tensor>& key_mask) {
  if (!torch::autograd::compute_requires_grad(q, k, v)) {
    at::AutoDispatchBelowADInplaceOrView below;
    return Op_gather_fwd::get().call(q, k, v, scale, key_mask);
  }
  Two rest;
  const Tensor z = GatherFn::apply(q, k, v, scale, key_mask, &rest);
  return {z, std::get<0>(rest), std::get<1>(rest)};
}
Two scatter_fwd_autograd(const Tensor& q, const Tensor& k, const Tensor& z, double scale, const optional<Tensor>& key_mask) {
  if (!torch::autograd::compute_requires_grad(q, k, z)) {
    at::AutoDispatchBelowADInplaceOrView below;
    return Op_scatter_fwd::get().call(q, k, z, scale, key_mask);
  }
  Tensor lse_n;
  const Tensor y = ScatterFn::apply(q, k, z, scale, key_mask, &lse_n);
  return {y, lse_n};
}

// ------------------------------------------------------------------------------------------------
// causal FLARE
// ------------------------------------------------------------------------------------------------
Two causal_prefill(const Tensor& q_, const Tensor& k_, const Tensor& v_, double scale, const optional<Tensor>& state_) {
  for (const Tensor* t : {&q_, &k_, &v_}) need_cuda(*t);
  same_dtype("q, k, v must share a dtype", {&q_, &k_, &v_});
  c10::cuda::CUDAGuard guard(k_.device());
  const Tensor q = latents(q_), k = tok(k_), v = tok(v_);
  FlareProblem p = problem(q, k, scale);
  Tensor y = at::detail::empty_cuda(k.sizes(), k.options());
  Tensor out = f32({p.B, p.H, p.M, p.D + 2}, k);
  set_stride(p.v_stride, v);
  set_stride(p.y_stride, y);
  const Tensor state = state_.has_value() ? state_->contiguous() : Tensor();
  const Tensor ws = scratch(flare_causal_workspace_bytes(&p), k);
  check_rc(flare_causal_prefill(&p, q.data_ptr(), k.data_ptr(), v.data_ptr(), y.data_ptr(),
                                state.defined() ? fp(state) : nullptr, fp(out), fp(ws), stream_of(k)), "flare_causal_prefill");
  return {y, out};
}

Tensor causal_decode(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& state, double scale) {
  for (const Tensor* t : {&q_, &k_, &v_, &state}) need_cuda(*t);
  c10::cuda::CUDAGuard guard(k_.device());
  const Tensor q = latents(q_), k = tok(k_), v = tok(v_);
  FlareProblem p = problem(q, k, scale);
  if (state.scalar_type() != at::kFloat || !state.is_contiguous() || state.sizes() != at::IntArrayRef({p.B, p.H, p.M, p.D + 2}))
    raise_py(PyExc_ValueError, "state must be a contiguous fp32 [B,H,M,D+2] tensor");
  Tensor y = at::detail::empty_cuda(k.sizes(), k.options());
  set_stride(p.v_stride, v);
  set_stride(p.y_stride, y);
  check_rc(flare_causal_decode(&p, q.data_ptr(), k.data_ptr(), v.data_ptr(), y.data_ptr(), fp(state), stream_of(k)),
           "flare_causal_decode");
  return y;
}

class CausalFn : public torch::autograd::Function<CausalFn> {
 public:
  // train: a gradient is wanted (asked by the caller: nothing requires one in here).  Without, it is the plain prefill: the
  // training forward takes 294 us where that takes 230 (B = 4, H = 16, N = 8192, M = 128, D = 64).
  static Tensor forward(AutogradContext* ctx, const Tensor& q_, const Tensor& k_, const Tensor& v_, double scale, bool train) {
    at::AutoDispatchBelowADInplaceOrView below;
    for (const Tensor* t : {&q_, &k_, &v_}) need_cuda(*t);
    same_dtype("q, k, v must share a dtype", {&q_, &k_, &v_});
    ctx->saved_data["scale"] = scale;
    c10::cuda::CUDAGuard guard(k_.device());
    const Tensor q = latents(q_), k = tok(k_), v = tok(v_);
    FlareProblem p = problem(q, k, scale);
    // the tensor-core shapes keep the chunk-start states for the backward (M (4 D + 8) bytes per 128 tokens and head);
    // the others rebuild them there
    const size_t bytes = train ? flare_causal_train_bytes(&p) : 0;
    Tensor y, saved;
    if (bytes) {
      y = at::detail::empty_cuda(k.sizes(), k.options());
      set_stride(p.v_stride, v);
      set_stride(p.y_stride, y);
      saved = scratch(bytes, k);
      check_rc(flare_causal_train_fwd(&p, q.data_ptr(), k.data_ptr(), v.data_ptr(), y.data_ptr(), saved.data_ptr(), stream_of(k)),
               "flare_causal_train_fwd");
    } else {
      y = std::get<0>(causal_prefill(q_, k_, v_, scale, std::nullopt));
    }
    ctx->save_for_backward({q_, k_, v_, saved});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    const auto s = ctx->get_saved_variables();
    const Tensor &q_ = s[0], &saved = s[3];
    c10::cuda::CUDAGuard guard(s[1].device());
    // a batch made by expand() is a batch here: its entries have gradients of their own, which autograd folds back itself
    const Tensor q = tok(q_), k = tok(s[1]), v = tok(s[2]), dy = tok(g[0]);
    FlareProblem p = problem(q, k, ctx->saved_data["scale"].toDouble());
    Tensor dk = at::detail::empty_cuda(k.sizes(), k.options()), dv = at::detail::empty_cuda(v.sizes(), v.options());
    set_stride(p.v_stride, v);
    set_stride(p.dy_stride, dy);
    set_stride(p.dk_stride, dk);
    set_stride(p.dv_stride, dv);
    const flare_stream_t st = stream_of(k);
    Tensor dq;
    if (saved.defined()) {
      dq = f32(q.sizes(), k);
      const Tensor ws = scratch(flare_causal_train_bwd_workspace_bytes(&p), k);
      check_rc(flare_causal_train_bwd(&p, q.data_ptr(), k.data_ptr(), v.data_ptr(), dy.data_ptr(), saved.data_ptr(), fp(dq),
                                      dk.data_ptr(), dv.data_ptr(), ws.data_ptr(), st), "flare_causal_train_bwd");
    } else {
      dq = f32({p.B, p.H, p.M, p.D}, k);
      const Tensor ws = scratch(flare_causal_bwd_workspace_bytes(&p), k);
      check_rc(flare_causal_bwd(&p, q.data_ptr(), k.data_ptr(), v.data_ptr(), dy.data_ptr(), fp(dq), dk.data_ptr(),
                                dv.data_ptr(), fp(ws), st), "flare_causal_bwd");
      // one latent gradient per (b, h): shared latents sum over the batch
      if (q.dim() == 3) {
        Tensor sum = f32({p.H, p.M, p.D}, k);
        check_rc(flare_reduce_sum(fp(dq), p.B, (int64_t)p.H * p.M, p.D, fp(sum), st), "flare_reduce_sum");
        dq = sum;
      }
    }
    return {as_dtype(dq, q_.scalar_type()), dk, dv, Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------------------------
// triple attention and causal linear attention
// ------------------------------------------------------------------------------------------------
Tensor flat(const Tensor& t) {
  return t.dim() == 3 ? t : t.reshape({t.size(0) * t.size(1), t.size(2), t.size(3)}).contiguous();
}
// What the backward keeps of an input: the input itself where flat() is a view of it (made here, that view would not
// share its version counter, and a change in place before the backward would go unnoticed), else flat()'s copy.
Tensor keep(const Tensor& t, const Tensor& flat_t) { return flat_t.is_alias_of(t) ? t : flat_t; }

Tensor triple_outer(const Tensor& a, const Tensor& b, const Tensor& c, double alpha) {
  const int BH = (int)a.size(0), N = (int)a.size(1), Da = (int)a.size(2), Db = (int)b.size(2), Dc = (int)c.size(2);
  Tensor out = f32({BH, Da, Db, Dc}, a);
  const Tensor ws = scratch(flare_triple_workspace_bytes(BH, N, Da, Db, Dc), a);
  check_rc(flare_triple_outer(BH, N, Da, Db, Dc, dtype_code(a), a.data_ptr(), b.data_ptr(), c.data_ptr(), (float)alpha,
                              fp(out), fp(ws), stream_of(a)), "flare_triple_outer");
  return out;
}
// out[n,x] = alpha * sum_{y,z} t.permute(perm)[x,y,z] a[n,y] b[n,z]; t is [BH,D0,D1,D2] fp32 contiguous
Tensor triple_contract(const Tensor& t, int x, int y, int z, const Tensor& a, const Tensor& b, double alpha) {
  const int BH = (int)a.size(0), N = (int)a.size(1), Dx = (int)t.size(1 + x);
  Tensor out = at::detail::empty_cuda({BH, N, Dx}, a.options());
  check_rc(flare_triple_contract(BH, N, Dx, (int)a.size(2), (int)b.size(2), dtype_code(a), fp(t), t.stride(1 + x),
                                 t.stride(1 + y), t.stride(1 + z), a.data_ptr(), b.data_ptr(), (float)alpha,
                                 out.data_ptr(), stream_of(a)), "flare_triple_contract");
  return out;
}

// The kernels take every size from one operand and index the others and the rank-3 tensor by it: q1 and q2 must agree in
// heads and tokens, so must k1, k2 and v, and q1, q2, k1, k2 in features.
void check_triple(const Tensor& q1, const Tensor& q2, const Tensor& k1, const Tensor& k2, const Tensor& v) {
  for (const Tensor* t : {&q1, &q2, &k1, &k2, &v})
    if (t->dim() != 4) raise_py(PyExc_ValueError, "q1, q2, k1, k2, v must be [B,H,N,D]");
  auto rows = [](const Tensor& a, const Tensor& b) { return a.size(0) * a.size(1) == b.size(0) * b.size(1) && a.size(2) == b.size(2); };
  if (!rows(q1, q2) || !rows(k1, k2) || !rows(k1, v) || q1.size(0) * q1.size(1) != k1.size(0) * k1.size(1))
    raise_py(PyExc_ValueError, "q1, q2 (and k1, k2, v) must agree in batch, heads and tokens");
  for (const Tensor* t : {&q2, &k1, &k2})
    if (t->size(3) != q1.size(3)) raise_py(PyExc_ValueError, "q1, q2, k1, k2 must share a feature dimension");
}

class TripleFn : public torch::autograd::Function<TripleFn> {
 public:
  static variable_list forward(AutogradContext* ctx, const Tensor& q1, const Tensor& q2, const Tensor& k1, const Tensor& k2,
                               const Tensor& v) {
    at::AutoDispatchBelowADInplaceOrView below;
    for (const Tensor* t : {&q1, &q2, &k1, &k2, &v}) need_cuda(*t);
    same_dtype("q1, q2, k1, k2, v must share a dtype", {&q1, &q2, &k1, &k2, &v});
    check_triple(q1, q2, k1, k2, v);
    c10::cuda::CUDAGuard guard(v.device());
    const int64_t B = q1.size(0), H = q1.size(1), N = q1.size(2), Dq = q1.size(3), Dv = v.size(3);
    const Tensor fq1 = flat(q1), fq2 = flat(q2), fk1 = flat(k1), fk2 = flat(k2), fv = flat(v);
    const Tensor state = triple_outer(fk1, fv, fk2, 1.0 / (double)N);                 // [BH, Dq, Dv, Dq]
    const Tensor o = triple_contract(state, 1, 0, 2, fq1, fq2, 1.0);                  // x = j, y = i, z = k
    const Tensor out = state.view({B, H, Dq, Dv, Dq});       // kept as the output it is: changing it in place is noticed too
    ctx->save_for_backward({keep(q1, fq1), keep(q2, fq2), keep(k1, fk1), keep(k2, fk2), keep(v, fv), out});
    ctx->saved_data["B"] = B;
    ctx->saved_data["H"] = H;
    ctx->set_materialize_grads(false);             // a loss on O alone adds no zero tensor to dSTATE
    return {out, o.view({B, H, N, Dv})};
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    if (!g[0].defined() && !g[1].defined()) return variable_list(5);
    const auto s = ctx->get_saved_variables();
    const Tensor fq1 = flat(s[0]), fq2 = flat(s[1]), fk1 = flat(s[2]), fk2 = flat(s[3]), fv = flat(s[4]);
    const Tensor state = s[5].flatten(0, 1);
    const int64_t B = ctx->saved_data["B"].toInt(), H = ctx->saved_data["H"].toInt();
    const int64_t N = fq1.size(1), Dq = fq1.size(2), Dv = fv.size(2);
    c10::cuda::CUDAGuard guard(fv.device());
    const Tensor fdo = g[1].defined() ? flat(as_dtype(g[1], fv.scalar_type())) : at::zeros({B * H, N, Dv}, fv.options());
    Tensor dstate = triple_outer(fq1, fdo, fq2, 1.0);
    if (g[0].defined()) dstate = dstate + g[0].reshape({B * H, Dq, Dv, Dq}).to(at::kFloat);
    const double in = 1.0 / (double)N;
    auto four = [&](const Tensor& t, int64_t D) { return t.view({B, H, N, D}); };
    return {four(triple_contract(state, 0, 1, 2, fdo, fq2, 1.0), Dq),                 // x = i, y = j, z = k
            four(triple_contract(state, 2, 0, 1, fq1, fdo, 1.0), Dq),                 // x = k, y = i, z = j
            four(triple_contract(dstate, 0, 1, 2, fv, fk2, in), Dq), four(triple_contract(dstate, 2, 0, 1, fk1, fv, in), Dq),
            four(triple_contract(dstate, 1, 0, 2, fk1, fk2, in), Dv)};
  }
};

Tensor causal_linear(const Tensor& q_, const Tensor& k_, const Tensor& v_) {
  for (const Tensor* t : {&q_, &k_, &v_}) need_cuda(*t);
  same_dtype("q, k, v must share a dtype", {&q_, &k_, &v_});
  c10::cuda::CUDAGuard guard(k_.device());
  auto rows = [](const Tensor& t) { return t.stride(-1) == 1 ? t : t.contiguous(); };
  const Tensor q = rows(q_), k = rows(k_), v = rows(v_);
  const int B = (int)k.size(0), H = (int)k.size(1), N = (int)k.size(2), Dk = (int)k.size(3), Dv = (int)v.size(3);
  Tensor y = at::detail::empty_cuda({B, H, N, Dv}, v.options());
  const Tensor ws = scratch(flare_causal_linear_workspace_bytes(B, H, N, Dk, Dv), k);
  int64_t qs[3], ks[3], vs[3], ys[3];
  set_stride(qs, q); set_stride(ks, k); set_stride(vs, v); set_stride(ys, y);
  check_rc(flare_causal_linear(B, H, N, Dk, Dv, dtype_code(k), q.data_ptr(), qs, k.data_ptr(), ks, v.data_ptr(), vs,
                               y.data_ptr(), ys, fp(ws), stream_of(k)), "flare_causal_linear");
  return y;
}

// ------------------------------------------------------------------------------------------------
// the Python module
// ------------------------------------------------------------------------------------------------
const Tensor& tensor_arg(PyObject* o) {
  if (!THPVariable_Check(o)) raise_py(PyExc_TypeError, std::string("expected a torch.Tensor, got ") + Py_TYPE(o)->tp_name);
  return THPVariable_Unpack(o);
}
optional<Tensor> optional_arg(PyObject* o) {
  if (o == Py_None) return std::nullopt;
  return tensor_arg(o);
}
double double_arg(PyObject* o) {
  const double x = PyFloat_AsDouble(o);
  if (x == -1.0 && PyErr_Occurred()) throw python_error();
  return x;
}
int64_t int_arg(PyObject* o) {
  const long long x = PyLong_AsLongLong(o);
  if (x == -1 && PyErr_Occurred()) throw python_error();
  return x;
}
void arg_count(Py_ssize_t n, Py_ssize_t want, const char* name) {
  if (n != want) raise_py(PyExc_TypeError, std::string(name) + " takes " + std::to_string(want) + " arguments, got " + std::to_string(n));
}
PyObject* pair(const Tensor& a, const Tensor& b) {
  THPObjectPtr t(PyTuple_New(2));
  if (!t) throw python_error();
  PyTuple_SET_ITEM(t.get(), 0, THPVariable_Wrap(a));
  PyTuple_SET_ITEM(t.get(), 1, THPVariable_Wrap(b));
  return t.release();
}

// Every function drops the GIL around the call, as torch's own bindings do: several threads of one process may call in.
#define FLARE_PY(name, nargs, ...)                                                  \
  PyObject* py_##name(PyObject*, PyObject* const* a, Py_ssize_t n) {                \
    HANDLE_TH_ERRORS                                                                \
    arg_count(n, nargs, #name);                                                     \
    __VA_ARGS__                                                                     \
    END_HANDLE_TH_ERRORS                                                            \
  }

FLARE_PY(mixer, 7, {
  const Tensor &q = tensor_arg(a[0]), &k = tensor_arg(a[1]), &v = tensor_arg(a[2]);
  const double scale = double_arg(a[3]), p = double_arg(a[5]);
  const optional<Tensor> mask = optional_arg(a[4]);
  const int64_t seed = int_arg(a[6]);
  need_cuda(q); need_cuda(k); need_cuda(v);
  Tensor y;
  {
    pybind11::gil_scoped_release nogil;
    // fp32 latents under autocast: MixerFn rounds them where a gradient is wanted.  The other calls round them here, since
    // the autograd kernel does not run on inference tensors or in inference mode.
    const bool grad = at::GradMode::is_enabled() && q.requires_grad();
    y = std::get<0>(Op_mixer_fwd::get().call(grad ? q : as_dtype(q, k.scalar_type()), k, v, scale, mask, p, seed));
  }
  return THPVariable_Wrap(std::move(y));
})
FLARE_PY(causal_prefill, 5, {
  const Tensor &q = tensor_arg(a[0]), &k = tensor_arg(a[1]), &v = tensor_arg(a[2]);
  const double scale = double_arg(a[3]);
  const optional<Tensor> state = optional_arg(a[4]);
  Two r;
  { pybind11::gil_scoped_release nogil; at::AutoDispatchBelowADInplaceOrView below; r = causal_prefill(q, k, v, scale, state); }
  return pair(std::get<0>(r), std::get<1>(r));
})
FLARE_PY(causal_decode, 5, {
  const Tensor &q = tensor_arg(a[0]), &k = tensor_arg(a[1]), &v = tensor_arg(a[2]), &state = tensor_arg(a[3]);
  const double scale = double_arg(a[4]);
  Tensor y;
  { pybind11::gil_scoped_release nogil; at::AutoDispatchBelowADInplaceOrView below; y = causal_decode(q, k, v, state, scale); }
  return THPVariable_Wrap(std::move(y));
})
FLARE_PY(causal_mixer, 4, {
  const Tensor &q = tensor_arg(a[0]), &k = tensor_arg(a[1]), &v = tensor_arg(a[2]);
  const double scale = double_arg(a[3]);
  Tensor y;
  const bool train = torch::autograd::compute_requires_grad(q, k, v);
  { pybind11::gil_scoped_release nogil; y = CausalFn::apply(q, k, v, scale, train); }
  return THPVariable_Wrap(std::move(y));
})
FLARE_PY(triple, 5, {
  const Tensor &q1 = tensor_arg(a[0]), &q2 = tensor_arg(a[1]), &k1 = tensor_arg(a[2]), &k2 = tensor_arg(a[3]), &v = tensor_arg(a[4]);
  variable_list r;
  { pybind11::gil_scoped_release nogil; r = TripleFn::apply(q1, q2, k1, k2, v); }
  return pair(r[0], r[1]);
})
FLARE_PY(causal_linear, 3, {
  const Tensor &q = tensor_arg(a[0]), &k = tensor_arg(a[1]), &v = tensor_arg(a[2]);
  Tensor y;
  { pybind11::gil_scoped_release nogil; at::AutoDispatchBelowADInplaceOrView below; y = causal_linear(q, k, v); }
  return THPVariable_Wrap(std::move(y));
})

PyObject* py_set_error_type(PyObject*, PyObject* type) {
  Py_XINCREF(type);
  Py_XDECREF(g_flare_error);
  g_flare_error = type;
  Py_RETURN_NONE;
}

#define FLARE_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(&py_##name)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {FLARE_METHOD(mixer), FLARE_METHOD(causal_prefill), FLARE_METHOD(causal_decode), FLARE_METHOD(causal_mixer),
                           FLARE_METHOD(triple), FLARE_METHOD(causal_linear), {"set_error_type", py_set_error_type, METH_O, nullptr},
                           {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_flare_torch", "flare_b200 operators", -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

TORCH_LIBRARY(flare_b200, m) {
  m.def("mixer_fwd(Tensor q, Tensor k, Tensor v, float scale, Tensor? key_mask, float dropout_p, int dropout_seed) -> (Tensor, Tensor, Tensor, Tensor)");
  m.def("mixer_bwd(Tensor q, Tensor k, Tensor v, Tensor dy, Tensor y, Tensor z32, Tensor lse_m, Tensor lse_n, float scale, Tensor? key_mask, float dropout_p, int dropout_seed) -> (Tensor, Tensor, Tensor)");
  m.def("gather_fwd(Tensor q, Tensor k, Tensor v, float scale, Tensor? key_mask) -> (Tensor, Tensor, Tensor)");
  m.def("gather_bwd(Tensor q, Tensor k, Tensor v, Tensor dz, Tensor z32, Tensor lse_m, float scale, Tensor? key_mask) -> (Tensor, Tensor, Tensor)");
  m.def("scatter_fwd(Tensor q, Tensor k, Tensor z, float scale, Tensor? key_mask) -> (Tensor, Tensor)");
  m.def("scatter_bwd(Tensor q, Tensor k, Tensor z, Tensor dy, Tensor y, Tensor lse_n, float scale, Tensor? key_mask) -> (Tensor, Tensor, Tensor)");
}
TORCH_LIBRARY_IMPL(flare_b200, CUDA, m) {
  m.impl("mixer_fwd", &mixer_fwd);
  m.impl("mixer_bwd", &mixer_bwd);
  m.impl("gather_fwd", &gather_fwd);
  m.impl("gather_bwd", &gather_bwd);
  m.impl("scatter_fwd", &scatter_fwd);
  m.impl("scatter_bwd", &scatter_bwd);
}
TORCH_LIBRARY_IMPL(flare_b200, Autograd, m) {
  m.impl("scatter_bwd", &scatter_bwd_autograd);
  m.impl("gather_bwd", &gather_bwd_autograd);
  m.impl("mixer_bwd", &mixer_bwd_autograd);
  m.impl("mixer_fwd", &mixer_fwd_autograd);
  m.impl("gather_fwd", &gather_fwd_autograd);
  m.impl("scatter_fwd", &scatter_fwd_autograd);
}

PyMODINIT_FUNC PyInit__flare_torch(void) { return PyModule_Create(&g_module); }
