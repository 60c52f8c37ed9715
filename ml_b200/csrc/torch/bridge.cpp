// Host path of the operators: from a torch tensor to a kernel launch without the interpreter in between.
//
// A call of a small operator costs the host more than the device: through a Python autograd.Function and ctypes a linear layer took
// ~20 us forward and ~50 us backward for kernels of 3-10 us each.  Here are
//   * the differentiable operators of ops/autograd.py as torch::autograd::Functions (the same kernels in the same order, the same
//     saved tensors, so saved-tensor hooks and checkpointing are given what they were given; what a hook gives back goes through unpacked()), and
//   * the entry points that the training engine calls most, taking tensors (ops/native.py).
// Every operator looks at its arguments first and returns NotImplemented for whatever is not the plain case (bf16 tensors of the current
// device, two-dimensional, not empty, aligned, no transform or trace or dispatch mode active): ops/autograd.py then takes the Python
// form, with the behaviour and the errors it has always had.
//
// The kernels live in libmlb_cuda.so, whose C functions are looked up by name in bind().
#include <ATen/ATen.h>
#include <ATen/SavedTensorHooks.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/graph_task.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <dlfcn.h>

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;
typedef struct MlbStream* St;
typedef std::optional<Tensor> Maybe;      // (an undefined tensor is no argument of a Function)

// ------------------------------------------------------------------ the kernel library (void*: bf16)
#define MLB_ENTRIES(X)                                                                                                                        \
  X(mlb_linear_fwd, int, (void*, const void*, const void*, int, int, int, int, int, int, St))                                                  \
  X(mlb_linear_fwd_posembed, int, (void*, const void*, const void*, const void*, int, int, int, int, int, int, int, St))                       \
  X(mlb_linear_fwd_rope, int, (void*, const void*, const void*, int, int, int, int, int, int, const float*, const float*, int, int, St))       \
  X(mlb_linear_fwd_swiglu, int, (void*, void*, const void*, const void*, int, int, int, int, int, int, St))                                    \
  X(mlb_linear_dx, int, (void*, const void*, const void*, int, int, int, int, int, int, St))                                                   \
  X(mlb_linear_dx_delta, int, (void*, const void*, const void*, const void*, float*, int, int, int, int, int, int, int, int, St))              \
  X(mlb_linear_dw, int, (float*, const void*, const void*, int, int, int, int, int, int, St))                                                  \
  X(mlb_gemm, int, (void*, const void*, const void*, int, int, int, int, int, int, int, int, int, St))                                         \
  X(mlb_gemm_dw_direct, int, (int, int, int))                                                                                                  \
  X(mlb_linear_fwd_fp8, int, (void*, const uint8_t*, const uint8_t*, int, int, int, int, int, int, float, St))                                 \
  X(mlb_capture_id, unsigned long long, (St))                                                                                                  \
  X(mlb_zero, int, (void*, long, St))                                                                                                          \
  X(mlb_cast_f2b, int, (void*, const float*, long, float, St))                                                                                 \
  X(mlb_colsum_splits, int, (long, int))                                                                                                       \
  X(mlb_colsum, int, (void*, const void*, long, int, float*, St))                                                                              \
  X(mlb_rmsnorm_fwd, int, (void*, float*, const void*, const void*, long, int, float, St))                                                     \
  X(mlb_add_rmsnorm_fwd, int, (void*, void*, float*, const void*, const void*, const void*, long, int, float, St))                             \
  X(mlb_rmsnorm_fwd_fp8, int, (void*, uint8_t*, float*, const void*, const void*, long, int, float, float, St))                                \
  X(mlb_rmsnorm_bwd_blocks, int, (long))                                                                                                       \
  X(mlb_rmsnorm_bwd, int, (void*, float*, const void*, const void*, const void*, const float*, const void*, long, int, float*, int*, St))      \
  X(mlb_rmsnorm_bwd_cast, int, (void*, void*, const void*, const void*, const void*, const float*, const void*, long, int, float*, St))        \
  X(mlb_layernorm_fwd, int, (void*, float*, float*, const void*, const void*, const void*, long, int, float, St))                              \
  X(mlb_layernorm_bwd2, int, (void*, void*, void*, int, const void*, const void*, const void*, const float*, const float*, long, int, float*, St)) \
  X(mlb_swiglu_fwd, int, (void*, const void*, long, int, St))                                                                                  \
  X(mlb_swiglu_fwd_fp8, int, (void*, uint8_t*, const void*, long, int, float, St))                                                             \
  X(mlb_swiglu_bwd, int, (void*, const void*, const void*, long, int, St))                                                                     \
  X(mlb_rope, int, (void*, const float*, const float*, long, int, int, int, float, St))                                                        \
  X(mlb_rope_copy, int, (void*, const void*, const float*, const float*, long, int, int, int, int, St))                                        \
  X(mlb_kv_group_sum, int, (void*, const void*, long, int, int, int, St))                                                                      \
  X(mlb_attn_fwd, int, (void*, float*, const void*, int, int, int, int, St))                                                                   \
  X(mlb_attn_bwd_scratch_bytes, long, (int, int, int, int))                                                                                    \
  X(mlb_attn_bwd, int, (void*, const void*, const void*, const void*, const float*, float*, void*, int, int, int, int, const float*, const float*, St)) \
  X(mlb_attn_bwd_have_delta, int, (void*, const void*, const void*, const void*, const float*, float*, void*, int, int, int, int, const float*, const float*, St)) \
  X(mlb_attn_bidir_fwd, int, (void*, float*, const void*, int, int, int, int, St))                                                             \
  X(mlb_attn_bidir_bwd, int, (void*, const void*, const void*, const void*, const float*, float*, int, int, int, int, St))                     \
  X(mlb_ce_mean, int, (float*, float*, float*, void*, const void*, const int*, long, int, St))                                                 \
  X(mlb_ce_fwd_bwd, int, (float*, void*, const int*, long, int, long, float, int, St))                                                         \
  X(mlb_scale_dev, int, (void*, const void*, const float*, long, St))                                                                          \
  X(mlb_embed_fwd, int, (void*, const void*, const int*, long, int, int, St))                                                                  \
  X(mlb_embed_bwd, int, (float*, const void*, const int*, long, int, int, int, int, St))                                                       \
  X(mlb_adamw, int, (float*, void*, const float*, float*, float*, long, float, float, float, float, float, float, float, float, const float*, St)) \
  X(mlb_sum_scale, int, (float*, const float*, long, float, St))
#define MLB_POINTER(name, ret, args) ret(*name) args = nullptr;
struct Entries { MLB_ENTRIES(MLB_POINTER) } K;

PyObject* address_type = nullptr;  // ops.native.Address
PyObject* settings = nullptr;      // the Python module whose variables FUSED_ATTN_BWD and FUSED_ATTN_BWD_MAX_SCRATCH bound attn_bwd's workspace

St stream() { return (St)c10::cuda::getCurrentCUDAStream().stream(); }
void check(int rc, const char* what) { TORCH_CHECK(rc == 0, what, " failed: code ", rc); }

// ------------------------------------------------------------------ which calls are plain
// Something is watching or rewriting the operators of this thread.  Asked first: a transform's tensors have no address to look at.
bool transformed() {
  if (torch::jit::tracer::isTracing() || c10::impl::TorchDispatchModeTLS::any_modes_set()) return true;
  const auto inc = c10::impl::tls_local_dispatch_key_set().included_;
  return inc.has(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) || inc.has(c10::DispatchKey::FuncTorchDynamicLayerBackMode);
}
bool aligned(const Tensor& t) { return ((uintptr_t)t.data_ptr() & 15) == 0; }
// A strided tensor of exactly this type on the current device, not empty, without a tangent
bool plain(PyObject* o, Tensor& t, at::ScalarType type, int dim) {
  if (!THPVariable_CheckExact(o)) return false;      // (a subclass overrides operators)
  t = THPVariable_Unpack(o);
  return t.is_cuda() && t.scalar_type() == type && t.layout() == at::kStrided && t.dim() == dim && t.numel() > 0 &&
         t.get_device() == c10::cuda::current_device() && !t.is_inference() && !t._fw_grad(0).defined();
}
bool plain_bf(PyObject* o, Tensor& t, int dim) { return plain(o, t, at::kBFloat16, dim) && aligned(t); }
bool int_arg(PyObject* o, long& v) {
  if (!PyLong_CheckExact(o)) return false;
  int over = 0;
  v = PyLong_AsLongAndOverflow(o, &over);
  return over == 0 && v >= 0 && v < (1L << 31);
}
bool wants_grad(std::initializer_list<const Tensor*> ts) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : ts)
    if (t->defined() && t->requires_grad()) return true;
  return false;
}
Maybe maybe(const Tensor& t) { return t.defined() ? Maybe(t) : Maybe(); }
Tensor f32(const Tensor& like, at::IntArrayRef sizes) { return at::empty(sizes, like.options().dtype(at::kFloat)); }
// A tensor as the kernels read it: rows behind each other, 16-byte aligned
Tensor rows_of(const Tensor& g) {
  const Tensor c = g.contiguous();
  return aligned(c) ? c : c.clone();
}

[[noreturn]] void refuse(const std::string& why) {
  pybind11::gil_scoped_acquire gil;
  PyErr_SetString(PyExc_AssertionError, why.c_str());
  python_error e;
  e.persist();      // (nodes run on threads of the autograd engine)
  throw e;
}
// A saved tensor: a hook may have handed back any other, and torch checks nothing of it.  Another device, type or size is refused
// here, in front of the node's launches, with the error of the entry points in ops/native.py; another layout, or an address off a
// 16-byte boundary, is copied into place.
Tensor unpacked(const Tensor& t, const Tensor& grad, at::ScalarType type, at::IntArrayRef sizes) {
  if (!t.defined() || t.device() != grad.device() || t.scalar_type() != type || t.layout() != at::kStrided || t.sizes() != sizes)
    refuse("saved tensor: need " + std::string(c10::toString(type)) + " of sizes " + c10::str(sizes) + " on " + grad.device().str() + ", not " +
           (t.defined() ? std::string(c10::toString(t.scalar_type())) + " of sizes " + c10::str(t.sizes()) + " on " + t.device().str() : "none"));
  return rows_of(t);
}
Tensor unpacked_bf(const Tensor& t, const Tensor& grad, at::IntArrayRef sizes) { return unpacked(t, grad, at::kBFloat16, sizes); }
Tensor unpacked_f32(const Tensor& t, const Tensor& grad, at::IntArrayRef sizes) { return unpacked(t, grad, at::kFloat, sizes); }

// ------------------------------------------------------------------ linear
Tensor linear_forward(const Tensor& x_, const Tensor& W_, const Tensor& b) {
  const Tensor x = x_.contiguous(), W = W_.contiguous();
  const int M = (int)x.size(0), Kd = (int)x.size(1), N = (int)W.size(0);
  Tensor out = at::empty({M, N}, x.options());
  const St st = stream();
  if (b.defined()) {
    const int rc = K.mlb_linear_fwd_posembed(out.data_ptr(), x.data_ptr(), W.data_ptr(), b.data_ptr(), 1, M, N, Kd, N, Kd, Kd, st);
    if (rc != -7) { check(rc, "linear_bias_fwd"); return out; }
  }
  check(K.mlb_linear_fwd(out.data_ptr(), x.data_ptr(), W.data_ptr(), M, N, Kd, N, Kd, Kd, st), "linear_fwd");
  if (b.defined()) out.add_(b);
  return out;
}
struct LinearFn : torch::autograd::Function<LinearFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& W, const Maybe& b) {
    ctx->save_for_backward({x, W});
    ctx->saved_data["inner"] = x.size(1);
    ctx->saved_data["bias"] = b.has_value();
    return linear_forward(x, W, b.value_or(Tensor()));
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto saved = ctx->get_saved_variables();
    const Tensor dout = g[0].contiguous();
    const int64_t rows = dout.size(0), cols = dout.size(1), inner = ctx->saved_data["inner"].toInt();
    const Tensor x = unpacked_bf(saved[0], dout, {rows, inner}), W = unpacked_bf(saved[1], dout, {cols, inner});
    const int M = (int)rows, Kd = (int)inner, N = (int)cols;
    const St st = stream();
    Tensor dx = at::empty({M, Kd}, x.options()), dW = at::empty({N, Kd}, W.options()), db;
    check(K.mlb_linear_dx(dx.data_ptr(), dout.data_ptr(), W.data_ptr(), M, N, Kd, Kd, N, Kd, st), "linear_dx");
    if (K.mlb_gemm_dw_direct(N, Kd, M)) {
      check(K.mlb_gemm(dW.data_ptr(), dout.data_ptr(), x.data_ptr(), N, Kd, M, Kd, N, Kd, 1, 1, 0, st), "gemm");
    } else {
      const Tensor acc = f32(W, {N, Kd});
      check(K.mlb_zero(acc.data_ptr(), acc.numel() * 4, st), "zero");
      check(K.mlb_linear_dw((float*)acc.data_ptr(), dout.data_ptr(), x.data_ptr(), M, N, Kd, Kd, N, Kd, st), "linear_dw");
      check(K.mlb_cast_f2b(dW.data_ptr(), (const float*)acc.data_ptr(), dW.numel(), 1.f, st), "cast_f2b");
    }
    if (ctx->saved_data["bias"].toBool()) {
      db = at::empty({N}, dout.options());
      const Tensor part = f32(dout, {(long)K.mlb_colsum_splits(M, N) * N});
      const int rc = K.mlb_colsum(db.data_ptr(), dout.data_ptr(), M, N, (float*)part.data_ptr(), st);
      if (rc == -7) db.copy_(dout.sum(0));
      else check(rc, "colsum");
    }
    return {dx, dW, db};
  }
};

// ------------------------------------------------------------------ norms (widths that the row kernels of the backward take)
bool norm_width(long C) { return C % 256 == 0 && C <= 2048; }
struct Normed { Tensor out, mean, rstd; };
Normed rmsnorm_forward(const Tensor& x, const Tensor& w, double eps) {
  const Tensor xc = x.contiguous();
  Normed r{at::empty_like(xc), Tensor(), f32(xc, {xc.size(0)})};
  check(K.mlb_rmsnorm_fwd(r.out.data_ptr(), (float*)r.rstd.data_ptr(), xc.data_ptr(), w.data_ptr(), xc.size(0), (int)xc.size(1), (float)eps, stream()), "rmsnorm_fwd");
  return r;
}
struct RMSNormFn : torch::autograd::Function<RMSNormFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, double eps) {
    const Normed r = rmsnorm_forward(x, w, eps);
    ctx->save_for_backward({x, w, r.rstd});
    return r.out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto saved = ctx->get_saved_variables();
    const Tensor dy = rows_of(g[0]);
    const int64_t rows = dy.size(0), C = dy.size(1);
    const Tensor x = unpacked_bf(saved[0], dy, {rows, C}), w = unpacked_bf(saved[1], dy, {C}), rstd = unpacked_f32(saved[2], dy, {rows});
    Tensor dx = at::empty_like(x), dw = at::empty_like(w);
    const Tensor part = f32(x, {K.mlb_rmsnorm_bwd_blocks(rows) * C});
    check(K.mlb_rmsnorm_bwd_cast(dx.data_ptr(), dw.data_ptr(), dy.data_ptr(), x.data_ptr(), w.data_ptr(), (const float*)rstd.data_ptr(), nullptr, rows, (int)C,
                                 (float*)part.data_ptr(), stream()), "rmsnorm_bwd_cast");
    return {dx, dw, Tensor()};
  }
};
Normed layernorm_forward(const Tensor& xc, const Tensor& w, const Tensor& b, double eps) {
  Normed r{at::empty_like(xc), f32(xc, {xc.size(0)}), f32(xc, {xc.size(0)})};
  check(K.mlb_layernorm_fwd(r.out.data_ptr(), (float*)r.mean.data_ptr(), (float*)r.rstd.data_ptr(), xc.data_ptr(), w.data_ptr(),
                            b.defined() ? b.data_ptr() : nullptr, xc.size(0), (int)xc.size(1), (float)eps, stream()), "layernorm_fwd");
  return r;
}
struct LayerNormFn : torch::autograd::Function<LayerNormFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const Maybe& b, double eps) {
    const Tensor xc = x.contiguous();
    const Normed r = layernorm_forward(xc, w, b.value_or(Tensor()), eps);
    ctx->save_for_backward({xc, w, r.mean, r.rstd});
    ctx->saved_data["bias"] = b.has_value();
    return r.out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto saved = ctx->get_saved_variables();
    const Tensor dy = rows_of(g[0]);
    const int64_t rows = dy.size(0), C = dy.size(1);
    const Tensor x = unpacked_bf(saved[0], dy, {rows, C}), w = unpacked_bf(saved[1], dy, {C}), mean = unpacked_f32(saved[2], dy, {rows}),
                 rstd = unpacked_f32(saved[3], dy, {rows});
    Tensor dx = at::empty_like(x), dw = at::empty_like(w), db;
    if (ctx->saved_data["bias"].toBool()) db = at::empty_like(w);
    const Tensor part = f32(x, {K.mlb_rmsnorm_bwd_blocks(rows) * 2 * C});
    check(K.mlb_layernorm_bwd2(dx.data_ptr(), dw.data_ptr(), db.defined() ? db.data_ptr() : nullptr, 1, dy.data_ptr(), x.data_ptr(), w.data_ptr(),
                               (const float*)mean.data_ptr(), (const float*)rstd.data_ptr(), rows, (int)C, (float*)part.data_ptr(), stream()),
          "layernorm_bwd_cast");
    return {dx, dw, db, Tensor()};
  }
};

// ------------------------------------------------------------------ SwiGLU
Tensor swiglu_forward(const Tensor& gu) {
  const Tensor g = gu.contiguous();
  const long rows = g.size(0), I = g.size(1) / 2;
  Tensor out = at::empty({rows, I}, g.options());
  check(K.mlb_swiglu_fwd(out.data_ptr(), g.data_ptr(), rows, (int)I, stream()), "swiglu_fwd");
  return out;
}
struct SwiGLUFn : torch::autograd::Function<SwiGLUFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& gu) {
    ctx->save_for_backward({gu});
    return swiglu_forward(gu);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const Tensor dout = rows_of(g[0]), gu = unpacked_bf(ctx->get_saved_variables()[0], dout, {dout.size(0), 2 * dout.size(1)});
    Tensor dgu = at::empty_like(gu);
    check(K.mlb_swiglu_bwd(dgu.data_ptr(), dout.data_ptr(), gu.data_ptr(), gu.size(0), (int)(gu.size(1) / 2), stream()), "swiglu_bwd");
    return {dgu};
  }
};

// ------------------------------------------------------------------ attention
struct Heads { int B, T, H, Hkv, hd; };
struct Attended { Tensor q, out, lse; };
Attended causal_forward(const Tensor& qkv, const Tensor& cos, const Tensor& sin, const Heads& h) {
  const St st = stream();
  const long n = (long)h.B * h.T;
  Attended r{at::empty({n, 3L * h.H * h.hd}, qkv.options()), at::empty({n, (long)h.H * h.hd}, qkv.options()), f32(qkv, {h.B, h.H, h.T})};
  check(K.mlb_rope_copy(r.q.data_ptr(), qkv.data_ptr(), (const float*)cos.data_ptr(), (const float*)sin.data_ptr(), n, h.T, h.H, h.Hkv, h.hd, st), "rope_copy");
  check(K.mlb_attn_fwd(r.out.data_ptr(), (float*)r.lse.data_ptr(), r.q.data_ptr(), h.B, h.T, h.H, h.hd, st), "attn_fwd");
  return r;
}
// May attn_bwd have a workspace of this size?  Asked in backward, as ops/native.py does: the variables may have been set since forward.
bool scratch_allowed(long bytes) {
  if (bytes <= 0) return false;
  pybind11::gil_scoped_acquire gil;
  const auto module = pybind11::reinterpret_borrow<pybind11::object>(settings);
  return pybind11::bool_(module.attr("FUSED_ATTN_BWD")) && pybind11::int_(bytes) <= module.attr("FUSED_ATTN_BWD_MAX_SCRATCH");
}
struct CausalFn : torch::autograd::Function<CausalFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& qkv, const Tensor& cos, const Tensor& sin, int64_t B, int64_t T, int64_t H, int64_t Hkv,
                        int64_t hd) {
    const Heads h{(int)B, (int)T, (int)H, (int)Hkv, (int)hd};
    const Attended r = causal_forward(qkv.contiguous(), cos, sin, h);
    ctx->save_for_backward({r.q, r.out, r.lse, cos, sin});
    ctx->saved_data["dims"] = std::vector<int64_t>{B, T, H, Hkv, hd, cos.size(0), sin.size(0)};
    ctx->saved_data["shape"] = qkv.sizes().vec();
    return r.out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto saved = ctx->get_saved_variables();
    const Tensor dout = rows_of(g[0]);
    const auto dims = ctx->saved_data["dims"].toIntVector();
    const Heads h{(int)dims[0], (int)dims[1], (int)dims[2], (int)dims[3], (int)dims[4]};
    const int64_t n = dims[0] * dims[1];
    const Tensor q = unpacked_bf(saved[0], dout, {n, 3 * dims[2] * dims[4]}), out = unpacked_bf(saved[1], dout, {n, dims[2] * dims[4]}),
                 lse = unpacked_f32(saved[2], dout, {dims[0], dims[2], dims[1]}), cos = unpacked_f32(saved[3], dout, {dims[5], dims[4] / 2}),
                 sin = unpacked_f32(saved[4], dout, {dims[6], dims[4] / 2});
    const St st = stream();
    Tensor dqkv = at::empty_like(q), part;
    const Tensor delta = f32(q, {n * h.H});
    const long bytes = h.hd == 64 ? K.mlb_attn_bwd_scratch_bytes(h.B, h.T, h.H, h.hd) : 0;
    if (scratch_allowed(bytes)) part = at::empty({bytes / 2}, q.options());
    const int rc = K.mlb_attn_bwd(dqkv.data_ptr(), dout.data_ptr(), q.data_ptr(), out.data_ptr(), (const float*)lse.data_ptr(), (float*)delta.data_ptr(),
                                  part.defined() ? part.data_ptr() : nullptr, h.B, h.T, h.H, h.hd, (const float*)cos.data_ptr(),
                                  (const float*)sin.data_ptr(), st);
    TORCH_CHECK(rc == 0 || rc == 1, "attn_bwd failed: code ", rc);
    if (rc == 0) check(K.mlb_rope(dqkv.data_ptr(), (const float*)cos.data_ptr(), (const float*)sin.data_ptr(), n, h.T, h.H, h.hd, -1.f, st), "rope_bwd");
    if (h.Hkv != h.H) {
      Tensor grouped = at::empty({n, (long)(h.H + 2 * h.Hkv) * h.hd}, q.options());
      check(K.mlb_kv_group_sum(grouped.data_ptr(), dqkv.data_ptr(), n, h.H, h.Hkv, h.hd, st), "kv_group_sum");
      dqkv = grouped;
    }
    return {dqkv.view(ctx->saved_data["shape"].toIntVector()), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};
struct Seen { Tensor q, out, lse; };
Seen bidir_forward(const Tensor& qkv, int64_t B, int64_t T, int64_t H, int64_t hd) {
  const Tensor q = qkv.contiguous();
  Seen r{q, at::empty({B * T, H * hd}, q.options()), f32(q, {B, H, T})};
  check(K.mlb_attn_bidir_fwd(r.out.data_ptr(), (float*)r.lse.data_ptr(), q.data_ptr(), (int)B, (int)T, (int)H, (int)hd, stream()), "attn_bidir_fwd");
  return r;
}
struct BidirFn : torch::autograd::Function<BidirFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& qkv, int64_t B, int64_t T, int64_t H, int64_t hd) {
    const Seen r = bidir_forward(qkv, B, T, H, hd);
    ctx->save_for_backward({r.q, r.out, r.lse});
    ctx->saved_data["dims"] = std::vector<int64_t>{B, T, H, hd};
    return r.out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto saved = ctx->get_saved_variables();
    const Tensor dout = rows_of(g[0]);
    const auto d = ctx->saved_data["dims"].toIntVector();
    const Tensor q = unpacked_bf(saved[0], dout, {d[0] * d[1], 3 * d[2] * d[3]}), out = unpacked_bf(saved[1], dout, {d[0] * d[1], d[2] * d[3]}),
                 lse = unpacked_f32(saved[2], dout, {d[0], d[2], d[1]});
    Tensor dqkv = at::empty_like(q);
    const Tensor delta = f32(q, {d[0] * d[1] * d[2]});
    check(K.mlb_attn_bidir_bwd(dqkv.data_ptr(), dout.data_ptr(), q.data_ptr(), out.data_ptr(), (const float*)lse.data_ptr(), (float*)delta.data_ptr(), (int)d[0],
                               (int)d[1], (int)d[2], (int)d[3], stream()), "attn_bidir_bwd");
    return {dqkv, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------ cross-entropy
struct Crossed { Tensor loss, grad; };
Crossed ce_forward(const Tensor& z, const Tensor& tgt, bool grad) {
  const long rows = z.size(0), V = z.size(1);
  Crossed r{f32(z, {}), grad ? at::empty_like(z) : Tensor()};
  const Tensor losses = f32(z, {rows}), stats = f32(z, {2});
  check(K.mlb_ce_mean((float*)r.loss.data_ptr(), (float*)losses.data_ptr(), (float*)stats.data_ptr(), grad ? r.grad.data_ptr() : nullptr, z.data_ptr(),
                      (const int*)tgt.data_ptr(), rows, (int)V, stream()), "ce_mean");
  return r;
}
struct CrossEntropyFn : torch::autograd::Function<CrossEntropyFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& logits, const Tensor& tgt) {
    const Crossed r = ce_forward(logits.contiguous(), tgt, true);
    ctx->save_for_backward({r.grad});
    ctx->saved_data["shape"] = logits.sizes().vec();
    ctx->saved_data["shared"] = at::SavedTensorDefaultHooks::get_hooks().has_value();
    ctx->saved_data["capture"] = (int64_t)K.mlb_capture_id(stream());
    return r.loss;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const Tensor d = unpacked_bf(ctx->get_saved_variables()[0], g[0], ctx->saved_data["shape"].toIntVector());
    // The last use of the saved gradient: scaled in place and handed out, and not even read when the factor is one.  Not when the graph
    // is kept for another pass, when a pack hook may hold the tensor itself, or when one of forward and backward is captured without the
    // other: then a replay of the backward is another pass.
    const bool last = !ctx->saved_data["shared"].toBool() && !torch::autograd::get_current_graph_task_keep_graph() &&
                      ctx->saved_data["capture"].toInt() == (int64_t)K.mlb_capture_id(stream());
    Tensor out = last ? d : at::empty_like(d);
    const Tensor s = g[0].to(at::kFloat).contiguous();
    check(K.mlb_scale_dev(out.data_ptr(), d.data_ptr(), (const float*)s.data_ptr(), out.numel(), stream()), "scale_dev");
    return {out, Tensor()};
  }
};

// ------------------------------------------------------------------ Python entry points
PyObject* declined() { Py_RETURN_NOTIMPLEMENTED; }
template <typename F>
PyObject* released(F&& f) {      // the launch without the interpreter lock
  Tensor out;
  {
    pybind11::gil_scoped_release no_gil;
    out = f();
  }
  return THPVariable_Wrap(std::move(out));
}

PyObject* py_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Tensor x, W, b;
  if (n != 3 || transformed() || !plain_bf(a[0], x, 2) || !plain_bf(a[1], W, 2) || x.size(1) != W.size(1)) return declined();
  if (a[2] != Py_None && (!plain_bf(a[2], b, 1) || b.size(0) != W.size(0) || !b.is_contiguous())) return declined();
  return released([&] { return wants_grad({&x, &W, &b}) ? LinearFn::apply(x, W, maybe(b)) : linear_forward(x, W, b); });
  END_HANDLE_TH_ERRORS
}
PyObject* py_rmsnorm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Tensor x, w;
  if (n != 3 || transformed() || !plain_bf(a[0], x, 2) || !plain_bf(a[1], w, 1) || w.size(0) != x.size(1) || !w.is_contiguous() || !norm_width(x.size(1)) ||
      !PyFloat_CheckExact(a[2]))
    return declined();
  const double eps = PyFloat_AS_DOUBLE(a[2]);
  return released([&] { return wants_grad({&x, &w}) ? RMSNormFn::apply(x, w, eps) : rmsnorm_forward(x, w, eps).out; });
  END_HANDLE_TH_ERRORS
}
PyObject* py_layer_norm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Tensor x, w, b;
  if (n != 4 || transformed() || !plain_bf(a[0], x, 2) || !plain_bf(a[1], w, 1) || w.size(0) != x.size(1) || !w.is_contiguous() || !norm_width(x.size(1)) ||
      !PyFloat_CheckExact(a[3]))
    return declined();
  if (a[2] != Py_None && (!plain_bf(a[2], b, 1) || b.size(0) != x.size(1) || !b.is_contiguous())) return declined();
  const double eps = PyFloat_AS_DOUBLE(a[3]);
  return released([&] { return wants_grad({&x, &w, &b}) ? LayerNormFn::apply(x, w, maybe(b), eps) : layernorm_forward(x.contiguous(), w, b, eps).out; });
  END_HANDLE_TH_ERRORS
}
PyObject* py_swiglu(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Tensor gu;
  if (n != 1 || transformed() || !plain_bf(a[0], gu, 2) || gu.size(1) % 16 != 0) return declined();
  return released([&] { return wants_grad({&gu}) ? SwiGLUFn::apply(gu) : swiglu_forward(gu); });
  END_HANDLE_TH_ERRORS
}
// (qkv, cos, sin, B, T, H, hd, Hkv or None)
PyObject* py_rope_causal_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Tensor qkv, cos, sin;
  long B, T, H, hd, Hkv;
  if (n != 8 || transformed() || !plain_bf(a[0], qkv, 2) || !plain(a[1], cos, at::kFloat, 2) || !plain(a[2], sin, at::kFloat, 2) || !int_arg(a[3], B) || !int_arg(a[4], T) ||
      !int_arg(a[5], H) || !int_arg(a[6], hd))
    return declined();
  if (a[7] == Py_None) Hkv = H;
  else if (!int_arg(a[7], Hkv)) return declined();
  if (B < 1 || T < 1 || H < 1 || Hkv < 1 || H % Hkv != 0 || hd % 16 != 0 || hd > 128 || hd < 16) return declined();
  const long rows = B * T;
  if (rows >= (1L << 31) || qkv.size(0) != rows || qkv.size(1) != (H + 2 * Hkv) * hd || rows * 3 * H * (hd / 16) >= (1L << 31) || !cos.is_contiguous() ||
      !sin.is_contiguous() || !aligned(cos) || !aligned(sin) || cos.size(0) < T || sin.size(0) < T || cos.size(1) != hd / 2 || sin.size(1) != hd / 2 ||
      cos.requires_grad() || sin.requires_grad())
    return declined();
  return released([&] {
    if (wants_grad({&qkv})) return CausalFn::apply(qkv, cos, sin, B, T, H, Hkv, hd);
    return causal_forward(qkv.contiguous(), cos, sin, Heads{(int)B, (int)T, (int)H, (int)Hkv, (int)hd}).out;
  });
  END_HANDLE_TH_ERRORS
}
PyObject* py_bidir_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Tensor qkv;
  long B, T, H, hd;
  if (n != 5 || transformed() || !plain_bf(a[0], qkv, 2) || !int_arg(a[1], B) || !int_arg(a[2], T) || !int_arg(a[3], H) || !int_arg(a[4], hd)) return declined();
  if (B < 1 || T < 1 || H < 1 || hd % 16 != 0 || hd > 128 || hd < 16 || qkv.size(0) != B * T || qkv.size(1) != 3 * H * hd) return declined();
  return released([&] { return wants_grad({&qkv}) ? BidirFn::apply(qkv, B, T, H, hd) : bidir_forward(qkv, B, T, H, hd).out; });
  END_HANDLE_TH_ERRORS
}
PyObject* py_cross_entropy(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Tensor z, tgt;
  if (n != 2 || transformed() || !plain_bf(a[0], z, 2) || !plain(a[1], tgt, at::kInt, 1) || tgt.size(0) != z.size(0) || !tgt.is_contiguous()) return declined();
  return released([&] { return wants_grad({&z}) ? CrossEntropyFn::apply(z, tgt) : ce_forward(z.contiguous(), tgt, false).loss; });
  END_HANDLE_TH_ERRORS
}

// ------------------------------------------------------------------ the entry points themselves
// Arguments by the C type of the parameter: a bf16 (void*), fp32, int32 or byte tensor, which has to be contiguous and on a GPU, or an Address
// of ops/native.py (a plain number, which may be anything, is refused); numbers.  The stream comes last and is the current one.
[[noreturn]] void bad_tensor(const char* want) {
  PyErr_Format(PyExc_AssertionError, "tensor: need contiguous CUDA %s", want);
  throw python_error();
}
template <typename P>
P pointer_arg(PyObject* o, at::ScalarType type, const char* want) {
  if (THPVariable_Check(o)) {
    const Tensor& t = THPVariable_Unpack(o);
    if (!t.is_cuda() || t.scalar_type() != type || !t.is_contiguous()) bad_tensor(want);
    return (P)t.data_ptr();
  }
  if ((PyObject*)Py_TYPE(o) != address_type) bad_tensor(want);
  const P p = (P)PyLong_AsVoidPtr(o);
  if (!p && PyErr_Occurred()) throw python_error();
  return p;
}
template <typename T> struct Arg;
#define MLB_POINTER_ARG(C, type, want) \
  template <> struct Arg<C*> { static C* get(PyObject* o) { return pointer_arg<C*>(o, type, want); } }; \
  template <> struct Arg<const C*> { static const C* get(PyObject* o) { return pointer_arg<const C*>(o, type, want); } };
MLB_POINTER_ARG(void, at::kBFloat16, "bf16")
MLB_POINTER_ARG(float, at::kFloat, "fp32")
MLB_POINTER_ARG(int, at::kInt, "int32")
MLB_POINTER_ARG(uint8_t, at::kByte, "uint8 (E4M3 bytes)")
long long_arg(PyObject* o) {
  const long v = PyLong_AsLong(o);
  if (v == -1 && PyErr_Occurred()) throw python_error();
  return v;
}
template <> struct Arg<long> { static long get(PyObject* o) { return long_arg(o); } };
template <> struct Arg<int> { static int get(PyObject* o) { return (int)long_arg(o); } };
template <> struct Arg<float> {
  static float get(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw python_error();
    return (float)v;
  }
};
// An entry point's parameters, a letter each (see _KINDS in ops/native.py)
template <typename T> constexpr char kind_of() {
  using P = std::remove_cv_t<std::remove_pointer_t<T>>;
  if constexpr (std::is_same_v<T, St>) return 's';
  else if constexpr (std::is_pointer_v<T>) return std::is_same_v<P, void> ? 'b' : std::is_same_v<P, float> ? 'f' : std::is_same_v<P, int> ? 'i' : 'u';
  else return std::is_same_v<T, float> ? 'd' : std::is_same_v<T, long> ? 'l' : 'n';
}
template <typename R, typename... A> std::string kinds_of(R (*)(A...)) { return {kind_of<A>()...}; }
template <typename R, typename... A, size_t... I>
PyObject* call_entry(R (*f)(A...), PyObject* const* a, Py_ssize_t n, std::index_sequence<I...>) {
  constexpr bool streamed = std::is_same_v<std::tuple_element_t<sizeof...(A) - 1, std::tuple<A...>>, St>;
  if (n != (Py_ssize_t)sizeof...(A) - streamed) { PyErr_Format(PyExc_TypeError, "%zd arguments, not %zd", n, (Py_ssize_t)sizeof...(A) - streamed); return nullptr; }
  auto one = [&](auto tag, size_t i) {
    using T = typename decltype(tag)::type;
    if constexpr (std::is_same_v<T, St>) return stream();
    else return Arg<T>::get(a[i]);
  };
  const std::tuple<A...> args{one(std::common_type<A>{}, I)...};
  R r;
  Py_BEGIN_ALLOW_THREADS
  r = std::apply(f, args);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong((long)r);
}
template <typename F> struct typed_call;
template <typename R, typename... A> struct typed_call<R(A...)> {
  static PyObject* go(R (*f)(A...), PyObject* const* a, Py_ssize_t n) { return call_entry(f, a, n, std::index_sequence_for<A...>{}); }
};
#define MLB_CALL(name, ret, args)                                              \
  PyObject* call_##name(PyObject*, PyObject* const* a, Py_ssize_t n) {         \
    HANDLE_TH_ERRORS                                                           \
    return typed_call<ret args>::go(K.name, a, n);                             \
    END_HANDLE_TH_ERRORS                                                       \
  }
MLB_ENTRIES(MLB_CALL)

// bind(path, settings): the kernel library whose functions are called, the module with the variables above
PyObject* py_bind(PyObject*, PyObject* args) {
  HANDLE_TH_ERRORS
  const char* p = nullptr;
  PyObject* module = nullptr;
  if (!PyArg_ParseTuple(args, "sO", &p, &module)) return nullptr;
  void* h = dlopen(p, RTLD_NOW);
  TORCH_CHECK(h != nullptr, "cannot load ", p, ": ", dlerror());
#define MLB_LOOKUP(name, ret, args)                                  \
  K.name = (ret(*) args)dlsym(h, #name);                             \
  TORCH_CHECK(K.name != nullptr, p, " has no function " #name);
  MLB_ENTRIES(MLB_LOOKUP)
  PyObject* address = PyObject_GetAttrString(module, "Address");
  if (!address) return nullptr;
  Py_XDECREF(address_type);
  address_type = address;
  Py_INCREF(module);
  Py_XDECREF(settings);
  settings = module;
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// signatures(): every entry point's parameters by name
PyObject* py_signatures(PyObject*, PyObject*) {
  HANDLE_TH_ERRORS
  pybind11::dict d;
#define MLB_KINDS(name, ret, args) d[#name] = kinds_of(K.name);
  MLB_ENTRIES(MLB_KINDS)
  return d.release().ptr();
  END_HANDLE_TH_ERRORS
}

#define MLB_FAST(name) {#name, (PyCFunction)(void (*)(void))py_##name, METH_FASTCALL, nullptr}
#define MLB_METHOD(name, ret, args) {#name, (PyCFunction)(void (*)(void))call_##name, METH_FASTCALL, nullptr},
PyMethodDef methods[] = {MLB_FAST(linear), MLB_FAST(rmsnorm), MLB_FAST(layer_norm), MLB_FAST(swiglu), MLB_FAST(rope_causal_attention), MLB_FAST(bidir_attention),
                         MLB_FAST(cross_entropy), MLB_ENTRIES(MLB_METHOD) {"bind", py_bind, METH_VARARGS, nullptr}, {"signatures", py_signatures, METH_NOARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "mlb_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_mlb_torch(void) { return PyModule_Create(&module); }
