// The operators as torch functions: allocation, autograd and autocast in native code over the C ABI of the library.
//
// A small call is bound by the host: with the argument structures filled through ctypes and the autograd functions in
// Python, a forward + backward pair of one operator kept one core busy for 180 to 330 us (attention to LayernormLinear
// under autocast) while the kernels of the single track take 60 to 70 us.  Here the same pair costs a few microseconds
// per call plus the launches, and the backward runs on the autograd thread without the interpreter lock.
//
// The library is opened by path at import (load()), so this module carries no link-time dependency on it and the
// library itself stays free of torch.
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/extension.h>
#include <ATen/FuncTorchTLS.h>
#include <ATen/autocast_mode.h>
#include <c10/core/AutogradState.h>

#include <array>
#include <optional>
#include <tuple>
#include <vector>

#include "../../include/megafold_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::tensor_list;
using torch::autograd::Variable;
using OptTensor = std::optional<Tensor>;

#define MF_ENTRY(name) decltype(&::name) name = nullptr
struct Api {
  MF_ENTRY(mf_evo_fwd_workspace_bytes);
  MF_ENTRY(mf_evo_fwd_with_workspace);
  MF_ENTRY(mf_evo_bwd_workspace_bytes);
  MF_ENTRY(mf_evo_bwd);
  MF_ENTRY(mf_lnl_fwd);
  MF_ENTRY(mf_lnl_bwd_workspace_bytes);
  MF_ENTRY(mf_lnl_bwd_add);
  MF_ENTRY(mf_gate_fwd);
  MF_ENTRY(mf_gate_bwd);
  MF_ENTRY(mf_bias_layout);
  MF_ENTRY(mf_evo_fwd_laid_out);
  MF_ENTRY(mf_evo_bwd_laid_out);
  MF_ENTRY(mf_swiglu_fwd);
  MF_ENTRY(mf_swiglu_bwd);
  MF_ENTRY(mf_transition_fwd_workspace_bytes);
  MF_ENTRY(mf_transition_fwd);
  MF_ENTRY(mf_transition_bwd_workspace_bytes);
  MF_ENTRY(mf_transition_bwd);
  MF_ENTRY(mf_cast_batch);
  MF_ENTRY(mf_last_error_string);
} api;
#undef MF_ENTRY

void load(const std::string& path) {
  void* h = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  TORCH_CHECK(h, "megafold_b200: cannot open ", path, ": ", dlerror());
  auto get = [&](const char* name) {
    void* p = dlsym(h, name);
    TORCH_CHECK(p, "megafold_b200: ", path, " does not export ", name);
    return p;
  };
#define MF_LOAD(name) api.name = reinterpret_cast<decltype(api.name)>(get(#name))
  MF_LOAD(mf_evo_fwd_workspace_bytes); MF_LOAD(mf_evo_fwd_with_workspace); MF_LOAD(mf_evo_bwd_workspace_bytes); MF_LOAD(mf_evo_bwd);
  MF_LOAD(mf_lnl_fwd); MF_LOAD(mf_lnl_bwd_workspace_bytes); MF_LOAD(mf_lnl_bwd_add);
  MF_LOAD(mf_gate_fwd); MF_LOAD(mf_gate_bwd); MF_LOAD(mf_bias_layout); MF_LOAD(mf_evo_fwd_laid_out); MF_LOAD(mf_evo_bwd_laid_out);
  MF_LOAD(mf_swiglu_fwd); MF_LOAD(mf_swiglu_bwd);
  MF_LOAD(mf_transition_fwd_workspace_bytes); MF_LOAD(mf_transition_fwd);
  MF_LOAD(mf_transition_bwd_workspace_bytes); MF_LOAD(mf_transition_bwd);
  MF_LOAD(mf_cast_batch); MF_LOAD(mf_last_error_string);
#undef MF_LOAD
}

void check(int status, const char* what) {
  TORCH_CHECK(status == MF_OK, "megafold_b200 ", what, " failed (status ", status, "): ", api.mf_last_error_string());
}

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return MF_F32;
    case at::kBFloat16: return MF_BF16;
    case at::kHalf: return MF_F16;
    case at::kBool: case at::kByte: return MF_U8;
    default: TORCH_CHECK_TYPE(false, "megafold_b200: unsupported dtype ", t);
  }
}

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

std::string shape(const Tensor& t) {
  std::string s = "(";
  for (int64_t i = 0; i < t.dim(); ++i) s += (i ? ", " : "") + std::to_string(t.size(i));
  return s + ")";
}

void require_cuda(std::initializer_list<const Tensor*> ts) {
  for (const Tensor* t : ts)
    TORCH_CHECK(!t->defined() || t->is_cuda(),
                "megafold_b200 operators run on CUDA tensors only (there is no CPU path); got a tensor on ", t->device());
}

// Forward-mode differentiation and torch.func transforms are refused by the autograd functions, which have no rule for them; a
// call that goes past these because gradients are off must not drop a tangent either.
void refuse_transforms(std::initializer_list<const Tensor*> ts) {
  if (const auto& tls = at::functorch::functorchTLSAccessor()) tls->checkSupportsCppAutogradFunction();
  if (!c10::AutogradState::get_tls_state().get_fw_grad_mode()) return;
  for (const Tensor* t : ts)
    TORCH_CHECK_NOT_IMPLEMENTED(!t->defined() || !t->unsafeGetTensorImpl()->_fw_grad(0, *t).defined(),
                                "megafold_b200 operators do not support forward-mode differentiation");
}

Tensor workspace(size_t bytes, const Tensor& like) {
  return at::empty({(int64_t)(bytes < 256 ? 256 : bytes)}, like.options().dtype(at::kByte));
}
Tensor empty_f32(at::IntArrayRef sizes, const Tensor& like) { return at::empty(sizes, like.options().dtype(at::kFloat)); }
void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
Tensor or_none(const OptTensor& t) { return t ? *t : Tensor(); }

// The values themselves where a negation is still pending (the imaginary part of a conjugate, say): kernels read memory.
Tensor plain(const Tensor& t) { return t.defined() && t.is_neg() ? t.resolve_neg() : t; }
const Tensor& plain(const Tensor& t, Tensor& hold) { return t.defined() && t.is_neg() ? (hold = t.resolve_neg()) : t; }      // no copy of the handle

// ---- conversions -------------------------------------------------------------------------------------------------
// Brings each tensor to its wanted type (and to contiguous memory), all of them in one launch: mixed-precision calls
// convert four to six small parameters at once, where a launch each costs more than the conversion.
struct Cast { Tensor* t; at::ScalarType to; };
void cast_batch(std::initializer_list<Cast> list) {
  mf_cast_item items[MF_CAST_MAX];
  Tensor keep[MF_CAST_MAX];
  int n = 0;
  Tensor any;
  for (const Cast& c : list) {
    if (!c.t->defined()) continue;
    if (c.t->is_neg()) *c.t = c.t->resolve_neg();
    if (!c.t->is_contiguous()) *c.t = c.t->contiguous();
    if (c.t->scalar_type() == c.to) continue;
    const auto from = c.t->scalar_type();
    const bool plain = from == at::kFloat || from == at::kBFloat16 || from == at::kHalf;
    if (!plain || n == MF_CAST_MAX) { *c.t = c.t->to(c.to); continue; }
    if (c.t->numel() == 0) { *c.t = at::empty(c.t->sizes(), c.t->options().dtype(c.to)); continue; }
    Tensor out = at::empty(c.t->sizes(), c.t->options().dtype(c.to));
    items[n] = mf_cast_item{c.t->data_ptr(), out.data_ptr(), c.t->numel(), dtype_code(from), dtype_code(c.to)};
    keep[n++] = *c.t;          // the source must outlive the launch
    any = out;
    *c.t = out;
  }
  if (n) check(api.mf_cast_batch(items, n, stream_of(any)), "mf_cast_batch");
}

// What torch.amp.custom_fwd(cast_inputs=torch.bfloat16) does to one argument while autocast is on.
bool autocast_on() { return at::autocast::is_autocast_enabled(at::kCUDA); }
at::ScalarType amp_type(const Tensor& t, bool on) {
  return on && t.defined() && t.is_cuda() && t.is_floating_point() && t.scalar_type() != at::kDouble ? at::kBFloat16 : t.scalar_type();
}

// ---- attention -----------------------------------------------------------------------------------------------------
std::array<int64_t, 5> check_shapes(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& mask, const OptTensor& bias) {
  TORCH_CHECK_VALUE(q.dim() == 5, "Q must be [B, N_seq, N_res, Head, Dim], got ", shape(q));
  TORCH_CHECK_VALUE(k.sizes() == q.sizes() && v.sizes() == q.sizes(), "Q, K, V shapes differ: ", shape(q), " ", shape(k), " ", shape(v));
  TORCH_CHECK_TYPE(q.scalar_type() == k.scalar_type() && q.scalar_type() == v.scalar_type(), "Q, K, V must share a dtype");
  TORCH_CHECK_VALUE(mask && mask->defined() && bias && bias->defined(), "res_mask and pair_bias are mandatory");
  const int64_t B = q.size(0), N = q.size(1), L = q.size(2), H = q.size(3), D = q.size(4);
  TORCH_CHECK_VALUE(bias->dim() == 5 && bias->size(1) == 1 && bias->size(2) == H && bias->size(3) == L && bias->size(4) == L &&
                        (bias->size(0) == 1 || bias->size(0) == B),
                    "pair_bias must be [B, 1, Head, N_res, N_res], got ", shape(*bias));
  TORCH_CHECK_VALUE(mask->dim() == 5 && mask->size(2) == 1 && mask->size(3) == 1 && mask->size(4) == L &&
                        (mask->size(0) == 1 || mask->size(0) == B) && (mask->size(1) == 1 || mask->size(1) == N),
                    "res_mask must be [B, N_seq, 1, 1, N_res], got ", shape(*mask));
  return {B, N, L, H, D};
}

template <typename A>
void fill_common(A& a, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& mask, const Tensor& bias, int64_t flags) {
  a.B = (int32_t)q.size(0); a.N = (int32_t)q.size(1); a.L = (int32_t)q.size(2); a.H = (int32_t)q.size(3); a.D = (int32_t)q.size(4);
  a.dtype = dtype_code(q.scalar_type()); a.bias_dtype = dtype_code(bias.scalar_type()); a.mask_dtype = dtype_code(mask.scalar_type());
  a.flags = (uint32_t)flags;
  a.q = q.data_ptr(); a.k = k.data_ptr(); a.v = v.data_ptr();
  for (int i = 0; i < 5; ++i) { a.q_strides[i] = q.stride(i); a.k_strides[i] = k.stride(i); a.v_strides[i] = v.stride(i); }
  // an extent of one that stands for B or N is read again for each of them
  auto step = [](const Tensor& t, int dim, int64_t want) { return t.size(dim) == 1 && want != 1 ? (int64_t)0 : t.stride(dim); };
  a.mask = mask.data_ptr();
  a.mask_strides[0] = step(mask, 0, a.B); a.mask_strides[1] = step(mask, 1, a.N); a.mask_strides[2] = mask.stride(4);
  a.bias = bias.data_ptr();
  a.bias_strides[0] = step(bias, 0, a.B); a.bias_strides[1] = bias.stride(2); a.bias_strides[2] = bias.stride(3); a.bias_strides[3] = bias.stride(4);
}

std::tuple<Tensor, Tensor> evo_forward(const Tensor& q_, const Tensor& k_, const Tensor& v_, const OptTensor& mask_, const OptTensor& bias_, int64_t flags) {
  const Tensor mask_t = or_none(mask_), bias_t = or_none(bias_);
  Tensor hold[5];
  const Tensor &q = plain(q_, hold[0]), &k = plain(k_, hold[1]), &v = plain(v_, hold[2]), &mask = plain(mask_t, hold[3]), &bias = plain(bias_t, hold[4]);
  require_cuda({&q, &k, &v, &mask, &bias});
  const auto s = check_shapes(q, k, v, mask_, bias_);
  const c10::cuda::CUDAGuard guard(q.device());
  Tensor o = at::empty({s[0], s[1], s[2], s[3], s[4]}, q.options());
  Tensor lse = empty_f32({s[0], s[1], s[3], s[2]}, q);
  mf_evo_fwd_args a{};
  fill_common(a, q, k, v, mask, bias, flags);
  a.o = o.data_ptr(); a.lse = lse.data_ptr<float>();
  Tensor ws;
  const size_t need = api.mf_evo_fwd_workspace_bytes(&a);
  if (need) ws = workspace(need, q);
  check(api.mf_evo_fwd_with_workspace(&a, ptr(ws), need, stream_of(q)), "mf_evo_fwd");
  return {o, lse};
}

std::tuple<Tensor, Tensor, Tensor, Tensor> evo_backward(const Tensor& d_o_, const Tensor& q_, const Tensor& k_, const Tensor& v_, const OptTensor& mask_,
                                                        const OptTensor& bias_, const Tensor& o_, const Tensor& lse, int64_t flags, int64_t event) {
  const Tensor mask_t = or_none(mask_), bias_t = or_none(bias_);
  Tensor hold[5];
  const Tensor &q = plain(q_, hold[0]), &k = plain(k_, hold[1]), &v = plain(v_, hold[2]), &mask = plain(mask_t, hold[3]), &bias = plain(bias_t, hold[4]);
  require_cuda({&d_o_, &q, &k, &v, &mask, &bias, &o_, &lse});
  const auto s = check_shapes(q, k, v, mask_, bias_);
  const c10::cuda::CUDAGuard guard(q.device());
  const Tensor d_o = plain(d_o_).contiguous(), o = plain(o_).contiguous();
  Tensor dq = at::empty({s[0], s[1], s[2], s[3], s[4]}, q.options()), dk = at::empty_like(dq), dv = at::empty_like(dq);
  const auto bt = bias.scalar_type();
  Tensor d_bias = at::empty({s[0], 1, s[3], s[2], s[2]}, q.options().dtype(bt == q.scalar_type() ? bt : at::kFloat));
  mf_evo_bwd_args a{};
  fill_common(a, q, k, v, mask, bias, flags);
  a.dbias_dtype = dtype_code(d_bias.scalar_type());
  a.o = o.data_ptr(); a.d_o = d_o.data_ptr(); a.lse = lse.data_ptr<float>();
  a.dq = dq.data_ptr(); a.dk = dk.data_ptr(); a.dv = dv.data_ptr(); a.d_bias = d_bias.data_ptr();
  a.dbias_ready_event = reinterpret_cast<void*>(event);
  Tensor ws = workspace(api.mf_evo_bwd_workspace_bytes(&a), q);
  a.workspace = ws.data_ptr(); a.workspace_bytes = (size_t)ws.numel();
  check(api.mf_evo_bwd(&a, stream_of(q)), "mf_evo_bwd");
  if (bias.size(0) != s[0]) d_bias = d_bias.sum(0, /*keepdim=*/true);      // bias broadcast over the batch
  if (d_bias.scalar_type() != bt) d_bias = d_bias.to(bt);
  return {dq, dk, dv, d_bias};
}

struct EvoFn : torch::autograd::Function<EvoFn> {
  static Variable forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& mask, const Tensor& bias) {
    auto [o, lse] = evo_forward(q, k, v, mask, bias, 0);
    ctx->save_for_backward({q, k, v, mask, bias, o, lse});
    return o;
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list g) {
    at::NoGradGuard no_grad;
    const auto s = ctx->get_saved_variables();
    auto [dq, dk, dv, db] = evo_backward(g[0], s[0], s[1], s[2], s[3], s[4], s[5], s[6], 0, 0);
    return {dq, dk, dv, Tensor(), db};
  }
};

Tensor evo_attention(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& mask, const OptTensor& bias) {
  const Tensor m = or_none(mask), b = or_none(bias);
  if (!at::GradMode::is_enabled()) {
    refuse_transforms({&q, &k, &v, &m, &b});
    return std::get<0>(evo_forward(q, k, v, mask, bias, 0));
  }
  require_cuda({&q, &k, &v, &m, &b});
  check_shapes(q, k, v, mask, bias);
  return EvoFn::apply(q, k, v, m, b);
}

// ---- LayernormLinear --------------------------------------------------------------------------------------------------
int64_t rows_of(const Tensor& x) { return x.size(-1) ? x.numel() / x.size(-1) : 0; }

// x, w and the vectors share one type and are contiguous
std::tuple<Tensor, Tensor, Tensor> lnl_fwd_raw(const Tensor& x, const Tensor& w, const Tensor& b, const Tensor& lw, const Tensor& lb, double eps, int64_t flags) {
  const int64_t K = x.size(-1), M = rows_of(x), N = w.size(1);
  auto sizes = x.sizes().vec();
  sizes.back() = N;
  Tensor y = at::empty(sizes, x.options()), mean = empty_f32({M}, x), rstd = empty_f32({M}, x);
  mf_lnl_fwd_args a{};
  a.M = M; a.K = (int32_t)K; a.N = (int32_t)N; a.dtype = dtype_code(x.scalar_type()); a.flags = (uint32_t)flags; a.eps = (float)eps;
  a.x = x.data_ptr(); a.ln_w = lw.data_ptr(); a.ln_b = ptr(lb); a.w = w.data_ptr(); a.b = ptr(b);
  a.y = y.data_ptr(); a.mean = mean.data_ptr<float>(); a.rstd = rstd.data_ptr<float>();
  check(api.mf_lnl_fwd(&a, stream_of(x)), "mf_lnl_fwd");
  return {y, mean, rstd};
}

// (dx, dw, db, d_ln_w, d_ln_b), parameter gradients fp32
std::array<Tensor, 5> lnl_bwd_raw(const Tensor& dy, const Tensor& x, const Tensor& w, const Tensor& lw, const Tensor& lb, const Tensor& mean,
                                  const Tensor& rstd, bool has_linear_bias, int64_t flags, const Tensor* add1 = nullptr, const Tensor* add2 = nullptr) {
  const int64_t K = x.size(-1), M = rows_of(x), N = w.size(1);
  Tensor dx = at::empty(x.sizes(), x.options());
  Tensor dw = empty_f32({K, N}, x), dlw = empty_f32({K}, x), dlb, db;
  if (lb.defined()) dlb = empty_f32({K}, x);
  if (has_linear_bias) db = empty_f32({N}, x);
  mf_lnl_bwd_args a{};
  a.M = M; a.K = (int32_t)K; a.N = (int32_t)N; a.dtype = dtype_code(x.scalar_type()); a.flags = (uint32_t)flags;
  a.x = x.data_ptr(); a.ln_w = lw.data_ptr(); a.ln_b = ptr(lb); a.w = w.data_ptr(); a.dy = dy.data_ptr();
  a.mean = mean.data_ptr<float>(); a.rstd = rstd.data_ptr<float>();
  a.dx = dx.data_ptr(); a.dw = dw.data_ptr<float>(); a.db = static_cast<float*>(ptr(db)); a.d_ln_w = dlw.data_ptr<float>();
  a.d_ln_b = static_cast<float*>(ptr(dlb));
  Tensor ws = workspace(api.mf_lnl_bwd_workspace_bytes(&a), x);
  a.workspace = ws.data_ptr(); a.workspace_bytes = (size_t)ws.numel();
  check(api.mf_lnl_bwd_add(&a, add1 ? add1->data_ptr() : nullptr, add2 ? add2->data_ptr() : nullptr, stream_of(x)), "mf_lnl_bwd");
  return {dx, dw, db, dlw, dlb};
}

std::tuple<Tensor, Tensor, Tensor> lnl_forward(const Tensor& x_, const Tensor& w_, const OptTensor& b_, const Tensor& lw_, const OptTensor& lb_, double eps,
                                               int64_t flags) {
  Tensor x = x_, w = w_, b = or_none(b_), lw = lw_, lb = or_none(lb_);
  require_cuda({&x, &w, &b, &lw, &lb});
  TORCH_CHECK_VALUE(w.dim() == 2 && x.dim() >= 1 && w.size(0) == x.size(-1), "Incompatible dimensions");
  const c10::cuda::CUDAGuard guard(x.device());
  const auto dt = x.scalar_type();
  cast_batch({{&x, dt}, {&w, dt}, {&b, dt}, {&lw, dt}, {&lb, dt}});
  return lnl_fwd_raw(x, w, b, lw, lb, eps, flags);
}

// The kernels read M x N values of dy, in whatever shape they come, and M of each row statistic.
void check_gradient(const Tensor& dy, int64_t M, int64_t N, const Tensor& mean, const Tensor& rstd) {
  TORCH_CHECK_VALUE(dy.numel() == M * N, "the gradient must hold ", M, " x ", N, " values, got ", shape(dy));
  TORCH_CHECK_VALUE(mean.numel() == M && rstd.numel() == M && mean.is_contiguous() && rstd.is_contiguous(), "mean and rstd must hold a value for each of the ", M,
                    " rows, got ", shape(mean), " and ", shape(rstd));
}

std::array<Tensor, 5> lnl_backward(const Tensor& dy_, const Tensor& x_, const Tensor& w_, const Tensor& lw_, const OptTensor& lb_, const Tensor& mean,
                                   const Tensor& rstd, bool has_linear_bias, int64_t flags) {
  Tensor dy = dy_, x = x_, w = w_, lw = lw_, lb = or_none(lb_);
  require_cuda({&dy, &x, &w, &lw, &lb, &mean, &rstd});
  TORCH_CHECK_VALUE(w.dim() == 2 && x.dim() >= 1 && w.size(0) == x.size(-1), "Incompatible dimensions");
  check_gradient(dy, rows_of(x), w.size(1), mean, rstd);
  const c10::cuda::CUDAGuard guard(x.device());
  const auto dt = x.scalar_type();
  cast_batch({{&x, dt}, {&dy, dt}, {&w, dt}, {&lw, dt}, {&lb, dt}});
  return lnl_bwd_raw(dy, x, w, lw, lb, mean, rstd, has_linear_bias, flags);
}

// types of the arguments before autocast converted them: the gradients go back in those
template <size_t N>
void save_types(AutogradContext* ctx, const std::array<at::ScalarType, N>& t) {
  std::vector<int64_t> v;
  for (auto x : t) v.push_back((int64_t)x);
  ctx->saved_data["types"] = v;
}
std::vector<at::ScalarType> saved_types(AutogradContext* ctx) {
  std::vector<at::ScalarType> out;
  for (int64_t x : ctx->saved_data["types"].toIntVector()) out.push_back((at::ScalarType)x);
  return out;
}
at::ScalarType type_of(const Tensor& t) { return t.defined() ? t.scalar_type() : at::kFloat; }

struct LnlFn : torch::autograd::Function<LnlFn> {
  static Variable forward(AutogradContext* ctx, const Tensor& x_, const Tensor& w_, const OptTensor& b_, const Tensor& lw_, const OptTensor& lb_) {
    Tensor x = x_, w = w_, b = or_none(b_), lw = lw_, lb = or_none(lb_);
    const c10::cuda::CUDAGuard guard(x.device());
    const auto dt = amp_type(x, autocast_on());
    save_types<5>(ctx, {type_of(x), type_of(w), type_of(b), type_of(lw), type_of(lb)});
    cast_batch({{&x, dt}, {&w, dt}, {&b, dt}, {&lw, dt}, {&lb, dt}});
    auto [y, mean, rstd] = lnl_fwd_raw(x, w, b, lw, lb, 1e-5, 0);
    ctx->save_for_backward({x, w, lw, lb, mean, rstd});
    ctx->saved_data["bias"] = b.defined();
    return y;
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list g) {
    at::NoGradGuard no_grad;
    const auto s = ctx->get_saved_variables();
    const auto t = saved_types(ctx);
    const c10::cuda::CUDAGuard guard(s[0].device());
    Tensor dy = g[0];
    cast_batch({{&dy, s[0].scalar_type()}});
    auto r = lnl_bwd_raw(dy, s[0], s[1], s[2], s[3], s[4], s[5], ctx->saved_data["bias"].toBool(), 0);
    cast_batch({{&r[0], t[0]}, {&r[1], t[1]}, {&r[2], t[2]}, {&r[3], t[3]}, {&r[4], t[4]}});
    return {r[0], r[1], r[2], r[3], r[4]};
  }
};

Tensor lnl(const Tensor& x, const Tensor& w, const OptTensor& b, const Tensor& lw, const OptTensor& lb) {
  const Tensor bt = or_none(b), lbt = or_none(lb);
  require_cuda({&x, &w, &bt, &lw, &lbt});
  TORCH_CHECK_VALUE(w.dim() == 2 && x.dim() >= 1 && w.size(0) == x.size(-1), "Incompatible dimensions");
  if (!at::GradMode::is_enabled()) {
    refuse_transforms({&x, &w, &bt, &lw, &lbt});
    const bool on = autocast_on();
    Tensor xc = x, wc = w, bc = bt, lwc = lw, lbc = lbt;
    const c10::cuda::CUDAGuard guard(x.device());
    const auto dt = amp_type(x, on);
    cast_batch({{&xc, dt}, {&wc, dt}, {&bc, dt}, {&lwc, dt}, {&lbc, dt}});
    return std::get<0>(lnl_fwd_raw(xc, wc, bc, lwc, lbc, 1e-5, 0));
  }
  return LnlFn::apply(x, w, b, lw, lb);
}

// ---- SwiGLU ---------------------------------------------------------------------------------------------------------
Tensor swiglu_fwd_raw(const Tensor& x) {
  const int64_t inner = x.size(-1) / 2;
  auto sizes = x.sizes().vec();
  sizes.back() = inner;
  Tensor y = at::empty(sizes, x.options());
  check(api.mf_swiglu_fwd(x.data_ptr(), y.data_ptr(), rows_of(x), (int32_t)inner, dtype_code(x.scalar_type()), stream_of(x)), "mf_swiglu_fwd");
  return y;
}

struct SwigluFn : torch::autograd::Function<SwigluFn> {
  static Variable forward(AutogradContext* ctx, const Tensor& x_) {
    Tensor x = x_;
    const c10::cuda::CUDAGuard guard(x.device());
    save_types<1>(ctx, {type_of(x)});
    cast_batch({{&x, amp_type(x, autocast_on())}});
    Tensor y = swiglu_fwd_raw(x);
    ctx->save_for_backward({x});
    return y;
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list g) {
    at::NoGradGuard no_grad;
    const Tensor x = ctx->get_saved_variables()[0];
    const c10::cuda::CUDAGuard guard(x.device());
    Tensor dy = g[0], dx = at::empty_like(x);
    cast_batch({{&dy, x.scalar_type()}});
    check(api.mf_swiglu_bwd(x.data_ptr(), dy.data_ptr(), dx.data_ptr(), rows_of(x), (int32_t)(x.size(-1) / 2), dtype_code(x.scalar_type()), stream_of(x)),
          "mf_swiglu_bwd");
    cast_batch({{&dx, saved_types(ctx)[0]}});
    return {dx};
  }
};

Tensor swiglu(const Tensor& x) {
  require_cuda({&x});
  TORCH_CHECK_VALUE(x.dim() >= 1 && x.size(-1) % 2 == 0, "SwiGLU needs an even last dimension");
  return SwigluFn::apply(x);
}

// ---- Transition -------------------------------------------------------------------------------------------------------
void check_transition(const Tensor& x, const Tensor& w1, const Tensor& w2) {
  const int64_t dim = x.size(-1), inner = w2.dim() == 2 ? w2.size(1) : -1;
  TORCH_CHECK_VALUE(w1.dim() == 2 && w2.dim() == 2 && w1.size(0) == dim && w1.size(1) == 2 * inner && w2.size(0) == dim, "weight shapes ", shape(w1),
                    " / ", shape(w2), " do not fit dim=", dim);
}

std::tuple<Tensor, Tensor, Tensor> transition_fwd_raw(const Tensor& x, const Tensor& lw, const Tensor& lb, const Tensor& w1, const Tensor& w2, double eps,
                                                      int64_t flags) {
  const int64_t M = rows_of(x);
  Tensor y = at::empty(x.sizes(), x.options()), mean = empty_f32({M}, x), rstd = empty_f32({M}, x);
  mf_transition_fwd_args a{};
  a.M = M; a.dim = (int32_t)x.size(-1); a.inner = (int32_t)w2.size(1); a.dtype = dtype_code(x.scalar_type()); a.flags = (uint32_t)flags; a.eps = (float)eps;
  a.x = x.data_ptr(); a.ln_w = ptr(lw); a.ln_b = ptr(lb); a.w1 = w1.data_ptr(); a.w2 = w2.data_ptr();
  a.y = y.data_ptr(); a.mean = mean.data_ptr<float>(); a.rstd = rstd.data_ptr<float>();
  Tensor ws;
  if (const size_t need = api.mf_transition_fwd_workspace_bytes(&a)) {
    ws = workspace(need, x);
    a.workspace = ws.data_ptr(); a.workspace_bytes = (size_t)ws.numel();
  }
  check(api.mf_transition_fwd(&a, stream_of(x)), "mf_transition_fwd");
  return {y, mean, rstd};
}

// (dx, d_ln_w, d_ln_b, dw1, dw2), parameter gradients fp32
std::array<Tensor, 5> transition_bwd_raw(const Tensor& dy, const Tensor& x, const Tensor& lw, const Tensor& lb, const Tensor& w1, const Tensor& w2,
                                         const Tensor& mean, const Tensor& rstd, int64_t flags) {
  const int64_t dim = x.size(-1), inner = w2.size(1);
  Tensor dx = at::empty(x.sizes(), x.options());
  Tensor dw1 = empty_f32({dim, 2 * inner}, x), dw2 = empty_f32({dim, inner}, x), dlw, dlb;
  if (lw.defined()) dlw = empty_f32({dim}, x);
  if (lb.defined()) dlb = empty_f32({dim}, x);
  mf_transition_bwd_args a{};
  a.M = rows_of(x); a.dim = (int32_t)dim; a.inner = (int32_t)inner; a.dtype = dtype_code(x.scalar_type()); a.flags = (uint32_t)flags;
  a.x = x.data_ptr(); a.ln_w = ptr(lw); a.ln_b = ptr(lb); a.w1 = w1.data_ptr(); a.w2 = w2.data_ptr(); a.dy = dy.data_ptr();
  a.mean = mean.data_ptr<float>(); a.rstd = rstd.data_ptr<float>();
  a.dx = dx.data_ptr(); a.dw1 = dw1.data_ptr<float>(); a.dw2 = dw2.data_ptr<float>();
  a.d_ln_w = static_cast<float*>(ptr(dlw)); a.d_ln_b = static_cast<float*>(ptr(dlb));
  Tensor ws = workspace(api.mf_transition_bwd_workspace_bytes(&a), x);
  a.workspace = ws.data_ptr(); a.workspace_bytes = (size_t)ws.numel();
  check(api.mf_transition_bwd(&a, stream_of(x)), "mf_transition_bwd");
  return {dx, dlw, dlb, dw1, dw2};
}

std::tuple<Tensor, Tensor, Tensor> transition_forward(const Tensor& x_, const OptTensor& lw_, const OptTensor& lb_, const Tensor& w1_, const Tensor& w2_,
                                                      double eps, int64_t flags) {
  Tensor x = x_, lw = or_none(lw_), lb = or_none(lb_), w1 = w1_, w2 = w2_;
  require_cuda({&x, &lw, &lb, &w1, &w2});
  check_transition(x, w1, w2);
  const c10::cuda::CUDAGuard guard(x.device());
  const auto dt = x.scalar_type();
  cast_batch({{&x, dt}, {&lw, dt}, {&lb, dt}, {&w1, dt}, {&w2, dt}});
  return transition_fwd_raw(x, lw, lb, w1, w2, eps, flags);
}

std::array<Tensor, 5> transition_backward(const Tensor& dy_, const Tensor& x_, const OptTensor& lw_, const OptTensor& lb_, const Tensor& w1_,
                                          const Tensor& w2_, const Tensor& mean, const Tensor& rstd, int64_t flags) {
  Tensor dy = dy_, x = x_, lw = or_none(lw_), lb = or_none(lb_), w1 = w1_, w2 = w2_;
  require_cuda({&dy, &x, &lw, &lb, &w1, &w2, &mean, &rstd});
  check_transition(x, w1, w2);
  check_gradient(dy, rows_of(x), x.size(-1), mean, rstd);
  const c10::cuda::CUDAGuard guard(x.device());
  const auto dt = x.scalar_type();
  cast_batch({{&x, dt}, {&dy, dt}, {&lw, dt}, {&lb, dt}, {&w1, dt}, {&w2, dt}});
  return transition_bwd_raw(dy, x, lw, lb, w1, w2, mean, rstd, flags);
}

struct TransitionFn : torch::autograd::Function<TransitionFn> {
  static Variable forward(AutogradContext* ctx, const Tensor& x_, const OptTensor& lw_, const OptTensor& lb_, const Tensor& w1_, const Tensor& w2_) {
    Tensor x = x_, lw = or_none(lw_), lb = or_none(lb_), w1 = w1_, w2 = w2_;
    const c10::cuda::CUDAGuard guard(x.device());
    const auto dt = amp_type(x, autocast_on());
    save_types<5>(ctx, {type_of(x), type_of(lw), type_of(lb), type_of(w1), type_of(w2)});
    cast_batch({{&x, dt}, {&lw, dt}, {&lb, dt}, {&w1, dt}, {&w2, dt}});
    auto [y, mean, rstd] = transition_fwd_raw(x, lw, lb, w1, w2, 1e-5, 0);
    ctx->save_for_backward({x, lw, lb, w1, w2, mean, rstd});
    return y;
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list g) {
    at::NoGradGuard no_grad;
    const auto s = ctx->get_saved_variables();
    const auto t = saved_types(ctx);
    const c10::cuda::CUDAGuard guard(s[0].device());
    Tensor dy = g[0];
    cast_batch({{&dy, s[0].scalar_type()}});
    auto r = transition_bwd_raw(dy, s[0], s[1], s[2], s[3], s[4], s[5], s[6], 0);
    cast_batch({{&r[0], t[0]}, {&r[1], t[1]}, {&r[2], t[2]}, {&r[3], t[3]}, {&r[4], t[4]}});
    return {r[0], r[1], r[2], r[3], r[4]};
  }
};

Tensor transition(const Tensor& x, const OptTensor& lw, const OptTensor& lb, const Tensor& w1, const Tensor& w2) {
  const Tensor lwt = or_none(lw), lbt = or_none(lb);
  require_cuda({&x, &lwt, &lbt, &w1, &w2});
  check_transition(x, w1, w2);
  if (!at::GradMode::is_enabled()) {
    refuse_transforms({&x, &lwt, &lbt, &w1, &w2});
    const auto dt = amp_type(x, autocast_on());
    Tensor xc = x, lwc = lwt, lbc = lbt, w1c = w1, w2c = w2;
    const c10::cuda::CUDAGuard guard(x.device());
    cast_batch({{&xc, dt}, {&lwc, dt}, {&lbc, dt}, {&w1c, dt}, {&w2c, dt}});
    return std::get<0>(transition_fwd_raw(xc, lwc, lbc, w1c, w2c, 1e-5, 0));
  }
  return TransitionFn::apply(x, lw, lb, w1, w2);
}

// ---- pieces of a Pairformer block -----------------------------------------------------------------------------------
// Attention with a merged q/k/v/gate projection, its output gate, output projection and residual connection as one
// function: q, k and v are strided views of the projection, their gradients are written straight into the projection's
// gradient, attention along the other axis of a square x (`swap`) works on strides, and the gradients of the residual
// connection and of the bias projection are added where the merged projection's backward produces dx.  Composed from
// separate autograd functions, the copies and additions between them took a quarter of the block's time.
//
// Sums and roundings follow the composed operators' as they were when this form was written.  The gradient of a bias
// projection's shift is 0 up to the rounding of d_pair_bias (a softmax's logit gradients sum to 0): it is another number as
// soon as one bit before it changes, and so two places below that could run a faster kernel with other last bits do not.
struct Attn { Tensor lw, lb, w, b, w_out; };
// The kernels take the parameters as contiguous arrays (only w_out is multiplied by torch, on strides): a transposed or
// otherwise strided parameter is copied.
Attn contiguous(const Tensor& lw, const Tensor& lb, const Tensor& w, const Tensor& b, const Tensor& w_out) {
  return {plain(lw).contiguous(), plain(lb).contiguous(), plain(w).contiguous(), plain(b).contiguous(), w_out};
}

// The matrix products between the kernels compute in the type of their operands, whose memory the kernels then read: autocast
// would change it, in a backward pass too that is run inside a region the forward pass was outside of.
struct NoAutocast { const c10::impl::ExcludeDispatchKeyGuard guard{c10::DispatchKey::AutocastCUDA}; };

mf_evo_layout token_layout(int64_t n, int64_t L, int64_t tok_o, int64_t tok_q, bool swap) {
  mf_evo_layout l{};
  for (int64_t* s : {l.o, l.d_o}) { s[0] = n * L * tok_o; s[1] = swap ? tok_o : L * tok_o; s[2] = swap ? L * tok_o : tok_o; }
  l.d_qkv[0] = n * L * tok_q; l.d_qkv[1] = swap ? tok_q : L * tok_q; l.d_qkv[2] = swap ? L * tok_q : tok_q;
  return l;
}
template <typename A>
void fill_attn(A& a, const Tensor& y, const Tensor& mask, const Tensor& bias, int64_t n, int64_t L, int64_t H, int64_t D, bool swap) {
  const int64_t inner = H * D, tok = 4 * inner, es = y.element_size();
  a.B = 1; a.N = (int32_t)(swap ? L : n); a.L = (int32_t)(swap ? n : L); a.H = (int32_t)H; a.D = (int32_t)D;
  a.dtype = dtype_code(y.scalar_type()); a.bias_dtype = dtype_code(bias.scalar_type()); a.mask_dtype = dtype_code(mask.scalar_type());
  const char* p = static_cast<const char*>(y.data_ptr());
  a.q = p; a.k = p + inner * es; a.v = p + 2 * inner * es;
  for (int64_t* s : {a.q_strides, a.k_strides, a.v_strides}) {
    s[0] = n * L * tok; s[1] = swap ? tok : L * tok; s[2] = swap ? L * tok : tok; s[3] = D; s[4] = 1;
  }
  a.mask = mask.data_ptr();
  a.mask_strides[0] = a.mask_strides[1] = 0; a.mask_strides[2] = mask.stride(0);
  a.bias = bias.data_ptr();
  a.bias_strides[0] = bias.stride(0); a.bias_strides[1] = bias.stride(2); a.bias_strides[2] = bias.stride(3); a.bias_strides[3] = bias.stride(4);
}

struct AttnSaved { Tensor y, mean, rstd, o, lse, og; };
// x [n, L, C] contiguous -> x + attention(x)
Tensor attn_fwd(const Tensor& x, const Attn& p, const Tensor& mask, const Tensor& bias, int64_t H, bool swap, AttnSaved& s, int64_t lnl_flags) {
  const NoAutocast no_autocast;
  const int64_t n = x.size(0), L = x.size(1), inner = p.w.size(1) / 4, D = inner / H;
  std::tie(s.y, s.mean, s.rstd) = lnl_fwd_raw(x, p.w, p.b, p.lw, p.lb, 1e-5, lnl_flags);
  s.o = at::empty({n, L, inner}, x.options());
  s.lse = empty_f32({swap ? L : n, H, swap ? n : L}, x);
  mf_evo_fwd_args a{};
  fill_attn(a, s.y, mask, bias, n, L, H, D, swap);
  a.o = s.o.data_ptr(); a.lse = s.lse.data_ptr<float>();
  const mf_evo_layout lay = token_layout(n, L, inner, 4 * inner, swap);
  // no scratch: with a bias that TMA cannot address (L not a multiple of 8) the general kernel reads it in place.  The
  // attention operator, which gives scratch, is faster there: a block of 467 tokens takes 6.1 ms, composed of the operators
  // 5.1 (464 tokens: 3.9 and 4.9).
  check(api.mf_evo_fwd_laid_out(&a, &lay, nullptr, 0, stream_of(x)), "mf_evo_fwd");
  s.og = at::empty_like(s.o);
  check(api.mf_gate_fwd(s.o.data_ptr(), static_cast<char*>(s.y.data_ptr()) + 3 * inner * x.element_size(), 4 * inner, s.og.data_ptr(), n * L, (int32_t)inner,
                        a.dtype, stream_of(x)), "mf_gate_fwd");
  Tensor out = at::mm(s.og.view({n * L, inner}), p.w_out.t());
  return out.add_(x.view({n * L, x.size(2)})).view(x.sizes());
}

struct AttnGrads { Tensor dx, dw, db, dlw, dlb, d_w_out, d_bias; };
// bias_dx turns d_bias into the gradient that x receives through the bias (undefined: none); dx comes with it and with
// d_out, the residual connection's, added in the order of the composed form
template <typename BiasDx>
AttnGrads attn_bwd(const Tensor& d_out, const Tensor& x, const Attn& p, const Tensor& mask, const Tensor& bias, int64_t H, bool swap, const AttnSaved& s,
                   BiasDx bias_dx) {
  const NoAutocast no_autocast;
  const int64_t n = x.size(0), L = x.size(1), C = x.size(2), inner = p.w.size(1) / 4, D = inner / H, P = n * L, es = x.element_size();
  AttnGrads g;
  const Tensor d2 = d_out.view({P, C});
  g.d_w_out = at::mm(d2.t(), s.og.view({P, inner}));
  Tensor d_og = at::mm(d2, p.w_out), d_o = at::empty({n, L, inner}, x.options()), dy = at::empty({P, 4 * inner}, x.options());
  const char* y = static_cast<const char*>(s.y.data_ptr());
  char* dyp = static_cast<char*>(dy.data_ptr());
  const int dt = dtype_code(x.scalar_type());
  check(api.mf_gate_bwd(d_og.data_ptr(), s.o.data_ptr(), y + 3 * inner * es, 4 * inner, d_o.data_ptr(), dyp + 3 * inner * es, 4 * inner, P, (int32_t)inner, dt,
                        stream_of(x)), "mf_gate_bwd");
  d_og.reset();
  g.d_bias = at::empty(bias.sizes(), bias.options());
  mf_evo_bwd_args a{};
  fill_attn(a, s.y, mask, bias, n, L, H, D, swap);
  a.dbias_dtype = dtype_code(g.d_bias.scalar_type());
  a.o = s.o.data_ptr(); a.d_o = d_o.data_ptr(); a.lse = s.lse.data_ptr<float>();
  a.dq = dyp; a.dk = dyp + inner * es; a.dv = dyp + 2 * inner * es; a.d_bias = g.d_bias.data_ptr();
  const mf_evo_layout lay = token_layout(n, L, inner, 4 * inner, swap);
  Tensor ws = workspace(api.mf_evo_bwd_workspace_bytes(&a), x);
  a.workspace = ws.data_ptr(); a.workspace_bytes = (size_t)ws.numel();
  check(api.mf_evo_bwd_laid_out(&a, &lay, stream_of(x)), "mf_evo_bwd");
  ws.reset(); d_o.reset();
  const Tensor through_bias = bias_dx(g.d_bias);
  const Tensor *add1 = through_bias.defined() ? &through_bias : nullptr, *add2 = &d_out;
  if (!swap) std::swap(add1, add2);
  auto r = lnl_bwd_raw(dy, x, p.w, p.lw, p.lb, s.mean, s.rstd, true, 0, add1, add2);
  cast_batch({{&r[1], p.w.scalar_type()}, {&r[2], p.b.scalar_type()}, {&r[3], p.lw.scalar_type()}, {&r[4], p.lb.scalar_type()}});
  g.dx = r[0]; g.dw = r[1]; g.db = r[2]; g.dlw = r[3]; g.dlb = r[4];
  return g;
}

// Pair bias [1, 1, H, L, L] projected from x [L, L, C]: element (i, j) from x[i, j], or from x[j, i] with `swap`.
struct BiasSaved { Tensor mean, rstd; };
Tensor bias_fwd(const Tensor& x, const Tensor& lw, const Tensor& lb, const Tensor& w, int64_t H, bool swap, BiasSaved& s) {
  const int64_t L = x.size(0);
  Tensor rows;
  std::tie(rows, s.mean, s.rstd) = lnl_fwd_raw(x, w, Tensor(), lw, lb, 1e-5, 0);
  Tensor bias = at::empty({1, 1, H, L, L}, x.options());
  check(api.mf_bias_layout(rows.data_ptr(), bias.data_ptr(), (int32_t)L, (int32_t)w.size(1), (int32_t)H, swap, 0, dtype_code(x.scalar_type()), stream_of(x)),
        "mf_bias_layout");
  return bias;
}
// (dx, dw, dlw, dlb)
std::array<Tensor, 4> bias_bwd(const Tensor& d_bias, const Tensor& x, const Tensor& lw, const Tensor& lb, const Tensor& w, bool swap, const BiasSaved& s) {
  const int64_t L = x.size(0), np = w.size(1);
  Tensor rows = at::empty({L * L, np}, x.options());
  check(api.mf_bias_layout(rows.data_ptr(), d_bias.data_ptr(), (int32_t)L, (int32_t)np, (int32_t)d_bias.size(2), swap, 1, dtype_code(x.scalar_type()),
                           stream_of(x)), "mf_bias_layout");
  auto r = lnl_bwd_raw(rows, x, w, lw, lb, s.mean, s.rstd, false, 0);
  cast_batch({{&r[1], w.scalar_type()}, {&r[3], lw.scalar_type()}, {&r[4], lb.scalar_type()}});
  return {r[0], r[1], r[3], r[4]};
}

// x [L, L, C] + attention over its rows (or, with `swap`, its columns) with a pair bias projected from x itself
struct TriangleFn : torch::autograd::Function<TriangleFn> {
  static Variable forward(AutogradContext* ctx, const Tensor& x_, const Tensor& lw, const Tensor& lb, const Tensor& w, const Tensor& b, const Tensor& w_out,
                          const Tensor& plw_, const Tensor& plb_, const Tensor& pw_, const Tensor& mask, int64_t H, bool swap) {
    const c10::cuda::CUDAGuard guard(x_.device());
    const Tensor x = plain(x_).contiguous(), plw = plain(plw_).contiguous(), plb = plain(plb_).contiguous(), pw = plain(pw_).contiguous();
    const Attn p = contiguous(lw, lb, w, b, w_out);
    AttnSaved s; BiasSaved bs;
    const Tensor bias = bias_fwd(x, plw, plb, pw, H, swap, bs);
    Tensor out = attn_fwd(x, p, mask, bias, H, swap, s, 0);
    ctx->save_for_backward({x, p.lw, p.lb, p.w, p.b, p.w_out, plw, plb, pw, mask, bias, s.y, s.mean, s.rstd, s.o, s.lse, s.og, bs.mean, bs.rstd});
    ctx->saved_data["H"] = H; ctx->saved_data["swap"] = swap;
    return out;
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list g) {
    at::NoGradGuard no_grad;
    const auto v = ctx->get_saved_variables();
    const c10::cuda::CUDAGuard guard(v[0].device());
    const int64_t H = ctx->saved_data["H"].toInt();
    const bool swap = ctx->saved_data["swap"].toBool();
    const AttnSaved s{v[11], v[12], v[13], v[14], v[15], v[16]};
    std::array<Tensor, 4> p;
    AttnGrads a = attn_bwd(plain(g[0]).contiguous(), v[0], {v[1], v[2], v[3], v[4], v[5]}, v[9], v[10], H, swap, s, [&](const Tensor& d_bias) {
      p = bias_bwd(d_bias, v[0], v[6], v[7], v[8], swap, BiasSaved{v[17], v[18]});
      return p[0];
    });
    return {a.dx, a.dlw, a.dlb, a.dw, a.db, a.d_w_out, p[2], p[3], p[1], Tensor(), Tensor(), Tensor()};
  }
};

// x [n, L, C] + attention over its rows with a given pair bias
struct GatedAttnFn : torch::autograd::Function<GatedAttnFn> {
  static Variable forward(AutogradContext* ctx, const Tensor& x_, const Tensor& lw, const Tensor& lb, const Tensor& w, const Tensor& b, const Tensor& w_out,
                          const Tensor& mask, const Tensor& bias, int64_t H) {
    const c10::cuda::CUDAGuard guard(x_.device());
    const Tensor x = plain(x_).contiguous();
    const Attn p = contiguous(lw, lb, w, b, w_out);
    AttnSaved s;
    // the projection of these few wide rows runs on the CUDA cores (46 us instead of 12, 0.4 % of a block at 768 tokens): see above
    Tensor out = attn_fwd(x, p, mask, bias, H, false, s, MF_FLAG_FORCE_SIMT);
    ctx->save_for_backward({x, p.lw, p.lb, p.w, p.b, p.w_out, mask, bias, s.y, s.mean, s.rstd, s.o, s.lse, s.og});
    ctx->saved_data["H"] = H;
    return out;
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list g) {
    at::NoGradGuard no_grad;
    const auto v = ctx->get_saved_variables();
    const c10::cuda::CUDAGuard guard(v[0].device());
    const AttnSaved s{v[8], v[9], v[10], v[11], v[12], v[13]};
    AttnGrads a = attn_bwd(plain(g[0]).contiguous(), v[0], {v[1], v[2], v[3], v[4], v[5]}, v[6], v[7], ctx->saved_data["H"].toInt(), false, s,
                           [](const Tensor&) { return Tensor(); });
    return {a.dx, a.dlw, a.dlb, a.dw, a.db, a.d_w_out, Tensor(), a.d_bias, Tensor()};
  }
};

struct PairBiasFn : torch::autograd::Function<PairBiasFn> {
  static Variable forward(AutogradContext* ctx, const Tensor& x_, const Tensor& lw_, const Tensor& lb_, const Tensor& w_, int64_t H) {
    const c10::cuda::CUDAGuard guard(x_.device());
    const Tensor x = plain(x_).contiguous(), lw = plain(lw_).contiguous(), lb = plain(lb_).contiguous(), w = plain(w_).contiguous();
    BiasSaved s;
    Tensor bias = bias_fwd(x, lw, lb, w, H, false, s);
    ctx->save_for_backward({x, lw, lb, w, s.mean, s.rstd});
    return bias;
  }
  static tensor_list backward(AutogradContext* ctx, tensor_list g) {
    at::NoGradGuard no_grad;
    const auto v = ctx->get_saved_variables();
    const c10::cuda::CUDAGuard guard(v[0].device());
    auto p = bias_bwd(plain(g[0]).contiguous(), v[0], v[1], v[2], v[3], false, BiasSaved{v[4], v[5]});
    return {p[0], p[2], p[3], p[1], Tensor()};
  }
};

Tensor triangle(const Tensor& x, const Tensor& lw, const Tensor& lb, const Tensor& w, const Tensor& b, const Tensor& w_out, const Tensor& plw, const Tensor& plb,
                const Tensor& pw, const Tensor& mask, int64_t H, bool swap) {
  require_cuda({&x, &lw, &lb, &w, &b, &w_out, &plw, &plb, &pw, &mask});
  TORCH_CHECK_VALUE(x.dim() == 3 && x.size(0) == x.size(1) && mask.dim() == 1 && mask.size(0) == x.size(1) && w.size(0) == x.size(2) && pw.size(0) == x.size(2) &&
                        w.size(1) % (4 * H) == 0 && pw.size(1) >= H, "x must be [L, L, C] with a mask [L], got ", shape(x), " and ", shape(mask));
  return TriangleFn::apply(x, lw, lb, w, b, w_out, plw, plb, pw, mask, H, swap);
}
Tensor gated_attention(const Tensor& x, const Tensor& lw, const Tensor& lb, const Tensor& w, const Tensor& b, const Tensor& w_out, const Tensor& mask,
                       const Tensor& bias, int64_t H) {
  require_cuda({&x, &lw, &lb, &w, &b, &w_out, &mask, &bias});
  TORCH_CHECK_VALUE(x.dim() == 3 && mask.dim() == 1 && mask.size(0) == x.size(1) && w.size(0) == x.size(2) && w.size(1) % (4 * H) == 0 && bias.dim() == 5 &&
                        bias.size(2) == H && bias.size(3) == x.size(1) && bias.size(4) == x.size(1), "x must be [n, L, C] with a mask [L] and a bias [1, 1, H, L, L], got ",
                    shape(x), ", ", shape(mask), " and ", shape(bias));
  return GatedAttnFn::apply(x, lw, lb, w, b, w_out, mask, bias, H);
}
Tensor pair_bias(const Tensor& x, const Tensor& lw, const Tensor& lb, const Tensor& w, int64_t H) {
  require_cuda({&x, &lw, &lb, &w});
  TORCH_CHECK_VALUE(x.dim() == 3 && x.size(0) == x.size(1) && w.size(0) == x.size(2) && w.size(1) >= H, "x must be [L, L, C], got ", shape(x));
  return PairBiasFn::apply(x, lw, lb, w, H);
}

// std::array of tensors, undefined ones as None
template <size_t N>
std::array<OptTensor, N> optional(std::array<Tensor, N> r) {
  std::array<OptTensor, N> o;
  for (size_t i = 0; i < N; ++i)
    if (r[i].defined()) o[i] = std::move(r[i]);
  return o;
}

}  // namespace

PYBIND11_MODULE(_native, m) {
  using release = pybind11::call_guard<pybind11::gil_scoped_release>;
  m.def("load", &load);
  m.def("check_shapes", [](const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& mask, const OptTensor& bias) {
    const auto s = check_shapes(q, k, v, mask, bias);
    return std::make_tuple(s[0], s[1], s[2], s[3], s[4]);
  });
  m.def("evo_forward", &evo_forward, release());
  m.def("evo_backward", &evo_backward, release());
  m.def("evo_attention", &evo_attention, release());
  m.def("lnl_forward", &lnl_forward, release());
  m.def("lnl_backward", [](const Tensor& dy, const Tensor& x, const Tensor& w, const Tensor& lw, const OptTensor& lb, const Tensor& mean, const Tensor& rstd,
                           bool has_linear_bias, int64_t flags) { return optional(lnl_backward(dy, x, w, lw, lb, mean, rstd, has_linear_bias, flags)); },
        release());
  m.def("lnl", &lnl, release());
  m.def("swiglu", &swiglu, release());
  m.def("transition_forward", &transition_forward, release());
  m.def("transition_backward", [](const Tensor& dy, const Tensor& x, const OptTensor& lw, const OptTensor& lb, const Tensor& w1, const Tensor& w2,
                                  const Tensor& mean, const Tensor& rstd, int64_t flags) {
    return optional(transition_backward(dy, x, lw, lb, w1, w2, mean, rstd, flags));
  }, release());
  m.def("transition", &transition, release());
  m.def("triangle", &triangle, release());
  m.def("gated_attention", &gated_attention, release());
  m.def("pair_bias", &pair_bias, release());
}
