// C ABI of the library: argument validation and dispatch to the kernel families.
#include "common.cuh"

#include <cuda.h>
#include <nvtx3/nvToolsExt.h>

namespace mf {

char* last_error_buf() {
  static thread_local char buf[512] = "no error";
  return buf;
}
static thread_local const char* t_last_path = "none";
void set_last_path(const char* p) { t_last_path = p; }
std::atomic<uint64_t> g_launches{0};

namespace {

// One NVTX range per entry point (the reference marks its fused operators the same way for its timeline traces); without
// a profiler attached the calls return at once.
struct Range {
  explicit Range(const char* name) { nvtxRangePushA(name); }
  ~Range() { nvtxRangePop(); }
  Range(const Range&) = delete;
  Range& operator=(const Range&) = delete;
};

bool float_dtype(int dt) { return dt == MF_F32 || dt == MF_BF16 || dt == MF_F16; }

// A thread that has made no runtime call yet (an autograd worker) has no current context, which the tensor-map encoding,
// a driver call, needs; cudaSetDevice of the device that is current already does not make one.  The calls used here are
// legal while any stream is being captured.
int bind_context(int dev) {
  static std::mutex mu;
  static CUcontext primary[64] = {};
  auto entry = [](const char* name) {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    return cudaGetDriverEntryPoint(name, &f, cudaEnableDefault, &q) == cudaSuccess ? f : nullptr;
  };
  static const auto get = reinterpret_cast<CUresult (*)(CUcontext*)>(entry("cuCtxGetCurrent"));
  static const auto set = reinterpret_cast<CUresult (*)(CUcontext)>(entry("cuCtxSetCurrent"));
  static const auto retain = reinterpret_cast<CUresult (*)(CUcontext*, CUdevice)>(entry("cuDevicePrimaryCtxRetain"));
  CUcontext cur = nullptr;
  MF_REQUIRE(get && set && retain && dev >= 0 && dev < 64, MF_ERR_CUDA, "the driver's context calls are not available");
  if (get(&cur) == CUDA_SUCCESS && cur) return MF_OK;
  std::lock_guard<std::mutex> lk(mu);
  if (!primary[dev]) MF_REQUIRE(retain(&primary[dev], dev) == CUDA_SUCCESS, MF_ERR_CUDA, "no primary context on device %d", dev);
  MF_REQUIRE(set(primary[dev]) == CUDA_SUCCESS, MF_ERR_CUDA, "the primary context of device %d cannot be made current", dev);
  return MF_OK;
}

int check_device() {
  static thread_local int checked_dev = -1;
  int dev = 0;
  MF_CUDA(cudaGetDevice(&dev));
  if (dev == checked_dev) return MF_OK;
  { int r = bind_context(dev); if (r) return r; }
  int major = 0;
  MF_CUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev));
  MF_REQUIRE(major == 10, MF_ERR_ARCH, "device %d has compute capability %d.x; this library is built for sm_100a only", dev, major);
  checked_dev = dev;
  return MF_OK;
}

template <typename A>
int check_evo_common(const A& a) {
  MF_REQUIRE(a.B > 0 && a.N > 0 && a.L > 0 && a.H > 0 && a.D > 0, MF_ERR_BAD_ARG,
             "sizes must be positive (B=%d N=%d L=%d H=%d D=%d)", a.B, a.N, a.L, a.H, a.D);
  MF_REQUIRE(float_dtype(a.dtype), MF_ERR_BAD_ARG, "q/k/v dtype %d is not a floating type", a.dtype);
  MF_REQUIRE(float_dtype(a.bias_dtype), MF_ERR_BAD_ARG, "pair_bias dtype %d is not a floating type", a.bias_dtype);
  MF_REQUIRE(float_dtype(a.mask_dtype) || a.mask_dtype == MF_U8, MF_ERR_BAD_ARG, "res_mask dtype %d unknown", a.mask_dtype);
  MF_REQUIRE(a.q && a.k && a.v, MF_ERR_BAD_ARG, "q, k and v must not be NULL");
  MF_REQUIRE(a.mask, MF_ERR_BAD_ARG, "res_mask must not be NULL");
  MF_REQUIRE(a.bias, MF_ERR_BAD_ARG, "pair_bias is mandatory and must not be NULL");
  MF_REQUIRE(a.D <= 128, MF_ERR_UNSUPPORTED, "head size %d > 128 is not supported", a.D);
  MF_REQUIRE((int64_t)a.B * a.N <= 65535 && a.H <= 65535, MF_ERR_UNSUPPORTED, "B*N=%lld or H=%d exceeds 65535",
             (long long)a.B * a.N, a.H);
  return MF_OK;
}

}  // namespace
}  // namespace mf

using namespace mf;

namespace mf {
namespace {

template <typename A>
mf_evo_layout contiguous_layout(const A& a) {
  mf_evo_layout l;
  const int64_t tok = (int64_t)a.H * a.D;
  for (int64_t* s : {l.o, l.d_o, l.d_qkv}) { s[0] = tok * a.L * a.N; s[1] = tok * a.L; s[2] = tok; }
  return l;
}
// the tensor-core kernels use 16-byte accesses on these arrays
bool rows16(const int64_t (&s)[3]) { return (s[0] % 8 | s[1] % 8 | s[2] % 8) == 0; }

bool evo_fwd_use_tc(const mf_evo_fwd_args& a, const mf_evo_layout& lay) {
  return !(a.flags & MF_FLAG_FORCE_SIMT) && ((uintptr_t)a.o & 15) == 0 && rows16(lay.o) &&
         evo_tc_supported(a.B, a.N, a.L, a.H, a.D, a.dtype, a.q_strides, a.k_strides, a.v_strides, a.q, a.k, a.v);
}
bool evo_bwd_use_tc(const mf_evo_bwd_args& a, const mf_evo_layout& lay) {
  const uintptr_t align = (uintptr_t)a.o | (uintptr_t)a.d_o | (uintptr_t)a.dq | (uintptr_t)a.dk | (uintptr_t)a.dv;
  return !(a.flags & MF_FLAG_FORCE_SIMT) && (align & 15) == 0 && rows16(lay.o) && rows16(lay.d_o) && rows16(lay.d_qkv) && evo_bwd_ws_shape_ok(a.L, a.D) &&
         evo_tc_supported(a.B, a.N, a.L, a.H, a.D, a.dtype, a.q_strides, a.k_strides, a.v_strides, a.q, a.k, a.v);
}

int check_evo_bwd(const mf_evo_bwd_args& a) {
  int r = check_evo_common(a); if (r) return r;
  MF_REQUIRE(a.o && a.d_o && a.lse, MF_ERR_BAD_ARG, "o, d_o and lse must not be NULL");
  MF_REQUIRE(a.dq && a.dk && a.dv && a.d_bias, MF_ERR_BAD_ARG, "dq, dk, dv and d_bias must not be NULL");
  MF_REQUIRE(a.dbias_dtype == MF_F32 || a.dbias_dtype == a.dtype, MF_ERR_BAD_ARG,
             "d_bias dtype must be fp32 or the q/k/v dtype");
  return MF_OK;
}

}  // namespace
}  // namespace mf

extern "C" {

size_t mf_evo_fwd_workspace_bytes(const mf_evo_fwd_args* args) {
  if (!args) return 0;
  return evo_fwd_use_tc(*args, contiguous_layout(*args)) ? evo_fwd_ws_workspace(*args) : 0;
}

int mf_evo_fwd_laid_out(const mf_evo_fwd_args* args, const mf_evo_layout* layout, void* workspace, size_t workspace_bytes, void* stream) {
  Range nvtx_range("mf_evo_fwd");
  MF_REQUIRE(args, MF_ERR_BAD_ARG, "args is NULL");
  const mf_evo_fwd_args& a = *args;
  int r = check_evo_common(a); if (r) return r;
  MF_REQUIRE(a.o && a.lse, MF_ERR_BAD_ARG, "o and lse must not be NULL");
  if (!workspace) workspace_bytes = 0;
  MF_REQUIRE(((uintptr_t)workspace & 255) == 0, MF_ERR_ALIGNMENT, "workspace must be 256-byte aligned");
  r = check_device(); if (r) return r;
  const mf_evo_layout lay = layout ? *layout : contiguous_layout(a);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (evo_fwd_use_tc(a, lay)) {
    r = evo_fwd_ws_supported(a, workspace_bytes) ? evo_fwd_ws(a, lay, workspace, st) : evo_fwd_tc(a, lay, st);
    if (r == MF_OK) set_last_path("tcgen05");
    return r;
  }
  r = evo_fwd_simt(a, lay, st);
  if (r == MF_OK) set_last_path("simt");
  return r;
}

int mf_evo_fwd_with_workspace(const mf_evo_fwd_args* args, void* workspace, size_t workspace_bytes, void* stream) {
  return mf_evo_fwd_laid_out(args, nullptr, workspace, workspace_bytes, stream);
}
int mf_evo_fwd(const mf_evo_fwd_args* args, void* stream) { return mf_evo_fwd_laid_out(args, nullptr, nullptr, 0, stream); }

size_t mf_evo_bwd_workspace_bytes(const mf_evo_bwd_args* args) {
  if (!args) return 0;
  return evo_bwd_use_tc(*args, contiguous_layout(*args)) ? evo_bwd_ws_workspace(*args) : evo_bwd_simt_workspace(*args);
}

int mf_evo_bwd_laid_out(const mf_evo_bwd_args* args, const mf_evo_layout* layout, void* stream) {
  Range nvtx_range("mf_evo_bwd");
  MF_REQUIRE(args, MF_ERR_BAD_ARG, "args is NULL");
  const mf_evo_bwd_args& a = *args;
  int r = check_evo_bwd(a); if (r) return r;
  const mf_evo_layout lay = layout ? *layout : contiguous_layout(a);
  const bool tc = evo_bwd_use_tc(a, lay);
  const size_t need = tc ? evo_bwd_ws_workspace(a) : evo_bwd_simt_workspace(a);
  MF_REQUIRE(a.workspace && a.workspace_bytes >= need, MF_ERR_WORKSPACE, "workspace of %zu bytes needed, %zu given", need,
             a.workspace ? a.workspace_bytes : (size_t)0);
  MF_REQUIRE(((uintptr_t)a.workspace & 255) == 0, MF_ERR_ALIGNMENT, "workspace must be 256-byte aligned");
  r = check_device(); if (r) return r;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (tc) {
    r = evo_bwd_ws(a, lay, st);
    if (r == MF_OK) set_last_path("tcgen05");
    return r;
  }
  r = evo_bwd_simt(a, lay, st);
  if (r == MF_OK && a.dbias_ready_event) MF_CUDA(cudaEventRecord(static_cast<cudaEvent_t>(a.dbias_ready_event), st));
  if (r == MF_OK) set_last_path("simt");
  return r;
}
int mf_evo_bwd(const mf_evo_bwd_args* args, void* stream) { return mf_evo_bwd_laid_out(args, nullptr, stream); }

int mf_evo_bwd_noalloc(const mf_evo_bwd_args* args, void* stream) {
  Range nvtx_range("mf_evo_bwd_noalloc");
  MF_REQUIRE(args, MF_ERR_BAD_ARG, "args is NULL");
  const mf_evo_bwd_args& a = *args;
  int r = check_evo_bwd(a); if (r) return r;
  r = check_device(); if (r) return r;
  r = evo_bwd_simt_noalloc(a, contiguous_layout(a), static_cast<cudaStream_t>(stream));
  if (r == MF_OK && a.dbias_ready_event)
    MF_CUDA(cudaEventRecord(static_cast<cudaEvent_t>(a.dbias_ready_event), static_cast<cudaStream_t>(stream)));
  if (r == MF_OK) set_last_path("simt");
  return r;
}

size_t mf_evo_bwd_noalloc_max_rows(void) { return evo_bwd_noalloc_max_rows(); }

int mf_lnl_fwd(const mf_lnl_fwd_args* args, void* stream) {
  Range nvtx_range("mf_lnl_fwd");
  MF_REQUIRE(args, MF_ERR_BAD_ARG, "args is NULL");
  const mf_lnl_fwd_args& a = *args;
  MF_REQUIRE(a.M >= 0 && a.K > 0 && a.N > 0, MF_ERR_BAD_ARG, "bad sizes M=%lld K=%d N=%d", (long long)a.M, a.K, a.N);
  MF_REQUIRE(float_dtype(a.dtype), MF_ERR_BAD_ARG, "dtype %d is not a floating type", a.dtype);
  MF_REQUIRE(a.x && a.ln_w && a.w && a.y && a.mean && a.rstd, MF_ERR_BAD_ARG, "x, ln_w, w, y, mean, rstd must not be NULL");
  if (a.M == 0) return MF_OK;
  int r = check_device(); if (r) return r;
  if (!(a.flags & MF_FLAG_FORCE_SIMT) && (lnl_fwd_tc_supported(a) || lnl_fwd_wide_supported(a))) {
    r = lnl_fwd_tc_supported(a) ? lnl_fwd_tc(a, static_cast<cudaStream_t>(stream)) : lnl_fwd_wide(a, static_cast<cudaStream_t>(stream));
    if (r == MF_OK) set_last_path("tcgen05");
    return r;
  }
  r = lnl_fwd_simt(a, static_cast<cudaStream_t>(stream));
  if (r == MF_OK) set_last_path("simt");
  return r;
}

size_t mf_lnl_bwd_workspace_bytes(const mf_lnl_bwd_args* args) {
  if (!args) return 0;
  return lnl_bwd_workspace(*args);
}

int mf_lnl_bwd(const mf_lnl_bwd_args* args, void* stream) { return mf_lnl_bwd_add(args, nullptr, nullptr, stream); }

int mf_lnl_bwd_add(const mf_lnl_bwd_args* args, const void* add1, const void* add2, void* stream) {
  Range nvtx_range("mf_lnl_bwd");
  MF_REQUIRE(args, MF_ERR_BAD_ARG, "args is NULL");
  const mf_lnl_bwd_args& a = *args;
  MF_REQUIRE(a.M > 0 && a.K > 0 && a.N > 0, MF_ERR_BAD_ARG, "bad sizes M=%lld K=%d N=%d", (long long)a.M, a.K, a.N);
  MF_REQUIRE(float_dtype(a.dtype), MF_ERR_BAD_ARG, "dtype %d is not a floating type", a.dtype);
  MF_REQUIRE(a.x && a.ln_w && a.w && a.dy && a.mean && a.rstd && a.dx && a.dw && a.d_ln_w, MF_ERR_BAD_ARG,
             "x, ln_w, w, dy, mean, rstd, dx, dw, d_ln_w must not be NULL");
  const size_t need = mf_lnl_bwd_workspace_bytes(args);
  MF_REQUIRE(a.workspace && a.workspace_bytes >= need, MF_ERR_WORKSPACE, "workspace of %zu bytes needed, %zu given", need,
             a.workspace ? a.workspace_bytes : (size_t)0);
  MF_REQUIRE(((uintptr_t)a.workspace & 255) == 0, MF_ERR_ALIGNMENT, "workspace must be 256-byte aligned");
  int r = check_device(); if (r) return r;
  r = lnl_bwd(a, add1, add2, static_cast<cudaStream_t>(stream));
  if (r == MF_OK) set_last_path(lnl_bwd_runs_on_tc(a, add1, add2) ? "tcgen05" : "simt");
  return r;
}

int mf_swiglu_fwd(const void* x, void* y, int64_t M, int32_t inner, int32_t dtype, void* stream) {
  Range nvtx_range("mf_swiglu_fwd");
  MF_REQUIRE(x && y && M >= 0 && inner > 0, MF_ERR_BAD_ARG, "bad swiglu arguments");
  MF_REQUIRE(float_dtype(dtype), MF_ERR_BAD_ARG, "dtype %d is not a floating type", dtype);
  int r = check_device(); if (r) return r;
  return swiglu_fwd(x, y, M, inner, dtype, static_cast<cudaStream_t>(stream));
}

int mf_swiglu_bwd(const void* x, const void* dy, void* dx, int64_t M, int32_t inner, int32_t dtype, void* stream) {
  Range nvtx_range("mf_swiglu_bwd");
  MF_REQUIRE(x && dy && dx && M >= 0 && inner > 0, MF_ERR_BAD_ARG, "bad swiglu arguments");
  MF_REQUIRE(float_dtype(dtype), MF_ERR_BAD_ARG, "dtype %d is not a floating type", dtype);
  int r = check_device(); if (r) return r;
  return swiglu_bwd(x, dy, dx, M, inner, dtype, static_cast<cudaStream_t>(stream));
}

static bool transition_fwd_use_tc(const mf_transition_fwd_args& a) {
  return !(a.flags & MF_FLAG_FORCE_SIMT) && transition_fwd_tc_supported(a);
}
static bool transition_fwd_use_wide(const mf_transition_fwd_args& a) {
  return !(a.flags & MF_FLAG_FORCE_SIMT) && transition_fwd_wide_supported(a);
}

size_t mf_transition_fwd_workspace_bytes(const mf_transition_fwd_args* args) {
  if (!args) return 0;
  if (transition_fwd_use_tc(*args)) return 0;      // the fused kernel keeps the hidden activation on chip
  return transition_fwd_use_wide(*args) ? transition_fwd_wide_workspace(*args) : transition_fwd_simt_workspace(*args);
}

int mf_transition_fwd(const mf_transition_fwd_args* args, void* stream) {
  Range nvtx_range("mf_transition_fwd");
  MF_REQUIRE(args, MF_ERR_BAD_ARG, "args is NULL");
  const mf_transition_fwd_args& a = *args;
  MF_REQUIRE(a.M > 0 && a.dim > 0 && a.inner > 0, MF_ERR_BAD_ARG, "bad sizes");
  MF_REQUIRE(float_dtype(a.dtype), MF_ERR_BAD_ARG, "dtype %d is not a floating type", a.dtype);
  MF_REQUIRE(a.x && a.w1 && a.w2 && a.y, MF_ERR_BAD_ARG, "x, w1, w2, y must not be NULL");
  MF_REQUIRE(!a.ln_w || (a.mean && a.rstd), MF_ERR_BAD_ARG, "mean and rstd are needed with LayerNorm");
  const size_t need = mf_transition_fwd_workspace_bytes(args);
  MF_REQUIRE(need == 0 || (a.workspace && a.workspace_bytes >= need), MF_ERR_WORKSPACE,
             "workspace of %zu bytes needed, %zu given", need, a.workspace ? a.workspace_bytes : (size_t)0);
  int r = check_device(); if (r) return r;
  if (transition_fwd_use_tc(a) || transition_fwd_use_wide(a)) {
    r = transition_fwd_use_tc(a) ? transition_fwd_tc(a, static_cast<cudaStream_t>(stream)) : transition_fwd_wide(a, static_cast<cudaStream_t>(stream));
    if (r == MF_OK) set_last_path("tcgen05");
    return r;
  }
  r = transition_fwd_simt(a, static_cast<cudaStream_t>(stream));
  if (r == MF_OK) set_last_path("simt");
  return r;
}

size_t mf_transition_bwd_workspace_bytes(const mf_transition_bwd_args* args) {
  if (!args) return 0;
  return transition_bwd_workspace(*args);
}

int mf_transition_bwd(const mf_transition_bwd_args* args, void* stream) {
  Range nvtx_range("mf_transition_bwd");
  MF_REQUIRE(args, MF_ERR_BAD_ARG, "args is NULL");
  const mf_transition_bwd_args& a = *args;
  MF_REQUIRE(a.M > 0 && a.dim > 0 && a.inner > 0, MF_ERR_BAD_ARG, "bad sizes");
  MF_REQUIRE(float_dtype(a.dtype), MF_ERR_BAD_ARG, "dtype %d is not a floating type", a.dtype);
  MF_REQUIRE(a.x && a.w1 && a.w2 && a.dy && a.dx && a.dw1 && a.dw2, MF_ERR_BAD_ARG,
             "x, w1, w2, dy, dx, dw1, dw2 must not be NULL");
  MF_REQUIRE(!a.ln_w || (a.mean && a.rstd && a.d_ln_w), MF_ERR_BAD_ARG, "mean, rstd, d_ln_w are needed with LayerNorm");
  const size_t need = mf_transition_bwd_workspace_bytes(args);
  MF_REQUIRE(a.workspace && a.workspace_bytes >= need, MF_ERR_WORKSPACE, "workspace of %zu bytes needed, %zu given", need,
             a.workspace ? a.workspace_bytes : (size_t)0);
  MF_REQUIRE(((uintptr_t)a.workspace & 255) == 0, MF_ERR_ALIGNMENT, "workspace must be 256-byte aligned");
  int r = check_device(); if (r) return r;
  r = transition_bwd(a, static_cast<cudaStream_t>(stream));
  if (r == MF_OK) set_last_path(transition_bwd_runs_on_tc(a) ? "tcgen05" : "simt");
  return r;
}

int mf_gate_fwd(const void* o, const void* g, int64_t g_stride, void* out, int64_t rows, int32_t cols, int32_t dtype, void* stream) {
  Range nvtx_range("mf_gate_fwd");
  MF_REQUIRE(o && g && out && rows >= 0 && cols > 0 && float_dtype(dtype), MF_ERR_BAD_ARG, "bad gate arguments");
  int r = check_device(); if (r) return r;
  return gate_fwd(o, g, g_stride, out, rows, cols, dtype, static_cast<cudaStream_t>(stream));
}

int mf_gate_bwd(const void* d, const void* o, const void* g, int64_t g_stride, void* d_o, void* d_g, int64_t dg_stride, int64_t rows, int32_t cols,
                int32_t dtype, void* stream) {
  Range nvtx_range("mf_gate_bwd");
  MF_REQUIRE(d && o && g && d_o && d_g && rows >= 0 && cols > 0 && float_dtype(dtype), MF_ERR_BAD_ARG, "bad gate arguments");
  int r = check_device(); if (r) return r;
  return gate_bwd(d, o, g, g_stride, d_o, d_g, dg_stride, rows, cols, dtype, static_cast<cudaStream_t>(stream));
}

int mf_bias_layout(void* rows, void* planes, int32_t L, int32_t np, int32_t H, int32_t swap, int32_t to_rows, int32_t dtype, void* stream) {
  Range nvtx_range("mf_bias_layout");
  MF_REQUIRE(rows && planes && L > 0 && np > 0 && H > 0 && float_dtype(dtype), MF_ERR_BAD_ARG, "bad pair-bias layout arguments");
  int r = check_device(); if (r) return r;
  return bias_layout(rows, planes, L, np, H, swap != 0, to_rows != 0, dtype, static_cast<cudaStream_t>(stream));
}

int mf_cast_batch(const mf_cast_item* items, int32_t n_items, void* stream) {
  Range nvtx_range("mf_cast_batch");
  MF_REQUIRE(items && n_items > 0 && n_items <= MF_CAST_MAX, MF_ERR_BAD_ARG, "between 1 and %d arrays are converted at once, got %d", MF_CAST_MAX, n_items);
  for (int i = 0; i < n_items; ++i) {
    MF_REQUIRE(items[i].n >= 0 && (items[i].n == 0 || (items[i].src && items[i].dst)), MF_ERR_BAD_ARG, "array %d: bad size or NULL", i);
    MF_REQUIRE(float_dtype(items[i].src_dtype) && float_dtype(items[i].dst_dtype), MF_ERR_BAD_ARG, "array %d: not a floating type", i);
  }
  int r = check_device(); if (r) return r;
  return cast_batch(items, n_items, static_cast<cudaStream_t>(stream));
}

const char* mf_last_error_string(void) { return last_error_buf(); }
int mf_version(void) { return MF_ABI_VERSION; }
uint64_t mf_kernel_launch_count(void) { return g_launches.load(); }
const char* mf_last_path(void) { return t_last_path; }
int mf_async_status(void) { return tc_async_status(); }

int mf_selftest_bounded_wait(void* stream) {
  int r = check_device(); if (r) return r;
  return bounded_wait_selftest(static_cast<cudaStream_t>(stream));
}

}  // extern "C"
