// Host-side support shared by the tensor-core attention kernels: status word, device queries and the
// test that decides whether a call can take the tensor-core path.
#include <type_traits>

#include "evo_tc_common.cuh"

namespace mf {
namespace tcx {

StatusWord* status_slot() {
  static std::mutex mu;
  static StatusWord words[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> lk(mu);
  StatusWord& w = words[dev];
  if (!w.host) {
    if (cudaHostAlloc(&w.host, sizeof(int), cudaHostAllocMapped) != cudaSuccess) { w.host = nullptr; return nullptr; }
    *w.host = 0;
    if (cudaHostGetDevicePointer(&w.dev, w.host, 0) != cudaSuccess) return nullptr;
  }
  return &w;
}

#ifdef MF_TRACE
long long* g_trace = nullptr;
#endif

int sm_count() {
  static int n[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return 148;
  if (!n[dev]) cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev);
  return n[dev] > 0 ? n[dev] : 148;
}

}  // namespace tcx

namespace {
// Rows of the pair bias to a pitch that TMA can address, in a 16-bit type.  A thread writes one 16-byte piece of a row;
// where the source allows it reads 16-byte pieces too, otherwise element by element (neighbouring threads read
// neighbouring pieces, so the lines are shared).  Bound: HBM, and at crop sizes latency: [4, 467, 467] bf16 (1.7 MB) takes
// 3 us, against 1000 us more in the general attention kernel that reads such a bias in place.
//
// The kernels that read the copy add it by a product with a multiple of the identity, where an infinite value times 0 would
// make its neighbours NaN.  So infinities (and fp32 values beyond the range of the copy) become the largest value that stays
// finite there: probability 0 for -inf, as it should be.
template <typename TO>
__device__ __forceinline__ TO bounded(float v) {
  constexpr float lim = std::is_same_v<TO, __half> ? 65504.f : -tcx::kMinusBig;
  return from_f<TO>(v < -lim ? -lim : v > lim ? lim : v);      // NaN stays
}
template <typename TB, typename TO>
__global__ void __launch_bounds__(256) copy_bias_rows_kernel(const TB* __restrict__ bias, TO* __restrict__ dst, int64_t pieces, int L, int per_row, int H,
                                                             int64_t sb, int64_t sh, int64_t si, int64_t sj, bool vec) {
  const int64_t q = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (q >= pieces) return;
  const int64_t row = q / per_row;                 // (b * H + h) * L + i
  const int j0 = (int)(q - row * per_row) * 8;
  const int64_t bh = row / L;
  const int i = (int)(row - bh * L);
  const TB* src = bias + bh / H * sb + bh % H * sh + i * si + j0 * sj;
  __align__(16) TO out[8];
  if (vec && j0 + 8 <= L) {
    __align__(16) TB in[8];
#pragma unroll
    for (int k = 0; k < (int)(8 * sizeof(TB) / 16); ++k) reinterpret_cast<uint4*>(in)[k] = __ldg(reinterpret_cast<const uint4*>(src) + k);
#pragma unroll
    for (int k = 0; k < 8; ++k) out[k] = bounded<TO>(to_f(in[k]));
  } else {
#pragma unroll
    for (int k = 0; k < 8; ++k) out[k] = bounded<TO>(j0 + k < L ? to_f(src[k * sj]) : 0.f);
  }
  *reinterpret_cast<uint4*>(dst + q * 8) = *reinterpret_cast<const uint4*>(out);
}

// One CTA waits, with a short cap, on an mbarrier that nobody completes, then takes the same exit path as the
// attention kernels: raise the CTA's flag, report through the status word, return normally.
__global__ void bounded_wait_selftest_kernel(int* status, int cap) {
  __shared__ uint64_t bar;
  __shared__ int abort_s;
  if (threadIdx.x == 0) { abort_s = 0; tc::mbar_init(&bar, 1); tc::mbar_fence_init(); }
  __syncthreads();
  bool done = false;
  for (int i = 0; i < cap && !done; ++i) done = tc::mbar_try_wait(&bar, 0);
  if (!done) abort_s = 1;
  __syncthreads();
  if (threadIdx.x == 0 && abort_s) *reinterpret_cast<volatile int*>(status) = 1;
}
}  // namespace

namespace tcx {
int copy_bias_rows(const void* bias, int dtype, const int64_t* s, void* dst, int dst_dtype, int B, int H, int L, cudaStream_t st) {
  const int per_row = bias_pitch(L) / 8;
  const int64_t pieces = (int64_t)bias_copies(s, B) * H * L * per_row;
  const unsigned grid = (unsigned)((pieces + 255) / 256);
  const int64_t es = (int64_t)dtype_size(dtype);
  const bool vec = s[3] == 1 && (reinterpret_cast<uintptr_t>(bias) & 15) == 0 && (s[0] * es) % 16 == 0 && (s[1] * es) % 16 == 0 && (s[2] * es) % 16 == 0;
  MF_DISPATCH_FLOAT(dtype, TB, {
    if (dst_dtype == MF_BF16)
      copy_bias_rows_kernel<TB, __nv_bfloat16><<<grid, 256, 0, st>>>(static_cast<const TB*>(bias), static_cast<__nv_bfloat16*>(dst), pieces, L, per_row, H, s[0], s[1], s[2], s[3], vec);
    else
      copy_bias_rows_kernel<TB, __half><<<grid, 256, 0, st>>>(static_cast<const TB*>(bias), static_cast<__half*>(dst), pieces, L, per_row, H, s[0], s[1], s[2], s[3], vec);
    MF_LAUNCHED("copy_bias_rows_kernel");
  });
  return MF_OK;
}
}  // namespace tcx

int bounded_wait_selftest(cudaStream_t st) {
  int* status = tcx::status_word();
  MF_REQUIRE(status, MF_ERR_CUDA, "could not allocate the device status word");
  bounded_wait_selftest_kernel<<<1, 128, 0, st>>>(status, 2048);
  MF_LAUNCHED("bounded_wait_selftest_kernel");
  return MF_OK;
}

int tc_async_status() {
  tcx::StatusWord* w = tcx::status_slot();
  return (w && w->host) ? *reinterpret_cast<volatile int*>(w->host) : 0;
}

bool evo_tc_supported(int B, int N, int L, int H, int D, int dtype, const int64_t* qs, const int64_t* ks,
                      const int64_t* vs, const void* q, const void* k, const void* v) {
  if (dtype != MF_BF16 && dtype != MF_F16) return false;
  if (D % 8 != 0 || D > 64 || L > 4096) return false;
  return tcx::qkv_strides_ok(q, qs, B, N, L, H) && tcx::qkv_strides_ok(k, ks, B, N, L, H) &&
         tcx::qkv_strides_ok(v, vs, B, N, L, H);
}

}  // namespace mf

#ifdef MF_TRACE
// debug builds only: device buffer of 8 * kTraceLen 64-bit words that the attention kernels' phase trace is written to
extern "C" __attribute__((visibility("default"))) void mf_debug_set_trace(long long* p) { mf::tcx::g_trace = p; }
#endif
