// LayerNorm backward of a 128-row tile whose gradient behind the normalisation sits in TMEM: shared by the kernels that
// produce that gradient (lnl_bwd_tc.cu, transition_bwd_tc.cu), so that it never goes through memory.
//
// P * 128 threads, thread (row, part): CW = K / P columns of its row.  With w = dyln * gain, xh = (x - mean) * rstd:
//     dx = (w - (mean_k(xh w) * xh + mean_k(w))) * rstd        d_gain += dyln xh        d_shift += dyln   (sums over rows)
// The parts of a row exchange their partial means through shared memory.
#pragma once
#include "evo_tc_common.cuh"

namespace mf {
namespace tcx {

// v[c] of 32 lanes -> the sum over the lanes of v[lane mod CW] (31 shuffles for 32 columns)
template <int CW>
__device__ __forceinline__ float column_sum(float (&v)[CW], int lane) {
#pragma unroll
  for (int s = CW / 2; s > 0; s >>= 1) {
    const bool up = lane & s;
#pragma unroll
    for (int i = 0; i < s; ++i) {
      const float give = up ? v[i] : v[i + s], keep = up ? v[i + s] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, s);
    }
  }
  float t = v[0];
#pragma unroll
  for (int s = CW; s < 32; s <<= 1) t += __shfl_xor_sync(0xffffffffu, t, s);
  return t;
}

// Sums over the rows, formed tile by tile by a transposing butterfly: two registers per 32 columns.
template <int CW> struct ColumnSums {
  float gain[CW / 32], shift[CW / 32];
  __device__ __forceinline__ ColumnSums() {
#pragma unroll
    for (int i = 0; i < CW / 32; ++i) gain[i] = shift[i] = 0.f;
  }
};

// dy: the thread's CW columns of dyln (fp32 bits); raw: the same columns of x; gam: the gain of them (shared memory,
// 16-byte aligned); red: [P][128] float2 of shared memory; `barrier`: a named barrier of the P * 128 threads.
// Rows beyond the last one come with dy = raw = 0 and mu = rs = 0 and contribute nothing.  Results leave NC columns at a
// time, packed: emit(first column / NC, dx); grad(k, d, xh) sees each pair of columns once.
template <typename T, int CW, int P, int NC, typename Emit, typename Grad>
__device__ __forceinline__ void ln_bwd_row(const uint32_t (&dy)[CW], const uint4 (&raw)[CW / 8], float mu, float rs, const float* gam,
                                           float2 (*red)[128], int part, int row, int barrier, Emit emit, Grad grad) {
  const float2 mm = make_float2(mu, mu), rr = make_float2(rs, rs);
  auto xhat = [&](int k) {             // columns k, k + 1 (k a compile-time constant after unrolling)
    const uint4& q = raw[k / 8];
    const uint32_t u = (k / 2) % 4 == 0 ? q.x : (k / 2) % 4 == 1 ? q.y : (k / 2) % 4 == 2 ? q.z : q.w;
    return mul2(sub2(Pack2<T>::unpack(u), mm), rr);
  };
  auto grad_of = [&](int k) { return make_float2(__uint_as_float(dy[k]), __uint_as_float(dy[k + 1])); };
  float2 c1p = make_float2(0.f, 0.f), c2p = c1p;
#pragma unroll
  for (int k = 0; k < CW; k += 4) {
    const float4 g = *reinterpret_cast<const float4*>(gam + k);
    const float2 w0 = mul2(grad_of(k), make_float2(g.x, g.y)), w1 = mul2(grad_of(k + 2), make_float2(g.z, g.w));
    c1p = fma2(xhat(k), w0, c1p); c1p = fma2(xhat(k + 2), w1, c1p);
    c2p = add2(c2p, add2(w0, w1));
  }
  red[part][row] = make_float2(c1p.x + c1p.y, c2p.x + c2p.y);
  named_sync(barrier, P * 128);
  float c1 = 0.f, c2 = 0.f;
#pragma unroll
  for (int i = 0; i < P; ++i) { const float2 o = red[i][row]; c1 += o.x; c2 += o.y; }
  named_sync(barrier, P * 128);              // everybody has read before the next tile writes
  constexpr float inv_k = 1.f / (CW * P);
  const float2 cc1 = make_float2(-c1 * inv_k, -c1 * inv_k), cc2 = make_float2(-c2 * inv_k, -c2 * inv_k);
#pragma unroll
  for (int n = 0; n < CW; n += NC) {
    uint32_t o[NC / 2];
#pragma unroll
    for (int i = 0; i < NC; i += 4) {
      const float4 g = *reinterpret_cast<const float4*>(gam + n + i);
#pragma unroll
      for (int e = 0; e < 4; e += 2) {
        const int k = n + i + e;
        const float2 h = xhat(k), d = grad_of(k), gg = e ? make_float2(g.z, g.w) : make_float2(g.x, g.y);
        const float2 z = mul2(fma2(d, gg, fma2(cc1, h, cc2)), rr);
        o[(i + e) / 2] = Pack2<T>::pack(z.x, z.y);
        grad(k, d, h);
      }
    }
    emit(n / NC, o);
  }
}

// TMA stores of staged tiles and their bulk groups
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* m, const void* src, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(src)), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void bulk_commit_group() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void bulk_wait_group_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
template <int N> __device__ __forceinline__ void bulk_wait_group() {
  asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}

}  // namespace tcx
}  // namespace mf
