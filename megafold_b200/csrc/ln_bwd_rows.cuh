// LayerNorm backward of a 128-row tile whose gradient behind the normalisation sits in TMEM: shared by the kernels that
// produce that gradient, so that it never goes through memory.
//
// P * 128 threads, thread (row, part): CW = K / P columns of its row.  With w = dyln * gain, xh = (x - mean) * rstd:
//     dx = (w - (mean_k(xh w) * xh + mean_k(w))) * rstd        d_gain += dyln xh   (a sum over rows)
// The parts of a row exchange sums of four neighbouring columns through shared memory, and every part adds them up in the
// order of the row-pass kernel (lnl_ops.cu: four columns per lane, then a butterfly over the lanes), each step with that
// kernel's rounding.  dx is thereby the same bit for bit whichever kernel a size takes.  Where it matters: the gradient of
// the shift of a pair-bias projection is 0 up to the rounding of d_pair_bias (the logit gradients of a softmax sum to 0), so
// one flipped bit of dx makes it another number.
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

// dy: the thread's CW columns of dyln (fp32 bits); raw: the same columns of x; gam: the gain of them (shared memory,
// 16-byte aligned); red: [P][CW / 8][128] float4 of shared memory; `barrier`: a named barrier of the P * 128 threads.
// Rows beyond the last one come with dy = raw = 0 and mu = rs = 0 and contribute nothing.  The result leaves packed through
// emit(dx); grad(k, d, xh) sees each pair of columns once.
template <typename T, int CW, int P, typename Emit, typename Grad>
__device__ __forceinline__ void ln_bwd_row(const uint32_t (&dy)[CW], const uint4 (&raw)[CW / 8], float mu, float rs, const float* gam,
                                           float4 (*red)[CW / 8][128], int part, int row, int barrier, Emit emit, Grad grad) {
  const float2 mm = make_float2(mu, mu), rr = make_float2(rs, rs);
  auto xhat = [&](int k) {             // columns k, k + 1 (k a compile-time constant after unrolling)
    const uint4& q = raw[k / 8];
    const uint32_t u = (k / 2) % 4 == 0 ? q.x : (k / 2) % 4 == 1 ? q.y : (k / 2) % 4 == 2 ? q.z : q.w;
    return mul2(sub2(Pack2<T>::unpack(u), mm), rr);
  };
  auto grad_of = [&](int k) { return make_float2(__uint_as_float(dy[k]), __uint_as_float(dy[k + 1])); };
  constexpr int G = CW / 4;                  // groups of four columns
  float s1[G], s2[G];
#pragma unroll
  for (int i = 0; i < G; ++i) {
    const int k = i * 4;
    const float4 g = *reinterpret_cast<const float4*>(gam + k);
    const float2 w0 = mul2(grad_of(k), make_float2(g.x, g.y)), w1 = mul2(grad_of(k + 2), make_float2(g.z, g.w)), h0 = xhat(k), h1 = xhat(k + 2);
    s1[i] = __fmaf_rn(h1.y, w1.y, __fmaf_rn(h1.x, w1.x, __fmaf_rn(h0.y, w0.y, __fmul_rn(h0.x, w0.x))));
    s2[i] = __fadd_rn(__fadd_rn(__fadd_rn(w0.x, w0.y), w1.x), w1.y);
  }
#pragma unroll
  for (int i = 0; i < G / 4; ++i) {
    red[part][i][row] = make_float4(s1[4 * i], s1[4 * i + 1], s1[4 * i + 2], s1[4 * i + 3]);
    red[part][G / 4 + i][row] = make_float4(s2[4 * i], s2[4 * i + 1], s2[4 * i + 2], s2[4 * i + 3]);
  }
  named_sync(barrier, P * 128);
  auto total = [&](int at) {                 // the butterfly: parts 0 + 2 and 1 + 3, then these, then the halves of a part's groups
    static_assert(P == 4, "four parts");
    float u[G];
#pragma unroll
    for (int i = 0; i < G / 4; ++i) {
      const float4 a = red[0][at + i][row], b = red[1][at + i][row], c = red[2][at + i][row], d = red[3][at + i][row];
      u[4 * i] = __fadd_rn(__fadd_rn(a.x, c.x), __fadd_rn(b.x, d.x)); u[4 * i + 1] = __fadd_rn(__fadd_rn(a.y, c.y), __fadd_rn(b.y, d.y));
      u[4 * i + 2] = __fadd_rn(__fadd_rn(a.z, c.z), __fadd_rn(b.z, d.z)); u[4 * i + 3] = __fadd_rn(__fadd_rn(a.w, c.w), __fadd_rn(b.w, d.w));
    }
#pragma unroll
    for (int h = G / 2; h > 0; h >>= 1)
#pragma unroll
      for (int i = 0; i < h; ++i) u[i] = __fadd_rn(u[i], u[i + h]);
    return u[0];
  };
  constexpr float inv_k = 1.f / (CW * P);
  const float c1 = __fmul_rn(total(0), inv_k), c2 = __fmul_rn(total(G / 4), inv_k);
  named_sync(barrier, P * 128);              // everybody has read before the next tile writes
  uint32_t o[CW / 2];
#pragma unroll
  for (int i = 0; i < CW; i += 4) {
    const float4 g = *reinterpret_cast<const float4*>(gam + i);
#pragma unroll
    for (int e = 0; e < 4; e += 2) {
      const int k = i + e;
      const float2 h = xhat(k), d = grad_of(k);
      const float2 t = make_float2(__fadd_rn(__fmul_rn(c1, h.x), c2), __fadd_rn(__fmul_rn(c1, h.y), c2));      // (packed, the two would be fused)
      const float2 z = mul2(fma2(d, e ? make_float2(g.z, g.w) : make_float2(g.x, g.y), make_float2(-t.x, -t.y)), rr);
      o[k / 2] = Pack2<T>::pack(z.x, z.y);
      grad(k, d, h);
    }
  }
  emit(o);
}

// The same for two threads a row of 128 columns: thread `part` has the 32-column quarters part and part + 2 in registers (dy:
// 32 columns of each).  at(q, c): where the raw columns 8 c .. 8 c + 7 of its q-th quarter lie in shared memory; dx replaces
// them.  sums: the gain and shift sums of the 32 rows so far, [2][128].  red: [2 parts][4][128] float4; `barrier`: a named barrier
// of the two warps that share 32 rows.
template <typename T, typename At>
__device__ __forceinline__ void ln_bwd_half_row(uint32_t (&dy)[64], float mu, float rs, const float* gam, float* sums, float4 (*red)[4][128],
                                                int part, int row, int lane, int barrier, At at) {
  const float2 mm = make_float2(mu, mu), rr = make_float2(rs, rs);
  auto xhat = [&](uint32_t u) { return mul2(sub2(Pack2<T>::unpack(u), mm), rr); };
  auto grad_of = [&](int k) { return make_float2(__uint_as_float(dy[k]), __uint_as_float(dy[k + 1])); };
  const float* g_of[2] = {gam + part * 32, gam + part * 32 + 64};
  // sums of four neighbouring columns, of groups i, i + 16 and i + 8, i + 24, then a tree over i: the butterfly's order
  float a1[8], a2[8];
#pragma unroll
  for (int j = 0; j < 4; ++j) {              // groups 2 j and 2 j + 1 of each quarter
    float q1[2][2], q2[2][2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const uint4 raw = *at(q, j);
      const uint32_t u[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = j * 8 + h * 4, k = q * 32 + c;
        const float4 g = *reinterpret_cast<const float4*>(g_of[q] + c);
        const float2 w0 = mul2(grad_of(k), make_float2(g.x, g.y)), w1 = mul2(grad_of(k + 2), make_float2(g.z, g.w)), h0 = xhat(u[2 * h]), h1 = xhat(u[2 * h + 1]);
        q1[q][h] = __fmaf_rn(h1.y, w1.y, __fmaf_rn(h1.x, w1.x, __fmaf_rn(h0.y, w0.y, __fmul_rn(h0.x, w0.x))));
        q2[q][h] = __fadd_rn(__fadd_rn(__fadd_rn(w0.x, w0.y), w1.x), w1.y);
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      a1[2 * j + h] = __fadd_rn(q1[0][h], q1[1][h]);
      a2[2 * j + h] = __fadd_rn(q2[0][h], q2[1][h]);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    red[part][i][row] = make_float4(a1[4 * i], a1[4 * i + 1], a1[4 * i + 2], a1[4 * i + 3]);
    red[part][2 + i][row] = make_float4(a2[4 * i], a2[4 * i + 1], a2[4 * i + 2], a2[4 * i + 3]);
  }
  named_sync(barrier, 64);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float4 x = red[part ^ 1][i][row], y = red[part ^ 1][2 + i][row];
    a1[4 * i] = __fadd_rn(a1[4 * i], x.x); a1[4 * i + 1] = __fadd_rn(a1[4 * i + 1], x.y); a1[4 * i + 2] = __fadd_rn(a1[4 * i + 2], x.z); a1[4 * i + 3] = __fadd_rn(a1[4 * i + 3], x.w);
    a2[4 * i] = __fadd_rn(a2[4 * i], y.x); a2[4 * i + 1] = __fadd_rn(a2[4 * i + 1], y.y); a2[4 * i + 2] = __fadd_rn(a2[4 * i + 2], y.z); a2[4 * i + 3] = __fadd_rn(a2[4 * i + 3], y.w);
  }
  named_sync(barrier, 64);                   // both have read before the next tile writes
#pragma unroll
  for (int h = 4; h > 0; h >>= 1)
#pragma unroll
    for (int i = 0; i < h; ++i) { a1[i] = __fadd_rn(a1[i], a1[i + h]); a2[i] = __fadd_rn(a2[i], a2[i + h]); }
  constexpr float inv_k = 1.f / 128;
  const float c1 = __fmul_rn(a1[0], inv_k), c2 = __fmul_rn(a2[0], inv_k);
  // 32 columns at a time: dx, and the first step of both column sums (columns k and k + 16 of the block) while they are at hand
  auto fold = [&](float a, float b, int s) {
    const bool up = lane & s;
    return (up ? b : a) + __shfl_xor_sync(0xffffffffu, up ? a : b, s);
  };
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    float vg[16], vs[16];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      float p[2][8];
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint4* slot = at(q, half * 2 + j);
        const uint4 raw = *slot;
        const uint32_t u[4] = {raw.x, raw.y, raw.z, raw.w};
        uint32_t o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int c = half * 16 + j * 8 + e * 2, k = q * 32 + c;
          const float2 g = *reinterpret_cast<const float2*>(g_of[q] + c), h = xhat(u[e]), d = grad_of(k);
          const float2 t = make_float2(__fadd_rn(__fmul_rn(c1, h.x), c2), __fadd_rn(__fmul_rn(c1, h.y), c2));      // (packed, the two would be fused)
          const float2 z = mul2(fma2(d, g, make_float2(-t.x, -t.y)), rr);
          o[e] = Pack2<T>::pack(z.x, z.y);
          const float2 dh = mul2(d, h);
          p[half][e * 2] = dh.x; p[half][e * 2 + 1] = dh.y;
        }
        *slot = make_uint4(o[0], o[1], o[2], o[3]);
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        vg[j * 8 + e] = fold(p[0][e], p[1][e], 16);
        vs[j * 8 + e] = fold(__uint_as_float(dy[q * 32 + j * 8 + e]), __uint_as_float(dy[q * 32 + 16 + j * 8 + e]), 16);
      }
    }
#pragma unroll
    for (int s = 8; s > 0; s >>= 1)
#pragma unroll
      for (int i = 0; i < s; ++i) { vg[i] = fold(vg[i], vg[i + s], s); vs[i] = fold(vs[i], vs[i + s], s); }
    sums[(part + 2 * q) * 32 + lane] += vg[0];
    sums[128 + (part + 2 * q) * 32 + lane] += vs[0];
  }
}

}  // namespace tcx
}  // namespace mf
