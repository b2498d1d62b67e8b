// LayerNorm fused into a product on the tensor cores for rows of 192 to 384 elements (the single representation's widths;
// K a multiple of 64, 16-bit types):
//
//     mode 0 (LayernormLinear forward)       Y = LN(X) W + b
//     mode 1 (first half of the Transition)  G = silu(H_gate) * H_value,  H = LN(X) W1
//
// These sizes ran on CUDA cores with LN(x) in fp32, so the product here takes LN(x) as the sum of two 16-bit terms (hi, then
// the rounding error lo through the same shared-memory tile): nothing is rounded that was not before.  The tensor pipe
// has the room: a [768, 384] x 1536 call is bound by launch and load latency.
//
// A CTA owns a 128-row tile and R blocks of 64 output columns (R chosen so that the grid fills the chip once, up to the 512
// TMEM columns).  256 threads:
//   1. TMA brings the rows (K-major, 128B swizzle) and the first two blocks of W (MN-major);
//   2. thread (row, half) reads its half row into registers, forms mean and variance in two passes with its partner, writes
//      the 16-bit LN(x) back in place; one lane issues the products of all R blocks as their W arrives;
//   3. when these are done the threads write the lo terms over the tile and the products run again (W again from the ring);
//   4. epilogue: bias, or value x silu(gate), to 16 bit through swizzled slabs and TMA stores.
// Every wait is bounded; on expiry the CTA raises a flag, drains and reports through mf_async_status().
//
// Measured: [768, 384] -> 1536 12 us (46 on CUDA cores), the whole Transition forward of [768, 384], inner 1536, 26 (228).
#include <type_traits>

#include "gemm_tc.cuh"
#include "ln_bwd_rows.cuh"

namespace mf {
namespace {
using namespace tcx;

constexpr int kRows = 128, kThreads = 256, kNB = 64, kMaxR = 8;

struct WideP {
  int64_t M; int N, n_blocks, R, inner;
  float eps;
  uint32_t ab_fmt, tmem_cols;
  const void *gamma, *beta, *bias;
  float *mean, *rstd;
  int* status;
};

struct Bars { uint64_t x_full, w_full[2], w_empty[2], done; };

// The hi terms of LN(x).  A value beyond fp16 becomes the largest one, so that its lo term is what is missing and not inf - inf;
// NaN stays NaN.  (With comparisons instead of the saturating conversion: 140 -> 147 us at [20000, 384] -> 1536.)
template <typename T>
__device__ __forceinline__ uint32_t pack_finite(float a, float b) {
  if constexpr (std::is_same_v<T, __half>) {
    uint32_t r;
    asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
  } else {
    return Pack2<T>::pack(a, b);
  }
}

template <int K, int MODE, typename T>
__global__ void __launch_bounds__(kThreads, 1)
ln_wide_kernel(const __grid_constant__ CUtensorMap mx, const __grid_constant__ CUtensorMap mw, const __grid_constant__ CUtensorMap my, const WideP p) {
  constexpr int kAtomB = kRows * 128;                // [128 rows][64 columns]
  constexpr int kWB = K * 128;                       // a block of W: [K][64], or [K][32] of value and of gate columns
  constexpr int CH = K / 16;                         // 16-byte chunks of a thread's half row
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sA = smem;                                // [K / 64] atoms
  uint8_t* sW = smem + K / 64 * kAtomB;              // two blocks
  __shared__ Bars bar;
  __shared__ __align__(16) float gam_s[K], bet_s[K];
  __shared__ float part_s[2][kRows];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row0 = blockIdx.x * kRows, b0 = blockIdx.y * p.R;
  const int nb = p.n_blocks - b0 < p.R ? p.n_blocks - b0 : p.R;      // my blocks of columns
  if (tid == 0) {
    abort_s = 0;
    mbar_init(&bar.x_full, 1); mbar_init(&bar.done, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(&bar.w_full[i], 1); mbar_init(&bar.w_empty[i], 1); }
    mbar_fence_init();
    mbar_expect_tx(&bar.x_full, K / 64 * kAtomB);
#pragma unroll
    for (int at = 0; at < K / 64; ++at) tma_load_2d(sA + at * kAtomB, &mx, &bar.x_full, at * 64, row0);
  }
  for (int k = tid; k < K; k += kThreads) {
    gam_s[k] = to_f(static_cast<const T*>(p.gamma)[k]);
    bet_s[k] = p.beta ? to_f(static_cast<const T*>(p.beta)[k]) : 0.f;
  }
  if (warp == 0) { tmem_alloc(&tmem_base_s, p.tmem_cols); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  volatile int* abort_flag = &abort_s;
  const uint32_t tm0 = tmem_base_s;

  // block u of the 2 nb passes over W (hi terms, then lo terms)
  int loaded = 0;                                    // blocks requested (thread 0)
  auto load_w = [&](int u) {
    loaded = u + 1;
    uint8_t* w = sW + (u & 1) * kWB;
    const int blk = b0 + u % nb;
    mbar_expect_tx(&bar.w_full[u & 1], kWB);
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {                 // a box has at most 256 rows
      if constexpr (MODE == 0) {
        tma_load_2d(w + hf * (kWB / 2), &mw, &bar.w_full[u & 1], blk * 64, hf * (K / 2));
      } else {
        tma_load_2d(w + hf * (kWB / 4), &mw, &bar.w_full[u & 1], blk * 32, hf * (K / 2));
        tma_load_2d(w + kWB / 2 + hf * (kWB / 4), &mw, &bar.w_full[u & 1], p.inner + blk * 32, hf * (K / 2));
      }
    }
  };
  // The issuing thread runs the products of one pass; W blocks beyond the two that fit are fetched as stages fall free.
  const uint32_t idesc = idesc_f16(128, kNB, p.ab_fmt, 0, 1);
  auto issue = [&](int pass) {
    for (int i = 0; i < nb; ++i) {
      const int u = pass * nb + i;
      wait_or_flag(&bar.w_full[u & 1], (u >> 1) & 1, abort_flag);
      tc_fence_after();
      if (*abort_flag) return;
      const uint32_t a_lo = desc_lo(smem_u32(sA), 16);
      const uint32_t w_lo = desc_lo(smem_u32(sW + (u & 1) * kWB), MODE == 0 ? 16 : kWB / 2);
      constexpr uint32_t w_hi = MODE == 0 ? desc_hi(1024, kSw128) : desc_hi(512, kSw64);
      constexpr uint32_t w_step = (MODE == 0 ? 2048 : 1024) / 16;
#pragma unroll
      for (int ks = 0; ks < K / 16; ++ks)
        mma_ss_lh(tm0 + i * kNB, a_lo + (ks >> 2) * (kAtomB / 16) + (ks & 3) * 2, desc_hi(1024, kSw128), w_lo + ks * w_step, w_hi, idesc, pass > 0 || ks > 0);
      tc_commit(&bar.w_empty[u & 1]);
      if (u + 2 < 2 * nb) {
        wait_or_flag(&bar.w_empty[u & 1], (u >> 1) & 1, abort_flag);
        if (*abort_flag) return;
        load_w(u + 2);
      }
    }
    tc_commit(&bar.done);
  };
  if (tid == 0) { load_w(0); if (2 * nb > 1) load_w(1); }

  // ---- LayerNorm: thread (row, half) owns CH chunks of its row, kept raw in registers for the lo terms
  const int row_l = (warp & 3) * 32 + lane, half = warp >> 2;
  const int64_t row = (int64_t)row0 + row_l;
  const bool ok = row < p.M;
  auto chunk = [&](int c) {            // chunk c of my half row: atom and swizzled place
    const int g = half * CH + c;
    return reinterpret_cast<uint4*>(sA + (g >> 3) * kAtomB + swz_offset(row_l, g & 7, 128));
  };
  wait_or_flag(&bar.x_full, 0, abort_flag);
  uint4 raw[CH];
  float2 s2 = make_float2(0.f, 0.f);
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    raw[c] = *chunk(c);
    s2 = add2(s2, add2(add2(Pack2<T>::unpack(raw[c].x), Pack2<T>::unpack(raw[c].y)), add2(Pack2<T>::unpack(raw[c].z), Pack2<T>::unpack(raw[c].w))));
  }
  part_s[half][row_l] = s2.x + s2.y;
  __syncthreads();
  const float mu = (part_s[0][row_l] + part_s[1][row_l]) * (1.f / K);
  __syncthreads();
  const float2 mm = make_float2(mu, mu);
  float2 v2 = make_float2(0.f, 0.f);
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const uint32_t u[4] = {raw[c].x, raw[c].y, raw[c].z, raw[c].w};
#pragma unroll
    for (int e = 0; e < 4; ++e) { const float2 d = sub2(Pack2<T>::unpack(u[e]), mm); v2 = fma2(d, d, v2); }
  }
  part_s[half][row_l] = v2.x + v2.y;
  __syncthreads();
  const float rs = rsqrtf((part_s[0][row_l] + part_s[1][row_l]) * (1.f / K) + p.eps);
  if (ok && blockIdx.y == 0 && half == 0) { p.mean[row] = mu; p.rstd[row] = rs; }
  const float2 rr = make_float2(rs, rs);
  auto write_terms = [&](bool lo) {
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const uint32_t u[4] = {raw[c].x, raw[c].y, raw[c].z, raw[c].w};
      uint32_t o[4];
#pragma unroll
      for (int e = 0; e < 4; e += 2) {
        const int k = (half * CH + c) * 8 + e * 2;
        const float4 g = *reinterpret_cast<const float4*>(gam_s + k), b = *reinterpret_cast<const float4*>(bet_s + k);
        float2 y[2] = {fma2(mul2(sub2(Pack2<T>::unpack(u[e]), mm), rr), make_float2(g.x, g.y), make_float2(b.x, b.y)),
                       fma2(mul2(sub2(Pack2<T>::unpack(u[e + 1]), mm), rr), make_float2(g.z, g.w), make_float2(b.z, b.w))};
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          uint32_t w = pack_finite<T>(y[i].x, y[i].y);
          if (lo) { const float2 d = sub2(y[i], Pack2<T>::unpack(w)); w = Pack2<T>::pack(d.x, d.y); }
          o[e + i] = ok ? w : 0u;
        }
      }
      *chunk(c) = make_uint4(o[0], o[1], o[2], o[3]);
    }
    fence_async_smem();
    __syncthreads();
  };
  write_terms(false);
  if (tid == 0) issue(0);
  __syncwarp();
  wait_or_flag(&bar.done, 0, abort_flag);            // the hi products have read the tile
  write_terms(true);
  if (tid == 0) issue(1);
  __syncwarp();
  wait_or_flag(&bar.done, 1, abort_flag);
  tc_fence_after();

  // ---- epilogue: the tile of X is free: warp (rows, half of the block's columns) stages its own slabs there, two in turn
  const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
  constexpr int OC = MODE == 0 ? 32 : 16;            // output columns per thread and block
  uint8_t* slabs = sA + warp * 2 * 2048;
  for (int i = 0; i < nb; ++i) {
    const int n0 = MODE == 0 ? (b0 + i) * 64 + half * 32 : (b0 + i) * 32 + half * 16;
    uint32_t out[OC / 2];
    if constexpr (MODE == 0) {
      uint32_t acc[32];
      tmem_ld32(tm0 + i * kNB + half * 32 + lane_addr, acc);
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const int n = n0 + 2 * e;
        const T* bias = static_cast<const T*>(p.bias);
        const float ba = bias && n < p.N ? to_f(bias[n]) : 0.f, bb = bias && n + 1 < p.N ? to_f(bias[n + 1]) : 0.f;
        out[e] = Pack2<T>::pack(__uint_as_float(acc[2 * e]) + ba, __uint_as_float(acc[2 * e + 1]) + bb);
      }
    } else {
      uint32_t hv[16], hg[16];
      tmem_ld16(tm0 + i * kNB + half * 16 + lane_addr, hv);
      tmem_ld16(tm0 + i * kNB + 32 + half * 16 + lane_addr, hg);
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        float g[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float b = __uint_as_float(hg[2 * e + q]);
          // exp(-b) beyond 2^126 divides to 0, and an infinite b to NaN, which the product with the value carries on
          g[q] = __fdividef(b, 1.f + __expf(-b)) * __uint_as_float(hv[2 * e + q]);
        }
        out[e] = Pack2<T>::pack(g[0], g[1]);
      }
    }
    uint8_t* slab = slabs + (i & 1) * 2048;
    if (lane == 0) bulk_wait_group_read<1>();
    __syncwarp();
    if (__any_sync(0xffffffffu, *abort_flag)) break;
#pragma unroll
    for (int c = 0; c < OC / 8; ++c)
      *reinterpret_cast<uint4*>(slab + swz_offset(lane, c, OC * 2)) = make_uint4(out[c * 4], out[c * 4 + 1], out[c * 4 + 2], out[c * 4 + 3]);
    fence_async_smem();
    __syncwarp();
    if (lane == 0) {
      const int r0 = row0 + (warp & 3) * 32;
      if (n0 < (MODE == 0 ? p.N : p.inner) && r0 < p.M) tma_store_2d(&my, slab, n0, r0);      // never start past an edge
      bulk_commit_group();
    }
  }
  if (lane == 0) bulk_wait_group<0>();
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && abort_s) {
    // copies already requested must land before the shared memory is given back (bounded)
    mbar_wait(&bar.x_full, 0);
    for (int u = loaded > 2 ? loaded - 2 : 0; u < loaded; ++u) mbar_wait(&bar.w_full[u & 1], (u >> 1) & 1);
    *reinterpret_cast<volatile int*>(p.status) = 1;
  }
  if (warp == 0) tmem_dealloc(tmem_base_s, p.tmem_cols);
}

struct WideArgs { int64_t M; int N, inner, dtype; float eps; const void *x, *gamma, *beta, *w, *bias; void* out; float *mean, *rstd; };

template <int K, int MODE, typename T>
int launch(const WideArgs& a, cudaStream_t st) {
  CUtensorMap mx, mw, my;
  int r;
  {
    const int64_t dims[2] = {K, a.M}, str[2] = {1, K};
    const int box[2] = {64, kRows};
    if ((r = make_tiled_map(&mx, a.x, a.dtype, 2, dims, str, box, 128))) return r;
  }
  const int64_t wn = MODE == 0 ? a.N : 2 * (int64_t)a.inner;
  {
    const int64_t dims[2] = {wn, K}, str[2] = {1, wn};
    const int box[2] = {MODE == 0 ? 64 : 32, K / 2};
    if ((r = make_tiled_map(&mw, a.w, a.dtype, 2, dims, str, box, box[0] * 2))) return r;
  }
  {
    const int64_t on = MODE == 0 ? a.N : a.inner;
    const int64_t dims[2] = {on, a.M}, str[2] = {1, on};
    const int box[2] = {MODE == 0 ? 32 : 16, 32};
    if ((r = make_tiled_map(&my, a.out, a.dtype, 2, dims, str, box, box[0] * 2))) return r;
  }
  WideP p{};
  p.M = a.M; p.N = a.N; p.inner = a.inner; p.eps = a.eps;
  p.n_blocks = MODE == 0 ? (a.N + kNB - 1) / kNB : a.inner / 32;
  const int64_t m_tiles = (a.M + kRows - 1) / kRows;
  int64_t R = (m_tiles * p.n_blocks + sm_count() - 1) / sm_count();
  p.R = (int)(R > kMaxR ? kMaxR : R < 1 ? 1 : R);
  p.tmem_cols = 64;
  while ((int)p.tmem_cols < p.R * kNB) p.tmem_cols *= 2;
  p.ab_fmt = a.dtype == MF_BF16 ? 1u : 0u;
  p.gamma = a.gamma; p.beta = a.beta; p.bias = a.bias; p.mean = a.mean; p.rstd = a.rstd;
  p.status = status_word();
  MF_REQUIRE(p.status, MF_ERR_CUDA, "could not allocate the device status word");
  MF_REQUIRE(tc_async_status() == 0, MF_ERR_CUDA, "an earlier tensor-core kernel gave up on a bounded wait; results are invalid");
  constexpr size_t smem = 1024 + (size_t)K / 64 * kRows * 128 + 2 * (size_t)K * 128;
  constexpr auto kern = ln_wide_kernel<K, MODE, T>;
  if (int e = opt_in_smem<kern>(smem)) return e;
  kern<<<dim3((unsigned)m_tiles, (p.n_blocks + p.R - 1) / p.R), kThreads, smem, st>>>(mx, mw, my, p);
  MF_LAUNCHED("ln_wide_kernel");
  return MF_OK;
}

template <int MODE>
int dispatch(int K, const WideArgs& a, cudaStream_t st) {
#define MF_WIDE(KK) case KK: return a.dtype == MF_BF16 ? launch<KK, MODE, __nv_bfloat16>(a, st) : launch<KK, MODE, __half>(a, st)
  switch (K) { MF_WIDE(192); MF_WIDE(256); MF_WIDE(320); MF_WIDE(384); }
#undef MF_WIDE
  return fail(MF_ERR_UNSUPPORTED, "row width %d", K);
}

bool wide_ok(int64_t M, int K, int dtype) {
  return (dtype == MF_BF16 || dtype == MF_F16) && K >= 192 && K <= 384 && K % 64 == 0 && M >= 1 && M <= (int64_t)INT32_MAX - kRows;
}

}  // namespace

bool lnl_fwd_wide_supported(const mf_lnl_fwd_args& a) {
  const uintptr_t al = reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.w) | reinterpret_cast<uintptr_t>(a.y);
  return wide_ok(a.M, a.K, a.dtype) && a.N % 8 == 0 && (al & 15) == 0;
}
int lnl_fwd_wide(const mf_lnl_fwd_args& a, cudaStream_t st) {
  return dispatch<0>(a.K, WideArgs{a.M, a.N, 0, a.dtype, a.eps, a.x, a.ln_w, a.ln_b, a.w, a.b, a.y, a.mean, a.rstd}, st);
}

// The workspace, which TMA writes, needs the alignment that the CUDA-core path, with a workspace of the same size, does without.
bool transition_fwd_wide_supported(const mf_transition_fwd_args& a) {
  const uintptr_t al = reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.w1) | reinterpret_cast<uintptr_t>(a.w2) | reinterpret_cast<uintptr_t>(a.y) |
                       reinterpret_cast<uintptr_t>(a.workspace);
  return wide_ok(a.M, a.dim, a.dtype) && a.ln_w && a.inner % 32 == 0 && (al & 15) == 0;
}
size_t transition_fwd_wide_workspace(const mf_transition_fwd_args& a) { return align_up((size_t)a.M * a.inner * dtype_size(a.dtype), 256); }
// Y = G W2^T with the gated product G [M, inner] in the workspace, in 16 bit as on the CUDA-core path
int transition_fwd_wide(const mf_transition_fwd_args& a, cudaStream_t st) {
  int r = dispatch<1>(a.dim, WideArgs{a.M, 0, a.inner, a.dtype, a.eps, a.x, a.ln_w, a.ln_b, a.w1, nullptr, a.workspace, a.mean, a.rstd}, st);
  if (r) return r;
  return gemm_tc(GemmTcArgs{a.workspace, a.w2, a.y, a.M, a.dim, a.inner, a.dtype, 0, 0, 0}, st);
}

}  // namespace mf
