// Fused Transition forward on the tensor cores:
//     Y[M, dim] = ( silu(H[:, inner:]) * H[:, :inner] ) W2^T,   H = LayerNorm(X) W1,   dim in {64, 128}.
// The hidden activation H [M, 2*inner] and the gated product never leave the SM.
//
// Bound: shared-memory bandwidth.  With all operands in shared memory a chunk of 64 hidden columns moved 180 KB (two products'
// A and B, the weights coming in, G going out), 1400 cycles at 128 bytes per clock against 770 of the tensor pipe.  So the
// A operands live in TMEM: LN(X) of the tile (GEMM1) and the gated product G (GEMM2), and
// only weights cross shared memory: 104 KB.
//
// Persistent CTA per SM, 128-row tiles of X.  Per tile the hidden dimension is walked in chunks of 64:
//   warps 16-19  (a warpgroup) LayerNorm: TMA brings the raw rows, a thread owns one: mean and variance in two passes from
//                registers, the 16-bit result waits in them until GEMM1 of the tile before is done with the TMEM buffer.
//   warps 20, 22 MMA issuers, one GEMM each (one elected lane issues): GEMM1 of chunk c: H = A W1 blocks (dim/16 MMAs, N = 128:
//                the value and the gate block are the two atoms of one MN-major B operand) into one of two TMEM buffers;
//                GEMM2: Y += G W2-block^T (4 MMAs, N = dim) once the workers have written G.
//   warps 0-15   workers, two teams that take alternate chunks, each with its own H buffer: thread (row, half) takes 32
//                columns of value and gate, g = silu(gate) * value with one MUFU op per element
//                (silu(x) = x/2 * (1 + tanh(x/2))), packed 16-bit G back to TMEM.  A chunk's chain - wait, load, gating,
//                store, hand-over - is mostly latency, so one team of eight warps left the pipes idle.  The Y tile is written
//                out (TMEM -> registers -> the warp's swizzled slab -> TMA store) one chunk into the next tile.
//   warps 21, 23 TMA: X and W1; W2 (whose stages are free later: GEMM1's loads must not queue behind that).
// [262144, 128] -> 512 -> 128: 135 us with one team and all operands in shared memory, 109 with two teams, 95 now.
// Every wait is bounded; on expiry the CTA raises a flag, drains and reports through mf_async_status().
#include <type_traits>

#include "evo_tc_common.cuh"

namespace mf {
namespace {
using namespace tcx;

constexpr int kRows = 128;
constexpr int kHC = 64;             // hidden columns per chunk
constexpr int kWorkWarps = 16;         // two teams of eight
constexpr int kThreads = (kWorkWarps + 8) * 32;      // then four normalising warps and four issuers (20, 22 MMA, 21, 23 TMA)
// registers per thread: at launch / workers / normalising warps / issuers after setmaxnreg (the raises draw on the drop)
constexpr int kLaunchRegs = 80, kWorkRegs = 80, kNormRegs = 128, kIssueRegs = 32;
static_assert(kWorkWarps * 32 * kWorkRegs + 128 * kNormRegs + 128 * kIssueRegs <= kThreads * kLaunchRegs, "setmaxnreg budget");
constexpr int kWStages = 3;

struct TrP {
  int64_t M; int dim, inner, n_mt, n_ch;
  float eps;
  uint32_t ab_fmt;
  int has_ln;
  const void *gamma, *beta;
  float *mean, *rstd;
  int* status;
};

struct Bars {
  uint64_t x_full, x_empty, a_full, a_empty;
  uint64_t w1_full[kWStages], w1_empty[kWStages], w2_full[kWStages], w2_empty[kWStages];
  uint64_t h_full[2], h_empty[2], g_full[2], g_empty[2], y_full, y_empty;
};

__device__ __forceinline__ float tanh_approx(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <int K, typename T>
__global__ void __launch_bounds__(kThreads, 1)
transition_fwd_tc_kernel(const __grid_constant__ CUtensorMap mx, const __grid_constant__ CUtensorMap mw1,
                         const __grid_constant__ CUtensorMap mw2, const __grid_constant__ CUtensorMap my, const TrP p) {
  constexpr int ATOMS = K / 64;
  constexpr int A_BYTES = kRows * K * 2;
  constexpr int W1B = K * 128;                 // one [K rows][64 columns] block of W1
  constexpr int W2B = K * 128;                 // one [dim = K rows][64 hidden] block of W2
  constexpr int W_BYTES = 2 * W1B + W2B;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sX = smem;                          // raw rows
  uint8_t* sW = sX + A_BYTES;                  // [kWStages][W1 value | W1 gate | W2]
  uint8_t* sY = sW + kWStages * W_BYTES;       // the workers' slabs

  __shared__ Bars bar;
  __shared__ __align__(16) float gam_s[K], bet_s[K];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  if (tid == 0) {
    abort_s = 0;
    mbar_init(&bar.x_full, 1); mbar_init(&bar.x_empty, 4);
    for (int i = 0; i < kWStages; ++i) {
      mbar_init(&bar.w1_full[i], 1); mbar_init(&bar.w1_empty[i], 1);
      mbar_init(&bar.w2_full[i], 1); mbar_init(&bar.w2_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bar.h_full[i], 1); mbar_init(&bar.h_empty[i], 8);
      mbar_init(&bar.g_full[i], 8); mbar_init(&bar.g_empty[i], 1);
    }
    mbar_init(&bar.a_full, 4); mbar_init(&bar.a_empty, 1);
    mbar_init(&bar.y_full, 1); mbar_init(&bar.y_empty, kWorkWarps);
    mbar_fence_init();
    prefetch_tmap(&mx); prefetch_tmap(&mw1); prefetch_tmap(&mw2); prefetch_tmap(&my);
  }
  for (int k = tid; k < K; k += kThreads) {
    gam_s[k] = p.has_ln ? to_f(static_cast<const T*>(p.gamma)[k]) : 1.f;
    bet_s[k] = (p.has_ln && p.beta) ? to_f(static_cast<const T*>(p.beta)[k]) : 0.f;
  }
  if (warp == 0) { tmem_alloc(&tmem_base_s, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  volatile int* abort_flag = &abort_s;
  const uint32_t tm0 = uniform(tmem_base_s);
  // H: two buffers of (value 64 | gate 64); G: two of 32 (64 packed); Y: K columns; A: K / 2
  const uint32_t tH = tm0, tG = tm0 + 256, tY = tm0 + 320, tA = tm0 + 448;
  const int my_tiles = p.n_mt > (int)blockIdx.x ? (p.n_mt - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
  const int nch = p.n_ch;
  const int row_l = (warp & 3) * 32 + lane;
  const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;

  if (warp < kWorkWarps) {
    // ------------------------------------------------------------------------------------ workers
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kWorkRegs));
    const int team = warp >> 3, half = (warp >> 2) & 1;
    const int part = warp >> 2;                     // my quarter of the columns of Y
    uint8_t* slab = sY + warp * (32 * K / 2);       // [32 rows][K / 4 columns]
    const uint32_t tMine = tH + team * 128 + half * 32 + lane_addr;      // my value columns; the gate's are 64 further
    const uint32_t tOut = tG + team * 32 + half * 16 + lane_addr;
    // my quarter of the columns of tile t of Y: TMEM -> registers -> slab -> TMA store.  Done one chunk into the next tile,
    // so that nobody waits for the last products of a tile.
    auto write_out = [&](int t) {
      wait_or_flag(&bar.y_full, t & 1, abort_flag);
      tc_fence_after();
      uint32_t acc[K / 4];
      if constexpr (K == 128) tmem_ld32(tY + part * 32 + lane_addr, acc);
      else tmem_ld16(tY + part * 16 + lane_addr, acc);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) { mbar_arrive(&bar.y_empty); bulk_wait_group_read<0>(); }     // the previous tile's store has read the slab
      __syncwarp();
      if (__any_sync(0xffffffffu, *abort_flag)) return;
#pragma unroll
      for (int ch = 0; ch < K / 32; ++ch) {
        uint4 v;
        v.x = Pack2<T>::pack(__uint_as_float(acc[ch * 8]), __uint_as_float(acc[ch * 8 + 1]));
        v.y = Pack2<T>::pack(__uint_as_float(acc[ch * 8 + 2]), __uint_as_float(acc[ch * 8 + 3]));
        v.z = Pack2<T>::pack(__uint_as_float(acc[ch * 8 + 4]), __uint_as_float(acc[ch * 8 + 5]));
        v.w = Pack2<T>::pack(__uint_as_float(acc[ch * 8 + 6]), __uint_as_float(acc[ch * 8 + 7]));
        *reinterpret_cast<uint4*>(slab + swz_offset(lane, ch, K / 2)) = v;
      }
      fence_async_smem();
      __syncwarp();
      if (lane == 0) {
        const int r0 = (int)(((int64_t)blockIdx.x + (int64_t)t * gridDim.x) * kRows) + (warp & 3) * 32;
        if (r0 < p.M) tma_store_2d(&my, slab, part * (K / 4), r0);       // a store must not start past the last row
        bulk_commit_group();
      }
    };
    uint32_t ch_cnt = 0;                            // chunks seen (buffer = team = ch_cnt & 1)
    int pending = -1;                               // tile whose Y has not been written out
    for (int t = 0; t < my_tiles && !__any_sync(0xffffffffu, *abort_flag); ++t) {
      for (int c = 0; c < nch; ++c, ++ch_cnt) {
        if ((int)(ch_cnt & 1) != team) continue;
        wait_or_flag(&bar.h_full[team], (ch_cnt >> 1) & 1, abort_flag);
        tc_fence_after();
        uint32_t gp[16];
#pragma unroll
        for (int q = 0; q < 2; ++q) {               // 16 columns at a time keeps the live registers down
          uint32_t ha[16], hg[16];
          tmem_ld16(tMine + q * 16, ha);
          tmem_ld16(tMine + 64 + q * 16, hg);
          tmem_ld_wait();
          if (q == 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar.h_empty[team]);
          }
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float a0 = __uint_as_float(ha[2 * e]), a1 = __uint_as_float(ha[2 * e + 1]);
            const float b0 = 0.5f * __uint_as_float(hg[2 * e]), b1 = 0.5f * __uint_as_float(hg[2 * e + 1]);
            // silu(b) * a = b/2 * (1 + tanh(b/2)) * a
            const float g0 = fmaf(b0, tanh_approx(b0), b0) * a0, g1 = fmaf(b1, tanh_approx(b1), b1) * a1;
            gp[q * 8 + e] = Pack2<T>::pack(g0, g1);
          }
        }
        if (ch_cnt >= 2) wait_or_flag(&bar.g_empty[team], ((ch_cnt >> 1) - 1) & 1, abort_flag);
        tc_fence_after();
        tmem_st16(tOut, gp);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar.g_full[team]);
        if (pending >= 0) { write_out(pending); pending = -1; }
      }
      if (pending >= 0) write_out(pending);         // a tile without a chunk of mine
      pending = t;
    }
    if (pending >= 0) write_out(pending);
    if (lane == 0) bulk_wait_group<0>();
  } else if (warp < kWorkWarps + 4) {
    // ------------------------------------------------------------------------------------ normalising warps, ahead of the MMAs
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kNormRegs));
    for (int t = 0; t < my_tiles && !*abort_flag; ++t) {
      const int64_t row = ((int64_t)blockIdx.x + (int64_t)t * gridDim.x) * kRows + row_l;
      const bool ok = row < p.M;
      wait_or_flag(&bar.x_full, t & 1, abort_flag);
      uint4 raw[K / 8];
#pragma unroll
      for (int c = 0; c < K / 8; ++c)
        raw[c] = *reinterpret_cast<const uint4*>(sX + (c >> 3) * (kRows * 128) + swz_offset(row_l, c & 7, 128));
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.x_empty);
      float2 mm = make_float2(0.f, 0.f), rr = mm;
      if (p.has_ln) {
        float s4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < K / 8; ++c) {
          const float2 f0 = Pack2<T>::unpack(raw[c].x), f1 = Pack2<T>::unpack(raw[c].y), f2 = Pack2<T>::unpack(raw[c].z), f3 = Pack2<T>::unpack(raw[c].w);
          s4[0] += f0.x + f0.y; s4[1] += f1.x + f1.y; s4[2] += f2.x + f2.y; s4[3] += f3.x + f3.y;
        }
        const float mu = ((s4[0] + s4[1]) + (s4[2] + s4[3])) * (1.f / K);
        mm = make_float2(mu, mu);
        float q4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < K / 8; ++c) {
          const uint32_t u[4] = {raw[c].x, raw[c].y, raw[c].z, raw[c].w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 d = sub2(Pack2<T>::unpack(u[e]), mm);
            q4[e] = fmaf(d.x, d.x, q4[e]); q4[e] = fmaf(d.y, d.y, q4[e]);
          }
        }
        const float rs = rsqrtf(((q4[0] + q4[1]) + (q4[2] + q4[3])) * (1.f / K) + p.eps);
        if (ok) { p.mean[row] = mu; p.rstd[row] = rs; }
        rr = make_float2(rs, rs);
      }
      if (p.has_ln) {
#pragma unroll
        for (int c = 0; c < K / 8; ++c) {
          asm volatile("" ::: "memory");               // gains and shifts are not fetched further ahead than this: registers
          uint32_t u[4] = {raw[c].x, raw[c].y, raw[c].z, raw[c].w};
#pragma unroll
          for (int e = 0; e < 4; e += 2) {
            const int k = c * 8 + e * 2;
            const float4 g = *reinterpret_cast<const float4*>(gam_s + k), h = *reinterpret_cast<const float4*>(bet_s + k);
            const float2 y0 = fma2(mul2(sub2(Pack2<T>::unpack(u[e]), mm), rr), make_float2(g.x, g.y), make_float2(h.x, h.y));
            const float2 y1 = fma2(mul2(sub2(Pack2<T>::unpack(u[e + 1]), mm), rr), make_float2(g.z, g.w), make_float2(h.z, h.w));
            u[e] = ok ? Pack2<T>::pack(y0.x, y0.y) : 0u; u[e + 1] = ok ? Pack2<T>::pack(y1.x, y1.y) : 0u;
          }
          raw[c] = make_uint4(u[0], u[1], u[2], u[3]);
        }
      }
      if (t > 0) wait_or_flag(&bar.a_empty, (t - 1) & 1, abort_flag);      // GEMM1 of the previous tile has read its rows
      tc_fence_after();
#pragma unroll
      for (int q = 0; q < K / 32; ++q) {
        const uint32_t o[16] = {raw[q * 4].x,     raw[q * 4].y,     raw[q * 4].z,     raw[q * 4].w,     raw[q * 4 + 1].x, raw[q * 4 + 1].y, raw[q * 4 + 1].z, raw[q * 4 + 1].w,
                                raw[q * 4 + 2].x, raw[q * 4 + 2].y, raw[q * 4 + 2].z, raw[q * 4 + 2].w, raw[q * 4 + 3].x, raw[q * 4 + 3].y, raw[q * 4 + 3].z, raw[q * 4 + 3].w};
        tmem_st16(tA + q * 16 + lane_addr, o);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.a_full);
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kIssueRegs));
    auto dead = [&] { return __any_sync(0xffffffffu, *abort_flag) != 0; };      // the MMA roles are run by whole warps
    if (warp == kWorkWarps + 4) {
      // ---------------------------------------------------------------------------------- MMA issuer: GEMM1
      const uint32_t id1 = idesc_f16(128, 2 * kHC, p.ab_fmt, 0, 1);     // B (W1 value | gate blocks) MN-major
      uint32_t ch_cnt = 0;
      for (int t = 0; t < my_tiles && !dead(); ++t) {
        wait_or_flag(&bar.a_full, t & 1, abort_flag);
        for (int c = 0; c < nch && !dead(); ++c, ++ch_cnt) {
          const int hb = ch_cnt & 1, ws = ch_cnt % kWStages;
          wait_or_flag(&bar.w1_full[ws], (ch_cnt / kWStages) & 1, abort_flag);
          if (ch_cnt >= 2) wait_or_flag(&bar.h_empty[hb], ((ch_cnt >> 1) - 1) & 1, abort_flag);
          tc_fence_after();
          if (dead()) break;
          const uint32_t w1_lo = desc_lo(smem_u32(sW + ws * W_BYTES), W1B);
#pragma unroll
          for (int ks = 0; ks < K / 16; ++ks)
            mma_ts_el(tH + hb * 128, tA + ks * 8, w1_lo + ks * (2048 / 16), desc_hi(1024, kSw128), id1, ks > 0);
          tc_commit_el(&bar.h_full[hb]);
          tc_commit_el(&bar.w1_empty[ws]);
        }
        if (dead()) break;
        tc_commit_el(&bar.a_empty);
      }
    } else if (warp == kWorkWarps + 6) {
      // ---------------------------------------------------------------------------------- second MMA issuer: GEMM2.
      // One warp issuing both GEMMs would wait for the workers' G of one chunk before it could start the next chunk's H.
      const uint32_t id2 = idesc_f16(128, K, p.ab_fmt, 0, 0);       // B (W2 block) K-major, N = dim
      uint32_t ch_cnt = 0;
      for (int t = 0; t < my_tiles && !dead(); ++t) {
        for (int c = 0; c < nch && !dead(); ++c, ++ch_cnt) {            // Y (+)= G(c) W2-block(c)^T
          const int gb = ch_cnt & 1, ws = ch_cnt % kWStages;
          wait_or_flag(&bar.w2_full[ws], (ch_cnt / kWStages) & 1, abort_flag);
          wait_or_flag(&bar.g_full[gb], (ch_cnt >> 1) & 1, abort_flag);
          if (c == 0 && t > 0) wait_or_flag(&bar.y_empty, (t - 1) & 1, abort_flag);
          tc_fence_after();
          if (dead()) break;
          const uint32_t g = tG + gb * 32, w2_lo = desc_lo(smem_u32(sW + ws * W_BYTES + 2 * W1B), 16);
#pragma unroll
          for (int ks = 0; ks < kHC / 16; ++ks)
            mma_ts_el(tY, g + ks * 8, w2_lo + ks * 2, desc_hi(1024, kSw128), id2, c > 0 || ks > 0);
          tc_commit_el(&bar.g_empty[gb]);
          tc_commit_el(&bar.w2_empty[ws]);
        }
        if (dead()) break;
        tc_commit_el(&bar.y_full);
      }
    } else if (warp == kWorkWarps + 5 && lane == 0) {
      // ---------------------------------------------------------------------------------- TMA producer of X and W1
      uint32_t ch_cnt = 0, n_x = 0;
      auto load_x = [&](int t) {           // (the normalising warps hold the rows of tile t - 1 in registers)
        if (t > 0) wait_or_flag(&bar.x_empty, (t - 1) & 1, abort_flag);
        if (*abort_flag) return;
        ++n_x;
        const int row0 = (int)(((int64_t)blockIdx.x + (int64_t)t * gridDim.x) * kRows);
        mbar_expect_tx(&bar.x_full, A_BYTES);
#pragma unroll
        for (int at = 0; at < ATOMS; ++at) tma_load_2d(sX + at * (kRows * 128), &mx, &bar.x_full, at * 64, row0);
      };
      if (my_tiles > 0) load_x(0);
      for (int t = 0; t < my_tiles && !*abort_flag; ++t) {
        for (int c = 0; c < nch; ++c, ++ch_cnt) {
          if (c == (nch > 1 ? 1 : 0) && t + 1 < my_tiles) load_x(t + 1);
          const int ws = ch_cnt % kWStages;
          uint8_t* w = sW + ws * W_BYTES;
          if (ch_cnt >= kWStages) wait_or_flag(&bar.w1_empty[ws], ((ch_cnt / kWStages) - 1) & 1, abort_flag);
          if (*abort_flag) break;
          mbar_expect_tx(&bar.w1_full[ws], 2 * W1B);
          tma_load_2d(w, &mw1, &bar.w1_full[ws], c * kHC, 0);                    // value columns of W1
          tma_load_2d(w + W1B, &mw1, &bar.w1_full[ws], p.inner + c * kHC, 0);   // gate columns of W1
        }
      }
      drain_ring(&bar.x_full, n_x, 1);
      drain_ring(bar.w1_full, ch_cnt, kWStages);
    } else if (warp == kWorkWarps + 7 && lane == 0) {
      // ---------------------------------------------------------------------------------- TMA producer of the W2 blocks
      uint32_t ch_cnt = 0;
      for (int t = 0; t < my_tiles && !*abort_flag; ++t)
        for (int c = 0; c < nch; ++c, ++ch_cnt) {
          const int ws = ch_cnt % kWStages;
          if (ch_cnt >= kWStages) wait_or_flag(&bar.w2_empty[ws], ((ch_cnt / kWStages) - 1) & 1, abort_flag);
          if (*abort_flag) break;
          mbar_expect_tx(&bar.w2_full[ws], W2B);
          tma_load_2d(sW + ws * W_BYTES + 2 * W1B, &mw2, &bar.w2_full[ws], c * kHC, 0);      // W2[:, chunk]
        }
      drain_ring(bar.w2_full, ch_cnt, kWStages);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (tid == 0 && abort_s) *reinterpret_cast<volatile int*>(p.status) = 1;
  if (warp == 0) tmem_dealloc(tmem_base_s, 512);
}

template <int K, typename T>
int launch_tr(const mf_transition_fwd_args& a, cudaStream_t st) {
  CUtensorMap mx, mw1, mw2, my;
  int r;
  {
    const int64_t dims[2] = {K, a.M}, str[2] = {1, K};
    const int box[2] = {64, kRows};
    if ((r = make_tiled_map(&mx, a.x, a.dtype, 2, dims, str, box, 128))) return r;
    const int slab[2] = {K / 4, 32};             // one worker warp's part of Y
    if ((r = make_tiled_map(&my, a.y, a.dtype, 2, dims, str, slab, K / 2))) return r;
  }
  {
    const int64_t dims[2] = {2 * (int64_t)a.inner, K}, str[2] = {1, 2 * (int64_t)a.inner};
    const int box[2] = {64, K};
    if ((r = make_tiled_map(&mw1, a.w1, a.dtype, 2, dims, str, box, 128))) return r;
  }
  {
    const int64_t dims[2] = {a.inner, K}, str[2] = {1, a.inner};
    const int box[2] = {64, K};
    if ((r = make_tiled_map(&mw2, a.w2, a.dtype, 2, dims, str, box, 128))) return r;
  }
  TrP p{};
  p.M = a.M; p.dim = K; p.inner = a.inner;
  p.n_mt = (int)((a.M + kRows - 1) / kRows);
  p.n_ch = a.inner / kHC;
  p.eps = a.eps;
  p.ab_fmt = a.dtype == MF_BF16 ? 1u : 0u;
  p.has_ln = a.ln_w != nullptr;
  p.gamma = a.ln_w; p.beta = a.ln_b;
  p.mean = a.mean; p.rstd = a.rstd;
  p.status = status_word();
  MF_REQUIRE(p.status, MF_ERR_CUDA, "could not allocate the device status word");
  MF_REQUIRE(tc_async_status() == 0, MF_ERR_CUDA, "an earlier tensor-core kernel gave up on a bounded wait; results are invalid");
  const size_t smem = 1024 + 2 * (size_t)kRows * K * 2 + kWStages * (size_t)(3 * K * 128);
  constexpr auto kern = transition_fwd_tc_kernel<K, T>;
  if (int e = opt_in_smem<kern>(smem, kLaunchRegs)) return e;
  int grid = sm_count();
  if (grid > p.n_mt) grid = p.n_mt;
  kern<<<grid, kThreads, smem, st>>>(mx, mw1, mw2, my, p);
  MF_LAUNCHED("transition_fwd_tc_kernel");
  return MF_OK;
}

}  // namespace

bool transition_fwd_tc_supported(const mf_transition_fwd_args& a) {
  if (a.dtype != MF_BF16 && a.dtype != MF_F16) return false;
  if (a.dim != 64 && a.dim != 128) return false;
  if (a.inner % 64 != 0 || a.inner < 64 || a.M < 1 || a.M > (int64_t)INT32_MAX) return false;
  const uintptr_t al = reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.w1) | reinterpret_cast<uintptr_t>(a.w2) |
                       reinterpret_cast<uintptr_t>(a.y);
  return (al & 15) == 0;
}

int transition_fwd_tc(const mf_transition_fwd_args& a, cudaStream_t st) {
  if (a.dtype == MF_BF16) return a.dim == 128 ? launch_tr<128, __nv_bfloat16>(a, st) : launch_tr<64, __nv_bfloat16>(a, st);
  return a.dim == 128 ? launch_tr<128, __half>(a, st) : launch_tr<64, __half>(a, st);
}

}  // namespace mf
