// LayernormLinear backward, input side, in one pass over dy (K in {64, 128}, 16-bit types, N <= 2048):
//
//     dyln = dy W^T   (TMEM only)      dx = LayerNorm'(dyln)
//     per CTA: column sums of dyln * xhat (gain gradient) and of dy (bias gradient)
//
// The shift gradient is the sum of dyln over the rows, which is (sum of dy) W^T: a [K, N] product afterwards
// (lnl_ops.cu), so no thread adds it up.
//
// Bound: HBM.  dy and x are read once, dx is written once: 2 (N + 2 K) bytes a row, 35 us at 147456 x 128 -> 512 at the
// measured copy rate.  Before, dyln went through memory in fp32 and dy was read a second time for the bias
// gradient: a GEMM, a row pass and a column-sum pass of 121 us together, now 60.  The copies alone take 45 us of those (with the
// arithmetic taken out): eight tiles per CTA leave a fill and a drain that a longer run would hide.
//
// Persistent CTA per SM, 128-row tiles, 640 threads:
//   warps 0-15  thread (row, quarter of the columns): the LayerNorm backward (ln_bwd_rows.cuh); the gain sums stay in the
//               thread's registers over all tiles.  With eight warps of 64 columns each the passes over a row were bound
//               by their own latency (65 us).  Results go through a swizzled staging slab of the warp to TMA stores.
//   warp 16     tcgen05.mma: dyln (+)= dy slab x W slab (4 products, N = K) into one of two accumulators; for the bias
//               gradient, per pair of slabs, eight N = 16 products dy^T x ones: the slabs as they are, read MN-major, give
//               the sums over the rows of 128 columns of dy, and stay in TMEM until the CTA is done.
//   warp 17     TMA: 64-column slabs of dy and of W (ring of four; W comes from L2: keeping it in shared memory where it
//               fits, up to N = 512, changed nothing).
// Every wait is bounded; on expiry the CTA raises a flag, drains and reports through mf_async_status().
#include "gemm_tc.cuh"
#include "ln_bwd_rows.cuh"

namespace mf {
namespace {
using namespace tcx;

constexpr int kRows = 128, kRowWarps = 16, kThreads = (kRowWarps + 4) * 32, kStages = 4;
// registers per thread: at launch / row warps / helper warps after setmaxnreg (the raise draws on what the drop releases)
constexpr int kLaunchRegs = 96, kRowRegs = 112, kHelperRegs = 32;
static_assert(kRowWarps * 32 * kRowRegs + 128 * kHelperRegs <= kThreads * kLaunchRegs, "setmaxnreg budget");
constexpr int kSlabB = kRows * 128;                  // [128 rows][64 columns] of dy
constexpr int kMaxN = 2048;                          // 16 TMEM columns per 128 columns of dy: 256 beside the accumulators
constexpr int kBarrier = 1;

struct LbP {
  int64_t M; int N, n_mt, n_slabs, has_db;
  uint32_t ab_fmt;
  const void *x, *gamma, *add1, *add2;
  const float *mean, *rstd;
  float *part, *db_part;
  int* status;
};

struct Bars { uint64_t full[kStages], empty[kStages], acc_full[2], acc_empty[2], db_full; };

__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {       // 16-byte multiples
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(reinterpret_cast<uint64_t>(p)), "r"(bytes) : "memory");
}

template <int K, typename T>
__global__ void __launch_bounds__(kThreads, 1)
lnl_bwd_tc_kernel(const __grid_constant__ CUtensorMap mdy, const __grid_constant__ CUtensorMap mw, const __grid_constant__ CUtensorMap mdx,
                  const LbP p) {
  constexpr int CW = K / 4;                          // columns per thread of the LayerNorm backward
  constexpr int kWSlabB = K * 128;                   // [K rows][64 columns] of W
  constexpr int kOutB = 32 * CW * 2;                 // a warp's staging slab: [32 rows][CW columns]
  constexpr int stage_b = kSlabB + kWSlabB;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sOut = smem;                              // [kRowWarps]
  uint8_t* sRing = sOut + kRowWarps * kOutB;
  float4 (*red)[CW / 8][128] = reinterpret_cast<float4 (*)[CW / 8][128]>(sRing + kStages * stage_b);      // [4 parts]
  __shared__ Bars bar;
  __shared__ __align__(16) float gam_s[K];
  __shared__ __align__(128) uint8_t ones_s[16 * 32];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    abort_s = 0;
    for (int i = 0; i < kStages; ++i) { mbar_init(&bar.full[i], 1); mbar_init(&bar.empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&bar.acc_full[i], 1); mbar_init(&bar.acc_empty[i], kRowWarps); }
    mbar_init(&bar.db_full, 1);
    mbar_fence_init();
    prefetch_tmap(&mdy); prefetch_tmap(&mw); prefetch_tmap(&mdx);
  }
  for (int k = tid; k < K; k += kThreads) gam_s[k] = to_f(static_cast<const T*>(p.gamma)[k]);
  for (int i = tid; i < 256; i += kThreads) reinterpret_cast<T*>(ones_s)[i] = from_f<T>(1.f);
  fence_async_smem();
  if (warp == 0) { tmem_alloc(&tmem_base_s, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  volatile int* abort_flag = &abort_s;
  const uint32_t tAcc = tmem_base_s, tDb = tmem_base_s + 2 * K;
  const int my_tiles = (p.n_mt - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  const int ns = p.n_slabs;

  if (warp < kRowWarps) {
    // ---------------------------------------------------------------------------------------- LayerNorm backward
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRowRegs));
    const int quarter = warp & 3, part = warp >> 2;      // TMEM lanes (rows) and columns of this warp
    const int row_l = quarter * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    uint8_t* slab = sOut + warp * kOutB;
    const float* gam = gam_s + part * CW;
    float2 gain[CW / 2];
#pragma unroll
    for (int i = 0; i < CW / 2; ++i) gain[i] = make_float2(0.f, 0.f);
    for (int t = 0; t < my_tiles; ++t) {
      const int ab = t & 1;
      const int row0 = ((int)blockIdx.x + t * (int)gridDim.x) * kRows;
      const int64_t row = (int64_t)row0 + row_l;
      const bool ok = row < p.M;
      // my part of the row of x, requested before the wait for the products
      uint4 raw[CW / 8];
      const uint4* xr = reinterpret_cast<const uint4*>(static_cast<const T*>(p.x) + row * K + part * CW);
#pragma unroll
      for (int c = 0; c < CW / 8; ++c) raw[c] = ok ? __ldg(xr + c) : make_uint4(0u, 0u, 0u, 0u);
      const float mu = ok ? p.mean[row] : 0.f, rs = ok ? p.rstd[row] : 0.f;
      wait_or_flag(&bar.acc_full[ab], (t >> 1) & 1, abort_flag);
      tc_fence_after();
      uint32_t dy[CW];
      if constexpr (CW == 32) tmem_ld32(tAcc + ab * K + part * CW + lane_addr, dy);
      else tmem_ld16(tAcc + ab * K + part * CW + lane_addr, dy);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.acc_empty[ab]);
      if (named_sync_or(kBarrier, kRowWarps * 32, *abort_flag)) break;
      const bool any = row0 + quarter * 32 < p.M;                    // a store must not start past the last row
      ln_bwd_row<T, CW, 4>(dy, raw, mu, rs, gam, red, part, row_l, kBarrier,
                               [&](uint32_t (&out)[CW / 2]) {
                                 auto add = [&](const void* from) {       // a gradient that reaches x beside the operator
                                   const uint4* ar = reinterpret_cast<const uint4*>(static_cast<const T*>(from) + row * K + part * CW);
#pragma unroll
                                   for (int c = 0; c < CW / 8; ++c) {
                                     const uint4 v = ok ? __ldg(ar + c) : make_uint4(0u, 0u, 0u, 0u);
                                     const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                                     for (int e = 0; e < 4; ++e) {
                                       const float2 y = add2(Pack2<T>::unpack(u[e]), Pack2<T>::unpack(out[c * 4 + e]));
                                       out[c * 4 + e] = Pack2<T>::pack(y.x, y.y);
                                     }
                                   }
                                 };
                                 if (p.add1) add(p.add1);
                                 if (p.add2) add(p.add2);
                                 if (lane == 0) bulk_wait_group_read<0>();  // the previous store has read the slab
                                 __syncwarp();
#pragma unroll
                                 for (int c = 0; c < CW / 8; ++c)
                                   *reinterpret_cast<uint4*>(slab + swz_offset(lane, c, CW * 2)) = make_uint4(out[c * 4], out[c * 4 + 1], out[c * 4 + 2], out[c * 4 + 3]);
                                 fence_async_smem();
                                 __syncwarp();
                                 if (lane == 0) {
                                   if (any) tma_store_2d(&mdx, slab, part * CW, row0 + quarter * 32);
                                   bulk_commit_group();
                                 }
                               },
                               [&](int k, float2 d, float2 h) { gain[k / 2] = fma2(d, h, gain[k / 2]); });
    }
    // the CTA's sums over its rows: a column sum per lane, then the four row quarters through shared memory
    float v[CW];
#pragma unroll
    for (int i = 0; i < CW / 2; ++i) { v[2 * i] = gain[i].x; v[2 * i + 1] = gain[i].y; }
    const float mine = column_sum(v, lane);
    float* scratch = reinterpret_cast<float*>(red);                  // [4][K]
    named_sync(kBarrier, kRowWarps * 32);
    if (lane < CW) scratch[quarter * K + part * CW + lane] = mine;
    named_sync(kBarrier, kRowWarps * 32);
    if (tid < K) p.part[(int64_t)blockIdx.x * K + tid] = (scratch[tid] + scratch[K + tid]) + (scratch[2 * K + tid] + scratch[3 * K + tid]);
    if (p.has_db && part == 0) {
      wait_or_flag(&bar.db_full, 0, abort_flag);
      tc_fence_after();
      for (int q = 0; q < ns / 2; ++q) {
        const uint32_t w = tmem_ld1(tDb + q * 16 + lane_addr);
        tmem_ld_wait();
        const int n = q * 128 + row_l;
        if (n < p.N && !*abort_flag) p.db_part[(int64_t)blockIdx.x * p.N + n] = __uint_as_float(w);
      }
      tc_fence_before();
    }
    if (lane == 0) bulk_wait_group<0>();
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kHelperRegs));
    if (warp == kRowWarps + 1 && lane == 0) {
    // ---------------------------------------------------------------------------------------- TMA producer
    uint32_t cnt = 0;
    for (int t = 0; t < my_tiles && !*abort_flag; ++t) {
      const int row0 = ((int)blockIdx.x + t * (int)gridDim.x) * kRows;
      for (int s = 0; s < ns; ++s, ++cnt) {
        const int st = cnt % kStages;
        if (cnt >= kStages) wait_or_flag(&bar.empty[st], ((cnt / kStages) - 1) & 1, abort_flag);
        if (*abort_flag) break;
        // the next tile of x, which the row warps read with plain loads once its products are done
        if (s == 0 && row0 + (int)gridDim.x * kRows + kRows <= p.M) {
          const int64_t next = (int64_t)(row0 + (int)gridDim.x * kRows) * K;
          prefetch_l2(static_cast<const T*>(p.x) + next, kRows * K * 2);
          if (p.add1) prefetch_l2(static_cast<const T*>(p.add1) + next, kRows * K * 2);
          if (p.add2) prefetch_l2(static_cast<const T*>(p.add2) + next, kRows * K * 2);
        }
        uint8_t* a = sRing + st * stage_b;
        mbar_expect_tx(&bar.full[st], stage_b);
        tma_load_2d(a, &mdy, &bar.full[st], s * 64, row0);           // columns beyond N and rows beyond M arrive as zeros
        tma_load_2d(a + kSlabB, &mw, &bar.full[st], s * 64, 0);
      }
    }
    drain_ring(bar.full, cnt, kStages);
    } else if (warp == kRowWarps) {
    // ---------------------------------------------------------------------------------------- MMA issuer
    // Run by the whole warp, one elected lane issuing: with a single lane's branch and run-time descriptors an MMA took 100
    // to 240 cycles to issue, more than it takes to execute (see mma_ss_el).
    auto dead = [&] { return __any_sync(0xffffffffu, *abort_flag) != 0; };
    const uint32_t id = idesc_f16(128, K, p.ab_fmt, 0, 0), id_db = idesc_f16(128, 16, p.ab_fmt, 1, 0);
    const uint32_t ones_lo = desc_lo(smem_u32(ones_s), 16);
    uint32_t cnt = 0;
    for (int t = 0; t < my_tiles && !dead(); ++t) {
      const int ab = t & 1;
      if (t >= 2) wait_or_flag(&bar.acc_empty[ab], ((t >> 1) - 1) & 1, abort_flag);
      for (int s = 0; s < ns; ++s, ++cnt) {
        const int st = cnt % kStages;
        wait_or_flag(&bar.full[st], (cnt / kStages) & 1, abort_flag);
        tc_fence_after();
        if (dead()) break;
        const uint32_t a = smem_u32(sRing + st * stage_b);
        const uint32_t a_lo = desc_lo(a, 16), w_lo = desc_lo(a + kSlabB, 16);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          mma_ss_el(tAcc + ab * K, a_lo + ks * 2, desc_hi(1024, kSw128), w_lo + ks * 2, desc_hi(1024, kSw128), id, s > 0 || ks > 0);
        if (p.has_db && (s & 1)) {        // slabs come in pairs and rings are even: this slab and the one before are neighbours
          const uint32_t d_lo = desc_lo(a - stage_b, stage_b);
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)
            mma_ss_el(tDb + (s >> 1) * 16, d_lo + ks * (2048 / 16), desc_hi(1024, kSw128), ones_lo, desc_hi(256, kSw32), id_db, t > 0 || ks > 0);
        }
        if (s & 1) { tc_commit_el(&bar.empty[st - 1]); tc_commit_el(&bar.empty[st]); }
      }
      tc_commit_el(&bar.acc_full[ab]);
    }
    tc_commit_el(&bar.db_full);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (tid == 0 && abort_s) *reinterpret_cast<volatile int*>(p.status) = 1;
  if (warp == 0) tmem_dealloc(tmem_base_s, 512);
}

template <int K, typename T>
int launch(const LnlBwdRowsArgs& a, int grid, cudaStream_t st) {
  CUtensorMap mdy, mw, mdx;
  int r;
  {
    const int64_t dims[2] = {a.N, a.M}, str[2] = {1, a.N};
    const int box[2] = {64, kRows};
    if ((r = make_tiled_map(&mdy, a.dy, a.dtype, 2, dims, str, box, 128))) return r;
  }
  {
    const int64_t dims[2] = {a.N, K}, str[2] = {1, a.N};
    const int box[2] = {64, K};
    if ((r = make_tiled_map(&mw, a.w, a.dtype, 2, dims, str, box, 128))) return r;
  }
  {
    const int64_t dims[2] = {K, a.M}, str[2] = {1, K};
    const int box[2] = {K / 4, 32};
    if ((r = make_tiled_map(&mdx, a.dx, a.dtype, 2, dims, str, box, K / 2))) return r;
  }
  LbP p{};
  p.M = a.M; p.N = a.N;
  p.n_mt = (int)((a.M + kRows - 1) / kRows);
  p.n_slabs = (a.N + 127) / 128 * 2;
  p.has_db = a.db_part != nullptr;
  p.ab_fmt = a.dtype == MF_BF16 ? 1u : 0u;
  p.x = a.x; p.gamma = a.gamma; p.add1 = a.add1; p.add2 = a.add2; p.mean = a.mean; p.rstd = a.rstd;
  p.part = a.part; p.db_part = a.db_part;
  p.status = status_word();
  MF_REQUIRE(p.status, MF_ERR_CUDA, "could not allocate the device status word");
  MF_REQUIRE(tc_async_status() == 0, MF_ERR_CUDA, "an earlier tensor-core kernel gave up on a bounded wait; results are invalid");
  constexpr size_t smem = 1024 + kRowWarps * 32 * (size_t)K / 2 + kStages * (size_t)(kSlabB + K * 128) + 128 * (size_t)K * 2;
  constexpr auto kern = lnl_bwd_tc_kernel<K, T>;
  if (int e = opt_in_smem<kern>(smem, kLaunchRegs)) return e;
  kern<<<grid, kThreads, smem, st>>>(mdy, mw, mdx, p);
  MF_LAUNCHED("lnl_bwd_tc_kernel");
  return MF_OK;
}

}  // namespace

bool lnl_bwd_rows_tc_ok(int64_t M, int K, int N) { return (K == 64 || K == 128) && N <= kMaxN && M <= (int64_t)INT32_MAX - kRows; }

int lnl_bwd_rows_tc_blocks(int64_t M) {
  const int64_t tiles = (M + kRows - 1) / kRows;
  return (int)(tiles < sm_count() ? tiles : sm_count());
}

int lnl_bwd_rows_tc(const LnlBwdRowsArgs& a, cudaStream_t st) {
  const int grid = lnl_bwd_rows_tc_blocks(a.M);
  if (a.dtype == MF_BF16) return a.K == 128 ? launch<128, __nv_bfloat16>(a, grid, st) : launch<64, __nv_bfloat16>(a, grid, st);
  return a.K == 128 ? launch<128, __half>(a, grid, st) : launch<64, __half>(a, grid, st);
}

}  // namespace mf
