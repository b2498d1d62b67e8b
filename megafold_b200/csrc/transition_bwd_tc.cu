// Fused core of the Transition backward on the tensor cores (dim = 128, 16-bit types):
//
//     h = LayerNorm(x) W1          (recomputed, never stored)            g  = silu(h_gate) * h_value   -> HBM (for dW2)
//     dg = dy W2                                                          dh = SwiGLU'(h, dg)           -> HBM (for dW1)
//     dyln = dh W1^T               (accumulated in TMEM over the hidden dimension)      dx = LayerNorm'(dyln)   -> HBM
//     per CTA: column sums of dyln * xhat and dyln (gain and shift gradients)
//
// so that the [M, 2*inner] pre-activation, the [M, inner] gradient of the gated product and dyln never touch HBM, and
// g / dh are written exactly once.  The weight gradients (dW2 = dy^T g, dW1 = LN(x)^T dh) are separate, streaming kernels.
//
// Bound: writing dh and g (3 KB a row at inner = 512: 123 us for 262144 rows), then shared-memory bandwidth.  With all A operands
// in shared memory a chunk of 32 hidden columns moved 220 KB, 1700 cycles; LN(X), dY and dh are TMEM operands now, which
// leaves 112 KB: weights in, B operands, dh and g on their way to the TMA stores.
//
// Persistent CTA per SM, 128-row tiles, the hidden dimension walked in chunks of 32 (value) + 32 (gate) columns:
//   warps 0-15   workers, two teams that take alternate chunks, thread (row, half): 16 value, 16 gate, 16 dg columns from
//                TMEM; g, dh in registers with one MUFU op per element; dh packed to TMEM (A operand of the dyln product,
//                column order inside a chunk: [value 0-15 | gate 0-15 | value 16-31 | gate 16-31]), dh and g to shared-memory
//                tiles that are TMA-stored.
//   warps 16-23  rows, two threads a row: LayerNorm of the next X tile (saved statistics) to TMEM, dY beside it; then this
//                tile's dyln row into registers, which frees the accumulator at once, and the LayerNorm backward of it while
//                the workers are in the next tile.  dx replaces the raw row of x in shared memory and is TMA-stored.
//   warp 24      MMAs of H(c) = A W1blocks (8 x N=64, the two blocks as the two swizzle atoms of one MN-major B operand)
//                and DG(c) = dY W2block (8 x N=32) into one of two TMEM buffers.
//   warp 25      TMA loads: per chunk the W1 value / gate blocks and the W2 block ([128 rows][32 columns], 64-byte swizzle).
//   warp 26      MMAs of dyln += dh(c) [W1 value block; W1 gate block]^T (4 x N=128; the same shared-memory blocks read
//                K-major) once the workers have written dh(c).
//   warp 27      TMA stores of the dh and g tiles of every chunk.
// (The workers doing the LayerNorm backward between two tiles, four threads a row, held up the dyln products, and with them
// the weight stages, for 14000 cycles a tile: 341 us.  One thread a row took 14000 to 20000 cycles for it, beside some 13000
// for the LayerNorm of the next tile and its waits: as long as a tile, 286 us.)
// dh is stored in that column order, a panel [M][64] per chunk; dW1 computed from it has its columns in the same order and is
// put back by a small kernel.  (Panels, of g too: a chunk of a tile is one run of 16 KB.  128-byte pieces at the pitch of a
// whole row took 25 us more.)
// [262144, 128], inner 512: 245 us; with one team, operands in shared memory and dyln in HBM 322 us, and 68 for the row pass.
// Every wait is bounded; on expiry the CTA raises a flag, drains and reports through mf_async_status().
#include "ln_bwd_rows.cuh"

namespace mf {
namespace {
using namespace tcx;

constexpr int kRows = 128;
constexpr int K = 128;               // dim
constexpr int kHC = 32;              // hidden (value) columns per chunk
constexpr int kWorkWarps = 16;       // two teams of eight
constexpr int kRowWarps = 8, kFirstIssuer = kWorkWarps + kRowWarps;         // row warps: two per 32 rows: the 32-column quarters 0 and 2, 1 and 3
constexpr int kThreads = (kWorkWarps + kRowWarps + 4) * 32;
// registers per thread: at launch / workers / row warps / issuers after setmaxnreg (the raises draw on the drop).  With 64 / 96 / 56 the
// row warps spilled: [100000, 128], inner 512, forward + backward 236 us, 231 with 64 / 104 / 40, 227 with these.
constexpr int kLaunchRegs = 72, kWorkRegs = 56, kRowRegs = 120, kIssueRegs = 40;
static_assert(kWorkWarps * 32 * kWorkRegs + kRowWarps * 32 * kRowRegs + 128 * kIssueRegs <= kThreads * kLaunchRegs, "setmaxnreg budget");
constexpr int A_BYTES = kRows * K * 2;          // 32 KB: X or dY tile, two 64-column atoms
constexpr int WB = K * 64;                       // 8 KB: one [128 rows][32 columns] weight block
constexpr int DH_BYTES = kRows * 128;            // [128 rows][64 columns] 16 bit
constexpr int G_BYTES = kRows * 64;              // [128 rows][32 columns] 16 bit
// Weight stages.  The W1 blocks of a chunk (value | gate) are held from its H products to its dyln product, about 6000 cycles with
// the copy, the W2 block only to its DG product.  With three stages of all three blocks a chunk took 2100 cycles, the time of
// that loop by three (1600 now); the room came from X and dY, which take turns in one buffer.
constexpr int kW1S = 4, kW2S = 3;
constexpr int kSlabB = 32 * 64;                   // a row warp's [32 rows][32 columns] piece of X, dY or dx, 64-byte swizzle

struct TbP {
  int64_t M; int inner, n_mt, n_ch;
  uint32_t ab_fmt;
  const void *gamma, *beta;
  const float *mean, *rstd;
  float* part;                                   // [gridDim.x][2 K]
  int* status;
};

struct Bars {
  uint64_t x_full[kRowWarps], dy_full[kRowWarps], a_full, a_empty;
  uint64_t w1_full[kW1S], w1_empty[kW1S], w2_full[kW2S], w2_empty[kW2S];
  uint64_t xr_full[kRowWarps], hd_full[2], hd_empty[2], dh_full[2], dh_empty[2], st_done[2], acc_full, acc_empty;
};

__device__ __forceinline__ float tanh_approx(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <typename T>
__global__ void __launch_bounds__(kThreads, 1)
transition_bwd_tc_kernel(const __grid_constant__ CUtensorMap mdy,
                         const __grid_constant__ CUtensorMap mw1, const __grid_constant__ CUtensorMap mw2,
                         const __grid_constant__ CUtensorMap mdh, const __grid_constant__ CUtensorMap mg,
                         const __grid_constant__ CUtensorMap mx, const __grid_constant__ CUtensorMap mdx, const TbP p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sX = smem;                          // raw rows of X, then rows of dY
  uint8_t* sW1 = sX + A_BYTES;                 // [kW1S] value | gate blocks
  uint8_t* sW2 = sW1 + kW1S * 2 * WB;          // [kW2S]
  uint8_t* sDH = sW2 + kW2S * WB;              // [2] dh tiles
  uint8_t* sG = sDH + 2 * DH_BYTES;            // [2] g tiles
  uint8_t* sXR = sG + 2 * G_BYTES;             // rows of X once more, then rows of dx
  float4 (*red)[4][128] = reinterpret_cast<float4 (*)[4][128]>(sXR + A_BYTES);      // [2] row sums, exchanged by the row warps

  __shared__ Bars bar;
  __shared__ __align__(16) float gam_s[K], bet_s[K];
  __shared__ float sum_s[4][2 * K];            // gain and shift sums over each quarter of a tile's rows
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  if (tid == 0) {
    abort_s = 0;
    mbar_init(&bar.a_full, kRowWarps); mbar_init(&bar.a_empty, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bar.hd_full[i], 1); mbar_init(&bar.hd_empty[i], 8);
      mbar_init(&bar.dh_full[i], 8); mbar_init(&bar.dh_empty[i], 1); mbar_init(&bar.st_done[i], 1);
    }
    for (int i = 0; i < kW1S; ++i) { mbar_init(&bar.w1_full[i], 1); mbar_init(&bar.w1_empty[i], 1); }
    for (int i = 0; i < kW2S; ++i) { mbar_init(&bar.w2_full[i], 1); mbar_init(&bar.w2_empty[i], 1); }
    mbar_init(&bar.acc_full, 1); mbar_init(&bar.acc_empty, kRowWarps);
    for (int i = 0; i < kRowWarps; ++i) { mbar_init(&bar.xr_full[i], 1); mbar_init(&bar.x_full[i], 1); mbar_init(&bar.dy_full[i], 1); }
    mbar_fence_init();
    prefetch_tmap(&mx); prefetch_tmap(&mdy); prefetch_tmap(&mw1); prefetch_tmap(&mw2); prefetch_tmap(&mdh); prefetch_tmap(&mg); prefetch_tmap(&mdx);
  }
  for (int k = tid; k < K; k += kThreads) {
    gam_s[k] = to_f(static_cast<const T*>(p.gamma)[k]);
    bet_s[k] = p.beta ? to_f(static_cast<const T*>(p.beta)[k]) : 0.f;
  }
  for (int k = tid; k < 4 * 2 * K; k += kThreads) (&sum_s[0][0])[k] = 0.f;
  if (warp == 0) { tmem_alloc(&tmem_base_s, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  volatile int* abort_flag = &abort_s;
  const uint32_t tm0 = uniform(tmem_base_s);
  // TMEM columns: two buffers of (H value 32 | H gate 32 | DG 32); dyln accumulator 128; LN(X) 64; dY 64; two dh of 32
  const uint32_t tHD = tm0, tACC = tm0 + 192, tA = tm0 + 320, tDY = tm0 + 384, tDH = tm0 + 448;
  const int my_tiles = p.n_mt > (int)blockIdx.x ? (p.n_mt - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
  const int nch = p.n_ch;
  const int row_l = (warp & 3) * 32 + lane;
  const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;

  if (warp < kWorkWarps) {
    // ---------------------------------------------------------------------------------- workers
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kWorkRegs));
    const int team = warp >> 3, half = (warp >> 2) & 1;
    const uint32_t tMine = tHD + team * 96 + half * 16 + lane_addr, tOut = tDH + team * 32 + half * 16 + lane_addr;
    uint8_t* dh = sDH + team * DH_BYTES;
    uint8_t* g = sG + team * G_BYTES;
    int t = 0, c = team;                                  // my next chunk: c of tile t, once c is brought below nch
    for (uint32_t n = 0;; ++n, c += 2) {                  // n: my chunks so far
      while (t < my_tiles && c >= nch) { c -= nch; ++t; }
      if (t >= my_tiles || __any_sync(0xffffffffu, *abort_flag)) break;
      wait_or_flag(&bar.hd_full[team], n & 1, abort_flag);
      tc_fence_after();
      uint32_t gp[8], dv[8], db[8];
#pragma unroll
      for (int s = 0; s < 2; ++s) {                     // 8 columns at a time: registers
        uint32_t hv[8], hg[8], dg[8];
        tmem_ld8(tMine + s * 8, hv);
        tmem_ld8(tMine + 32 + s * 8, hg);
        tmem_ld8(tMine + 64 + s * 8, dg);
        tmem_ld_wait();
        if (s == 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar.hd_empty[team]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 v = make_float2(__uint_as_float(hv[2 * e]), __uint_as_float(hv[2 * e + 1]));
          const float2 b = make_float2(__uint_as_float(hg[2 * e]), __uint_as_float(hg[2 * e + 1]));
          const float2 d = make_float2(__uint_as_float(dg[2 * e]), __uint_as_float(dg[2 * e + 1]));
          const float2 h = make_float2(0.5f, 0.5f), b2 = mul2(b, h);
          const float2 sg = fma2(h, make_float2(tanh_approx(b2.x), tanh_approx(b2.y)), h);      // sigmoid(b)
          const float2 sl = mul2(b, sg);                                                         // silu(b)
          const float2 ds = fma2(sl, sub2(make_float2(1.f, 1.f), sg), sg);                       // d/db silu(b) = sg + sl * (1 - sg)
          const float2 go = mul2(sl, v), dvo = mul2(d, sl), dbo = mul2(mul2(d, v), ds);
          gp[s * 4 + e] = Pack2<T>::pack(go.x, go.y); dv[s * 4 + e] = Pack2<T>::pack(dvo.x, dvo.y); db[s * 4 + e] = Pack2<T>::pack(dbo.x, dbo.y);
        }
      }
      // dh to TMEM, once the dyln product of two chunks ago has read it; dh and g to the tiles, once the TMA stores have
      if (n > 0) wait_or_flag(&bar.dh_empty[team], (n - 1) & 1, abort_flag);
      tc_fence_after();
      tmem_st8(tOut, dv);
      tmem_st8(tOut + 8, db);
      if (n > 0) wait_or_flag(&bar.st_done[team], (n - 1) & 1, abort_flag);
      // dh row (128 B): [value 0-15 | gate 0-15 | value 16-31 | gate 16-31]; my 16 + 16 columns are chunks half*4 .. +3
      *reinterpret_cast<uint4*>(dh + swz_offset(row_l, half * 4 + 0, 128)) = make_uint4(dv[0], dv[1], dv[2], dv[3]);
      *reinterpret_cast<uint4*>(dh + swz_offset(row_l, half * 4 + 1, 128)) = make_uint4(dv[4], dv[5], dv[6], dv[7]);
      *reinterpret_cast<uint4*>(dh + swz_offset(row_l, half * 4 + 2, 128)) = make_uint4(db[0], db[1], db[2], db[3]);
      *reinterpret_cast<uint4*>(dh + swz_offset(row_l, half * 4 + 3, 128)) = make_uint4(db[4], db[5], db[6], db[7]);
      // g row (64 B): columns in natural order, mine are chunks half*2, half*2 + 1
      *reinterpret_cast<uint4*>(g + swz_offset(row_l, half * 2 + 0, 64)) = make_uint4(gp[0], gp[1], gp[2], gp[3]);
      *reinterpret_cast<uint4*>(g + swz_offset(row_l, half * 2 + 1, 64)) = make_uint4(gp[4], gp[5], gp[6], gp[7]);
      fence_async_smem();
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.dh_full[team]);
    }
  } else if (warp < kWorkWarps + kRowWarps) {
    // ---------------------------------------------------------------------------------- row warps
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRowRegs));
    const int quarter = warp & 3, part = (warp >> 2) & 1, me = part * 4 + quarter;      // rows 32 quarter .., columns 32 part .. and 64 + 32 part ..
    uint64_t* xr_full = &bar.xr_full[me];
    uint64_t* x_full = &bar.x_full[me];
    uint64_t* dy_full = &bar.dy_full[me];
    uint8_t* xr = sXR + me * 2 * kSlabB;
    uint8_t* xd = sX + me * 2 * kSlabB;
    auto row_of = [&](int t) { return ((int64_t)blockIdx.x + (int64_t)t * gridDim.x) * kRows; };
    auto slot = [&](uint8_t* slab, int q, int c) { return reinterpret_cast<uint4*>(slab + q * kSlabB + swz_offset(lane, c, 64)); };
    uint32_t n_raw = 0, n_x = 0, n_dy = 0;
    // (lane 0) my pieces of tile t: X and dY, in turn into one slab, each requested once the other is in registers; X once more
    // for the write-out
    auto load_x = [&](int t) {
      ++n_x;
      mbar_expect_tx(x_full, 2 * kSlabB);
      for (int q = 0; q < 2; ++q) tma_load_2d(xd + q * kSlabB, &mx, x_full, q * 64 + part * 32, (int)row_of(t) + quarter * 32);
    };
    auto load_dy = [&](int t) {
      ++n_dy;
      mbar_expect_tx(dy_full, 2 * kSlabB);
      for (int q = 0; q < 2; ++q) tma_load_2d(xd + q * kSlabB, &mdy, dy_full, q * 64 + part * 32, (int)row_of(t) + quarter * 32);
    };
    auto load_raw = [&](int t) {
      ++n_raw;
      mbar_expect_tx(xr_full, 2 * kSlabB);
      for (int q = 0; q < 2; ++q) tma_load_2d(xr + q * kSlabB, &mx, xr_full, q * 64 + part * 32, (int)row_of(t) + quarter * 32);
    };
    // LN(X) and dY of tile t to TMEM
    auto normalise = [&](int t) {
      const int64_t row = row_of(t) + row_l;
      const bool ok = row < p.M;
      const float mu = ok ? p.mean[row] : 0.f, rs = ok ? p.rstd[row] : 0.f;     // saved by the forward pass
      const float2 mm = make_float2(mu, mu), rr = make_float2(rs, rs);
      wait_or_flag(x_full, t & 1, abort_flag);
      uint32_t o[2][16];
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint4 raw = *slot(xd, q, c);
          const uint32_t u[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
          for (int e = 0; e < 4; e += 2) {
            const int k = q * 64 + part * 32 + c * 8 + e * 2;
            const float4 ga = *reinterpret_cast<const float4*>(gam_s + k), be = *reinterpret_cast<const float4*>(bet_s + k);
            const float2 y0 = fma2(mul2(sub2(Pack2<T>::unpack(u[e]), mm), rr), make_float2(ga.x, ga.y), make_float2(be.x, be.y));
            const float2 y1 = fma2(mul2(sub2(Pack2<T>::unpack(u[e + 1]), mm), rr), make_float2(ga.z, ga.w), make_float2(be.z, be.w));
            o[q][c * 4 + e] = ok ? Pack2<T>::pack(y0.x, y0.y) : 0u; o[q][c * 4 + e + 1] = ok ? Pack2<T>::pack(y1.x, y1.y) : 0u;
          }
        }
      fence_async_smem();
      __syncwarp();
      if (lane == 0 && !*abort_flag) load_dy(t);
      __syncwarp();
      if (t > 0) wait_or_flag(&bar.a_empty, (t - 1) & 1, abort_flag);      // the H / DG products of the previous tile
      tc_fence_after();
#pragma unroll
      for (int q = 0; q < 2; ++q) tmem_st16(tA + q * 32 + part * 16 + lane_addr, o[q]);
      wait_or_flag(dy_full, t & 1, abort_flag);
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint4 raw = *slot(xd, q, c);
          o[q][c * 4] = raw.x; o[q][c * 4 + 1] = raw.y; o[q][c * 4 + 2] = raw.z; o[q][c * 4 + 3] = raw.w;
        }
      fence_async_smem();
      __syncwarp();
      if (lane == 0 && t + 1 < my_tiles && !*abort_flag) load_x(t + 1);
      __syncwarp();
#pragma unroll
      for (int q = 0; q < 2; ++q) tmem_st16(tDY + q * 32 + part * 16 + lane_addr, o[q]);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.a_full);
    };
    if (my_tiles > 0) {
      if (lane == 0) { load_x(0); load_raw(0); }
      __syncwarp();
      normalise(0);
    }
    for (int t = 0; t < my_tiles; ++t) {
      if (t + 1 < my_tiles) normalise(t + 1);
      const int64_t row = row_of(t) + row_l;
      const bool ok = row < p.M;
      const float mu = ok ? p.mean[row] : 0.f, rs = ok ? p.rstd[row] : 0.f;
      wait_or_flag(xr_full, t & 1, abort_flag);
      wait_or_flag(&bar.acc_full, t & 1, abort_flag);
      if (named_sync_or(1 + quarter, 64, *abort_flag)) break;          // the two warps that exchange sums leave together
      tc_fence_after();
      uint32_t dy[64];
#pragma unroll
      for (int q = 0; q < 2; ++q) tmem_ld32(tACC + q * 64 + part * 32 + lane_addr, *reinterpret_cast<uint32_t (*)[32]>(dy + q * 32));
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.acc_empty);
      ln_bwd_half_row<T>(dy, mu, rs, gam_s, sum_s[quarter], red, part, row_l, lane, 1 + quarter, [&](int q, int c) { return slot(xr, q, c); });
      fence_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (row_of(t) + quarter * 32 < p.M)                 // never past the last row
          for (int q = 0; q < 2; ++q) tma_store_2d(&mdx, xr + q * kSlabB, q * 64 + part * 32, (int)row_of(t) + quarter * 32);
        bulk_commit_group();
        bulk_wait_group_read<0>();
        if (t + 1 < my_tiles) load_raw(t + 1);
      }
      __syncwarp();
    }
    if (lane == 0) { drain_ring(xr_full, n_raw, 1); drain_ring(x_full, n_x, 1); drain_ring(dy_full, n_dy, 1); bulk_wait_group<0>(); }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kIssueRegs));
    auto dead = [&] { return __any_sync(0xffffffffu, *abort_flag) != 0; };      // the MMA roles are run by whole warps
    if (warp == kFirstIssuer + 0) {
      // -------------------------------------------------------------------------------- MMA issuer: H and DG
      const uint32_t id_h = idesc_f16(128, 64, p.ab_fmt, 0, 1);     // B = W1 value|gate blocks MN-major, N = 64
      const uint32_t id_g = idesc_f16(128, 32, p.ab_fmt, 0, 1);     // A = dY, B = W2 block MN-major, N = 32
      uint32_t ch_cnt = 0, s1 = 0, u1 = 0, s2 = 0, u2 = 0;          // stages and how often they have been used
      for (int t = 0; t < my_tiles; ++t) {
        wait_or_flag(&bar.a_full, t & 1, abort_flag);
        for (int c = 0; c < nch; ++c, ++ch_cnt) {
          const int hb = ch_cnt & 1;
          wait_or_flag(&bar.w1_full[s1], u1 & 1, abort_flag);
          wait_or_flag(&bar.w2_full[s2], u2 & 1, abort_flag);
          if (ch_cnt >= 2) wait_or_flag(&bar.hd_empty[hb], ((ch_cnt >> 1) - 1) & 1, abort_flag);
          tc_fence_after();
          if (dead()) break;
          const uint32_t wh_lo = desc_lo(smem_u32(sW1), WB) + s1 * (2 * WB / 16), wg_lo = desc_lo(smem_u32(sW2), 16) + s2 * (WB / 16);
#pragma unroll
          for (int ks = 0; ks < K / 16; ++ks)      // H value | gate: the two blocks are the two atoms along N (LBO = WB)
            mma_ts_el(tHD + hb * 96, tA + ks * 8, wh_lo + ((ks * 1024) >> 4), desc_hi(512, kSw64), id_h, ks > 0);
#pragma unroll
          for (int ks = 0; ks < K / 16; ++ks)      // DG
            mma_ts_el(tHD + hb * 96 + 64, tDY + ks * 8, wg_lo + ((ks * 1024) >> 4), desc_hi(512, kSw64), id_g, ks > 0);
          tc_commit_el(&bar.hd_full[hb]);
          tc_commit_el(&bar.w2_empty[s2]);
          if (++s1 == kW1S) { s1 = 0; ++u1; }
          if (++s2 == kW2S) { s2 = 0; ++u2; }
        }
        if (dead()) break;
        tc_commit_el(&bar.a_empty);      // the H / DG products of this tile are all issued: LN(X) and dY are free when they complete
      }
    } else if (warp == kFirstIssuer + 2) {
      // -------------------------------------------------------------------------------- second MMA issuer: the dyln products
      // (one warp issuing both would wait for the workers' dh of one chunk before it could start the next chunk's H)
      const uint32_t id_a = idesc_f16(128, 128, p.ab_fmt, 0, 0);    // B = W1 blocks K-major, N = dim
      uint32_t ch_cnt = 0, s1 = 0;
      for (int t = 0; t < my_tiles; ++t) {
        for (int c = 0; c < nch; ++c, ++ch_cnt) {                   // dyln (+)= dh(c) [W1v; W1g](c)^T
          const int hb = ch_cnt & 1;
          wait_or_flag(&bar.dh_full[hb], (ch_cnt >> 1) & 1, abort_flag);
          if (c == 0 && t > 0) wait_or_flag(&bar.acc_empty, (t - 1) & 1, abort_flag);
          tc_fence_after();
          if (dead()) break;
          const uint32_t w_lo = desc_lo(smem_u32(sW1), 16) + s1 * (2 * WB / 16);
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            // k-step ks covers dh columns ks*16 .. +15: value (ks even) or gate (ks odd) columns (ks / 2) * 16 .. of the chunk
            mma_ts_el(tACC, tDH + hb * 32 + ks * 8, w_lo + (((ks & 1) * WB + (ks >> 1) * 32) >> 4), desc_hi(512, kSw64), id_a, c > 0 || ks > 0);
          tc_commit_el(&bar.dh_empty[hb]);
          tc_commit_el(&bar.w1_empty[s1]);
          if (++s1 == kW1S) s1 = 0;
        }
        if (dead()) break;
        tc_commit_el(&bar.acc_full);
      }
    } else if (warp == kFirstIssuer + 3 && lane == 0) {
      // -------------------------------------------------------------------------------- TMA stores of the dh / g tiles
      uint32_t ch_cnt = 0;
      for (int t = 0; t < my_tiles && !*abort_flag; ++t) {
        const int row0 = (int)(((int64_t)blockIdx.x + (int64_t)t * gridDim.x) * kRows);
        for (int c = 0; c < nch && !*abort_flag; ++c, ++ch_cnt) {
          const int hb = ch_cnt & 1;
          wait_or_flag(&bar.dh_full[hb], (ch_cnt >> 1) & 1, abort_flag);      // written and fenced by the team's eight warps
          if (*abort_flag) break;
          tma_store_3d(&mdh, sDH + hb * DH_BYTES, 0, row0, c);               // rows >= M are clipped
          tma_store_3d(&mg, sG + hb * G_BYTES, (c & 1) * kHC, row0, c >> 1);
          bulk_commit_group();
          bulk_wait_group_read<0>();
          mbar_arrive(&bar.st_done[hb]);                                       // the tiles have been read
        }
      }
      bulk_wait_group<0>();
    } else if (warp == kFirstIssuer + 1 && lane == 0) {
      // -------------------------------------------------------------------------------- TMA producer
      uint32_t n1 = 0, n2 = 0, s1 = 0, u1 = 0, s2 = 0, u2 = 0;
      for (int t = 0; t < my_tiles && !*abort_flag; ++t) {
        for (int c = 0; c < nch; ++c) {
          if (u1 > 0) wait_or_flag(&bar.w1_empty[s1], (u1 - 1) & 1, abort_flag);
          if (*abort_flag) break;
          mbar_expect_tx(&bar.w1_full[s1], 2 * WB);
          tma_load_2d(sW1 + s1 * 2 * WB, &mw1, &bar.w1_full[s1], c * kHC, 0);                    // value columns of W1
          tma_load_2d(sW1 + s1 * 2 * WB + WB, &mw1, &bar.w1_full[s1], p.inner + c * kHC, 0);     // gate columns of W1
          ++n1;
          if (++s1 == kW1S) { s1 = 0; ++u1; }
          if (u2 > 0) wait_or_flag(&bar.w2_empty[s2], (u2 - 1) & 1, abort_flag);
          if (*abort_flag) break;
          mbar_expect_tx(&bar.w2_full[s2], WB);
          tma_load_2d(sW2 + s2 * WB, &mw2, &bar.w2_full[s2], c * kHC, 0);                        // W2[:, chunk]
          ++n2;
          if (++s2 == kW2S) { s2 = 0; ++u2; }
        }
      }
      drain_ring(bar.w1_full, n1, kW1S);
      drain_ring(bar.w2_full, n2, kW2S);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (tid < 2 * K) p.part[(int64_t)blockIdx.x * 2 * K + tid] = (sum_s[0][tid] + sum_s[1][tid]) + (sum_s[2][tid] + sum_s[3][tid]);
  if (tid == 0 && abort_s) *reinterpret_cast<volatile int*>(p.status) = 1;
  if (warp == 0) tmem_dealloc(tmem_base_s, 512);
}

// dw1[k][n] from the chunk-ordered columns: position c*64 + [v0-15 | g0-15 | v16-31 | g16-31]
__global__ void unpermute_dw1_kernel(const float* __restrict__ src, float* __restrict__ dst, int inner) {
  const int k = blockIdx.x, two_i = 2 * inner;
  for (int pcol = threadIdx.x; pcol < two_i; pcol += blockDim.x) {
    const int c = pcol >> 6, w = pcol & 63;
    const int seg = w >> 4, off = w & 15;            // seg: 0 value lo, 1 gate lo, 2 value hi, 3 gate hi
    const int n = c * kHC + (seg >> 1) * 16 + off + ((seg & 1) ? inner : 0);
    dst[(int64_t)k * two_i + n] = src[(int64_t)k * two_i + pcol];
  }
}

}  // namespace

bool transition_bwd_fused_ok(const mf_transition_bwd_args& a) {
  if (a.dtype != MF_BF16 && a.dtype != MF_F16) return false;
  if (a.dim != 128 || a.inner % 32 != 0 || a.inner < 32 || !a.ln_w) return false;
  if (a.M < 1 || a.M > (int64_t)INT32_MAX) return false;
  const uintptr_t al = reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.dy) | reinterpret_cast<uintptr_t>(a.w1) |
                       reinterpret_cast<uintptr_t>(a.w2) | reinterpret_cast<uintptr_t>(a.dx);
  return (al & 15) == 0;
}

int transition_bwd_fused_blocks(int64_t M) {
  const int64_t tiles = (M + kRows - 1) / kRows;
  return (int)(tiles < sm_count() ? tiles : sm_count());
}

// g [panels of 64 columns][M][64], dh [inner/32][M][64] (chunk-ordered columns), dx, and per block the column sums part [blocks][2 * 128]
int transition_bwd_fused(const mf_transition_bwd_args& a, void* g, void* dh, float* part, cudaStream_t st) {
  CUtensorMap mx, mdy, mw1, mw2, mdh, mg, mdx;
  int r;
  {
    const int64_t dims[2] = {K, a.M}, str[2] = {1, K};
    const int slab[2] = {32, 32};                // half of a row warp's piece
    if ((r = make_tiled_map(&mx, a.x, a.dtype, 2, dims, str, slab, 64))) return r;
    if ((r = make_tiled_map(&mdy, a.dy, a.dtype, 2, dims, str, slab, 64))) return r;
    if ((r = make_tiled_map(&mdx, a.dx, a.dtype, 2, dims, str, slab, 64))) return r;
  }
  {
    const int64_t dims[2] = {2 * (int64_t)a.inner, K}, str[2] = {1, 2 * (int64_t)a.inner};
    const int box[2] = {kHC, K};
    if ((r = make_tiled_map(&mw1, a.w1, a.dtype, 2, dims, str, box, 64))) return r;
  }
  {
    const int64_t dims[2] = {a.inner, K}, str[2] = {1, a.inner};
    const int box[2] = {kHC, K};
    if ((r = make_tiled_map(&mw2, a.w2, a.dtype, 2, dims, str, box, 64))) return r;
  }
  {
    const int64_t dims[3] = {64, a.M, a.inner / kHC}, str[3] = {1, 64, 64 * a.M};
    const int box[3] = {64, kRows, 1};
    if ((r = make_tiled_map(&mdh, dh, a.dtype, 3, dims, str, box, 128))) return r;
  }
  {
    const int64_t dims[3] = {64, a.M, (a.inner + 63) / 64}, str[3] = {1, 64, 64 * a.M};
    const int box[3] = {kHC, kRows, 1};
    if ((r = make_tiled_map(&mg, g, a.dtype, 3, dims, str, box, 64))) return r;
  }
  TbP p{};
  p.M = a.M; p.inner = a.inner;
  p.n_mt = (int)((a.M + kRows - 1) / kRows);
  p.n_ch = a.inner / kHC;
  p.ab_fmt = a.dtype == MF_BF16 ? 1u : 0u;
  p.gamma = a.ln_w; p.beta = a.ln_b; p.mean = a.mean; p.rstd = a.rstd;
  p.part = part;
  p.status = status_word();
  MF_REQUIRE(p.status, MF_ERR_CUDA, "could not allocate the device status word");
  MF_REQUIRE(tc_async_status() == 0, MF_ERR_CUDA, "an earlier tensor-core kernel gave up on a bounded wait; results are invalid");
  constexpr size_t smem = 1024 + 2 * (size_t)A_BYTES + (2 * kW1S + kW2S) * (size_t)WB + 2 * (size_t)DH_BYTES + 2 * (size_t)G_BYTES + 2 * 4 * 128 * sizeof(float4);
  const int grid = transition_bwd_fused_blocks(a.M);
  if (a.dtype == MF_BF16) {
    constexpr auto kern = transition_bwd_tc_kernel<__nv_bfloat16>;
    if (int e = opt_in_smem<kern>(smem, kLaunchRegs)) return e;
    kern<<<grid, kThreads, smem, st>>>(mdy, mw1, mw2, mdh, mg, mx, mdx, p);
  } else {
    constexpr auto kern = transition_bwd_tc_kernel<__half>;
    if (int e = opt_in_smem<kern>(smem, kLaunchRegs)) return e;
    kern<<<grid, kThreads, smem, st>>>(mdy, mw1, mw2, mdh, mg, mx, mdx, p);
  }
  MF_LAUNCHED("transition_bwd_tc_kernel");
  return MF_OK;
}

int unpermute_dw1(const float* src, float* dst, int dim, int inner, cudaStream_t st) {
  unpermute_dw1_kernel<<<dim, 256, 0, st>>>(src, dst, inner);
  MF_LAUNCHED("unpermute_dw1_kernel");
  return MF_OK;
}

}  // namespace mf
