// General 16-bit GEMM on the tensor cores (tcgen05 + TMEM + TMA), used by the backward passes of LayernormLinear
// and Transition:   C[M, N] (+)= op(A) op(B)   with fp32 accumulation.
//
// Operands are row-major matrices described by how they are laid out relative to the reduction index r:
//   A "K-major":  stored [M, R]  (r contiguous)        A "MN-major": stored [R, M]  (m contiguous, i.e. A^T is given)
//   B "K-major":  stored [N, R]                        B "MN-major": stored [R, N]
// so that y = x W^T, dW = x^T dy, dg = dy W2 and friends all map onto it without a transposed copy.
//
// Persistent CTAs walk work items (128 x BN output tile, slice of the reduction).  A TMA ring of 192 KB feeds
// 64-deep slabs of A and B (128B-swizzled boxes), one elected lane issues 4 tcgen05.mma (M = 128, N = BN, K = 16) per slab
// into one of two TMEM accumulators, and four epilogue warps move finished tiles (each its own 32 rows) TMEM ->
// registers -> swizzled staging -> TMA store (16-bit or fp32) or TMA add-reduction (fp32, when the reduction is split over CTAs; the
// output must then be zero on entry).  All waits are bounded.
//
// With LN set, A is LayerNorm(x) for a matrix x whose rows are the reduction index (a weight gradient): two more
// warpgroups, taking alternate slabs, normalise x in shared memory between its arrival and the products, so that LN(x) is
// neither written by the pass before nor read here (one warpgroup could not keep up: 81 us for [147456, 128] x 512, 56 with
// two, 38 with tiles 256 columns wide, which normalise each slab half as often).
#include <type_traits>

#include "evo_tc_common.cuh"
#include "gemm_tc.cuh"

namespace mf {
namespace {
using namespace tcx;

constexpr int kBM = 128, kBK = 64;
constexpr int kMaxStages = 8;
constexpr int kThreads = 256, kLnThreads = 256;
template <int BN> struct Geo {
  static constexpr int kStageBytes = 16384 + BN * 128;      // A slab 16 KB + B slab
  static constexpr int kStages = BN == 64 ? 8 : BN == 128 ? 6 : 4;
  static constexpr size_t kSmem = 1024 + kStages * (size_t)kStageBytes + 32768;
};

struct GemmP {
  int m_tiles, n_tiles, k_splits, slabs_total, slabs_per_split;
  int n_cols; int64_t n_rows;
  int a_mn, b_mn, b_panels, out_kind;     // out_kind: 0 = 16-bit store, 1 = fp32 store, 2 = fp32 add-reduction
  uint32_t ab_fmt;
  const float *mean, *rstd; const void *gain, *shift; int m_total; int64_t r_total;      // LN only
  int* status;
};

struct Bars { uint64_t ready[kMaxStages], full[kMaxStages], empty[kMaxStages], acc_full[2], acc_empty[2]; };

__device__ __forceinline__ void tma_reduce_add_2d(const CUtensorMap* m, const void* src, int c0, int c1) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(src)), "r"(c0), "r"(c1) : "memory");
}

template <typename T, bool LN, int kBN>
__global__ void __launch_bounds__(kThreads + (LN ? kLnThreads : 0), 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap ma, const __grid_constant__ CUtensorMap mb,
               const __grid_constant__ CUtensorMap mc, const GemmP p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  constexpr int kStages = Geo<kBN>::kStages, kStageBytes = Geo<kBN>::kStageBytes;
  uint8_t* sStage = smem;                                  // [kStages][A | B]
  uint8_t* sOut = smem + kStages * kStageBytes;            // staging: two blocks of 128 rows x 128 bytes
  __shared__ Bars bar;
  __shared__ __align__(16) float gain_s[LN ? kBM : 4], shift_s[LN ? kBM : 4];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  if (tid == 0) {
    abort_s = 0;
    for (int i = 0; i < kStages; ++i) { mbar_init(&bar.full[i], 1); mbar_init(&bar.empty[i], 1); mbar_init(&bar.ready[i], 4); }
    for (int i = 0; i < 2; ++i) { mbar_init(&bar.acc_full[i], 1); mbar_init(&bar.acc_empty[i], 4); }
    mbar_fence_init();
    prefetch_tmap(&ma); prefetch_tmap(&mb); prefetch_tmap(&mc);
  }
  if (warp == 0) { tmem_alloc(&tmem_base_s, 2 * kBN); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  volatile int* abort_flag = &abort_s;
  const uint32_t tm0 = uniform(tmem_base_s);
  const int n_items = p.m_tiles * p.n_tiles * p.k_splits;
  auto decode = [&](int item, int& mt, int& nt, int& s0, int& s1) {
    const int ks = item % p.k_splits, rest = item / p.k_splits;
    nt = rest % p.n_tiles; mt = rest / p.n_tiles;
    s0 = ks * p.slabs_per_split;
    s1 = s0 + p.slabs_per_split; if (s1 > p.slabs_total) s1 = p.slabs_total;
  };

  if (warp == 0 && lane == 0) {
    // ------------------------------------------------------------------------------------ TMA producer
    uint32_t cnt = 0;
    for (int item = blockIdx.x; item < n_items && !*abort_flag; item += gridDim.x) {
      int mt, nt, s0, s1; decode(item, mt, nt, s0, s1);
      for (int s = s0; s < s1; ++s, ++cnt) {
        const int st = cnt % kStages;
        if (cnt >= kStages) wait_or_flag(&bar.empty[st], ((cnt / kStages) - 1) & 1, abort_flag);
        if (*abort_flag) break;
        uint8_t* a = sStage + st * kStageBytes; uint8_t* b = a + 16384;
        mbar_expect_tx(&bar.full[st], kStageBytes);
        if (p.a_mn) {   // stored [R, M]: two [64 r][64 m] boxes
          tma_load_2d(a, &ma, &bar.full[st], mt * kBM, s * kBK);
          tma_load_2d(a + 8192, &ma, &bar.full[st], mt * kBM + 64, s * kBK);
        } else {        // stored [M, R]: one [128 m][64 r] box
          tma_load_2d(a, &ma, &bar.full[st], s * kBK, mt * kBM);
        }
        if (p.b_panels) {
#pragma unroll
          for (int at = 0; at < kBN / 64; ++at) tma_load_3d(b + at * 8192, &mb, &bar.full[st], 0, s * kBK, nt * (kBN / 64) + at);
        } else if (p.b_mn) {
#pragma unroll
          for (int at = 0; at < kBN / 64; ++at) tma_load_2d(b + at * 8192, &mb, &bar.full[st], nt * kBN + at * 64, s * kBK);
        } else {
          tma_load_2d(b, &mb, &bar.full[st], s * kBK, nt * kBN);
        }
      }
    }
    drain_ring(bar.full, cnt, kStages);
  } else if (warp == 1) {
    // ------------------------------------------------------------------------------------ MMA issuer
    // Run by the whole warp, one elected lane issuing: with a single lane's branch and run-time descriptors an MMA took 100
    // to 240 cycles to issue, more than it takes to execute (see mma_ss_el).
    auto dead = [&] { return __any_sync(0xffffffffu, *abort_flag) != 0; };
    const uint32_t idesc = idesc_f16(128, kBN, p.ab_fmt, p.a_mn, p.b_mn);
    uint32_t cnt = 0, acc_cnt = 0;
    for (int item = blockIdx.x; item < n_items && !dead(); item += gridDim.x, ++acc_cnt) {
      int mt, nt, s0, s1; decode(item, mt, nt, s0, s1);
      const int ab = acc_cnt & 1;
      if (acc_cnt >= 2) wait_or_flag(&bar.acc_empty[ab], ((acc_cnt >> 1) - 1) & 1, abort_flag);
      for (int s = s0; s < s1; ++s, ++cnt) {
        const int st = cnt % kStages;
        wait_or_flag(LN ? &bar.ready[st] : &bar.full[st], (cnt / kStages) & 1, abort_flag);
        tc_fence_after();
        if (dead()) break;
        const uint32_t a0 = smem_u32(sStage + st * kStageBytes), b0 = a0 + 16384;
        // descriptor low words stepped by (bytes >> 4) per k-step: 16 rows of 128 B for MN-major, 32 B for K-major
        const uint32_t a_lo = p.a_mn ? desc_lo(a0, 8192) : desc_lo(a0, 16), a_step = p.a_mn ? 128u : 2u;
        const uint32_t b_lo = p.b_mn ? desc_lo(b0, 8192) : desc_lo(b0, 16), b_step = p.b_mn ? 128u : 2u;
#pragma unroll
        for (int ks = 0; ks < kBK / 16; ++ks)
          mma_ss_el(tm0 + ab * kBN, a_lo + ks * a_step, desc_hi(1024, kSw128), b_lo + ks * b_step, desc_hi(1024, kSw128), idesc, s > s0 || ks > 0);
        tc_commit_el(&bar.empty[st]);
      }
      tc_commit_el(&bar.acc_full[ab]);
    }
  } else if (LN && warp >= kThreads / 32) {
    // ------------------------------------------------------------------------------------ LayerNorm of the slabs of A
    // thread (row, half): 64 columns of one of the slab's 64 rows, in place
    const int t = tid - kThreads, group = t >> 7, row = t & 63, half = (t >> 6) & 1;
    uint32_t cnt = 0;
    int mt_have = -1;
    for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
      int mt, nt, s0, s1; decode(item, mt, nt, s0, s1);
      if (mt != mt_have) {
        named_sync(1, kLnThreads);
        const int m = mt * kBM + (t & 127);
        float v = 0.f;
        if (m < p.m_total) v = group == 0 ? to_f(static_cast<const T*>(p.gain)[m]) : p.shift ? to_f(static_cast<const T*>(p.shift)[m]) : 0.f;
        (group == 0 ? gain_s : shift_s)[t & 127] = v;
        named_sync(1, kLnThreads);
        mt_have = mt;
      }
      // row statistics are requested one of this group's slabs ahead
      float mu_next = 0.f, rs_next = 0.f;
      auto stats = [&](int s) {
        const int64_t r = (int64_t)s * kBK + row;
        const bool in = s < s1 && r < p.r_total;
        mu_next = in ? __ldg(p.mean + r) : 0.f; rs_next = in ? __ldg(p.rstd + r) : 0.f;
      };
      const int first = s0 + (int)((group ^ cnt) & 1);
      stats(first);
      for (int s = s0; s < s1; ++s, ++cnt) {
        if ((int)(cnt & 1) != group) continue;
        const int st = cnt % kStages;
        const bool ok = (int64_t)s * kBK + row < p.r_total;
        const float2 mm = make_float2(mu_next, mu_next), rr = make_float2(rs_next, rs_next);
        stats(s + 2);
        wait_or_flag(&bar.full[st], (cnt / kStages) & 1, abort_flag);
        uint8_t* a = sStage + st * kStageBytes + half * 8192;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          uint4* q = reinterpret_cast<uint4*>(a + swz_offset(row, c, 128));
          const uint4 v = *q;
          const uint32_t u[4] = {v.x, v.y, v.z, v.w};
          uint32_t o[4];
#pragma unroll
          for (int e = 0; e < 4; e += 2) {
            const float4 g = *reinterpret_cast<const float4*>(gain_s + half * 64 + c * 8 + e * 2), b = *reinterpret_cast<const float4*>(shift_s + half * 64 + c * 8 + e * 2);
            const float2 y0 = fma2(mul2(sub2(Pack2<T>::unpack(u[e]), mm), rr), make_float2(g.x, g.y), make_float2(b.x, b.y));
            const float2 y1 = fma2(mul2(sub2(Pack2<T>::unpack(u[e + 1]), mm), rr), make_float2(g.z, g.w), make_float2(b.z, b.w));
            o[e] = ok ? Pack2<T>::pack(y0.x, y0.y) : 0u; o[e + 1] = ok ? Pack2<T>::pack(y1.x, y1.y) : 0u;
          }
          *q = make_uint4(o[0], o[1], o[2], o[3]);
        }
        fence_async_smem();
        __syncwarp();
        if (__any_sync(0xffffffffu, *abort_flag)) break;
        if (lane == 0) mbar_arrive(&bar.ready[st]);
      }
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------------------------------ epilogue (128 threads)
    const int ew = warp - 4;
    const int row = ew * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(ew * 32) << 16;
    uint32_t acc_cnt = 0;
    for (int item = blockIdx.x; item < n_items; item += gridDim.x, ++acc_cnt) {
      int mt, nt, s0, s1; decode(item, mt, nt, s0, s1);
      const int ab = acc_cnt & 1;
      wait_or_flag(&bar.acc_full[ab], (acc_cnt >> 1) & 1, abort_flag);
      tc_fence_after();
      // every epilogue warp stages and stores its own 32-row slabs: no barrier between them.  A slab is 32 rows of 128
      // bytes (64 16-bit or 32 fp32 columns); the warp has two and fills one while the other is being stored.
      if (__any_sync(0xffffffffu, *abort_flag)) break;
      const int r0 = mt * kBM + ew * 32;
      const bool rows_in = (int64_t)r0 < p.n_rows;              // never start a store past the last row
#pragma unroll
      for (int cb = 0; cb < kBN / 32; ++cb) {
        uint32_t v[32];
        tmem_ld32(tm0 + ab * kBN + cb * 32 + lane_addr, v);
        tmem_ld_wait();
        if (cb == kBN / 32 - 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar.acc_empty[ab]);
        }
        const bool wide = p.out_kind != 0;
        uint8_t* slab = sOut + ((wide ? cb : cb >> 1) & 1) * 16384;
        if (wide || !(cb & 1)) {
          if (lane == 0) bulk_wait_group_read<1>();             // the store before the last one has read this slab
          __syncwarp();
        }
        if (!wide) {
#pragma unroll
          for (int ch = 0; ch < 4; ++ch) {
            uint4 o;
            o.x = Pack2<T>::pack(__uint_as_float(v[ch * 8]), __uint_as_float(v[ch * 8 + 1]));
            o.y = Pack2<T>::pack(__uint_as_float(v[ch * 8 + 2]), __uint_as_float(v[ch * 8 + 3]));
            o.z = Pack2<T>::pack(__uint_as_float(v[ch * 8 + 4]), __uint_as_float(v[ch * 8 + 5]));
            o.w = Pack2<T>::pack(__uint_as_float(v[ch * 8 + 6]), __uint_as_float(v[ch * 8 + 7]));
            *reinterpret_cast<uint4*>(slab + swz_offset(row, (cb & 1) * 4 + ch, 128)) = o;
          }
        } else {
#pragma unroll
          for (int ch = 0; ch < 8; ++ch)
            *reinterpret_cast<uint4*>(slab + swz_offset(row, ch, 128)) = make_uint4(v[ch * 4], v[ch * 4 + 1], v[ch * 4 + 2], v[ch * 4 + 3]);
        }
        if (wide || (cb & 1)) {
          fence_async_smem();
          __syncwarp();
          if (lane == 0) {
            const int c0 = nt * kBN + (wide ? cb : cb - 1) * 32;
            if (rows_in && c0 < p.n_cols) {                     // nor past the last column
              if (p.out_kind == 2) tma_reduce_add_2d(&mc, slab + ew * (32 * 128), c0, r0);
              else tma_store_2d(&mc, slab + ew * (32 * 128), c0, r0);
            }
            bulk_commit_group();
          }
        }
      }
    }
    if (lane == 0) bulk_wait_group<0>();
  }

  tc_fence_before();
  __syncthreads();
  if (tid == 0 && abort_s) *reinterpret_cast<volatile int*>(p.status) = 1;
  if (warp == 0) tmem_dealloc(tmem_base_s, 2 * kBN);
}

}  // namespace

bool gemm_tc_ok(const GemmTcArgs& g) {
  if (g.dtype != MF_BF16 && g.dtype != MF_F16) return false;
  if (g.M < 1 || g.N < 1 || g.R < 1 || g.M > INT32_MAX || g.R > INT32_MAX) return false;
  const int64_t a_pitch = g.a_mn ? g.M : g.R, b_pitch = g.b_mn ? g.N : g.R;
  if (a_pitch % 8 || b_pitch % 8) return false;
  if (g.out_kind == 0 ? (g.N % 8 != 0) : (g.N % 4 != 0)) return false;
  const uintptr_t al = reinterpret_cast<uintptr_t>(g.a) | reinterpret_cast<uintptr_t>(g.b) | reinterpret_cast<uintptr_t>(g.c);
  return (al & 15) == 0;
}

int gemm_tc(const GemmTcArgs& g, cudaStream_t st) {
  MF_REQUIRE(gemm_tc_ok(g), MF_ERR_UNSUPPORTED, "gemm_tc: shape or alignment not supported");
  CUtensorMap ma, mb, mc;
  int r;
  {
    const int64_t dims[2] = {g.a_mn ? g.M : g.R, g.a_mn ? g.R : g.M}, str[2] = {1, dims[0]};
    const int box[2] = {64, g.a_mn ? 64 : 128};
    if ((r = make_tiled_map(&ma, g.a, g.dtype, 2, dims, str, box, 128))) return r;
  }
  {
    const int64_t dims[2] = {g.N, g.M}, str[2] = {1, g.N};
    const int box[2] = {g.out_kind == 0 ? 64 : 32, 32};      // one epilogue warp's slab
    if ((r = make_tiled_map(&mc, g.c, g.out_kind == 0 ? g.dtype : MF_F32, 2, dims, str, box, 128))) return r;
  }
  GemmP p{};
  p.m_tiles = (int)((g.M + kBM - 1) / kBM);
  p.slabs_total = (int)((g.R + kBK - 1) / kBK);
  const int sms = sm_count();
  // Columns of an output tile.  256 where the reduction is split anyway and long enough that every SM still gets 16 slabs:
  // A (and its normalisation) is then gone through half as often.  64 where 128 would leave half of the chip without a tile.
  int bn = 128;
  if (g.out_kind == 2 && g.N > 128 && (int64_t)p.m_tiles * ((g.N + 255) / 256) * (p.slabs_total / 16) >= sms) bn = 256;
  else if ((int64_t)p.m_tiles * ((g.N + 127) / 128) * (g.out_kind == 2 ? (p.slabs_total + 3) / 4 : 1) <= sms / 2) bn = 64;
  p.n_tiles = (int)((g.N + bn - 1) / bn);
  if (g.b_panels) {
    const int64_t dims[3] = {64, g.R, (g.N + 63) / 64}, str[3] = {1, 64, 64 * g.R};
    const int box[3] = {64, 64, 1};
    if ((r = make_tiled_map(&mb, g.b, g.dtype, 3, dims, str, box, 128))) return r;
  } else {
    const int64_t dims[2] = {g.b_mn ? g.N : g.R, g.b_mn ? g.R : g.N}, str[2] = {1, dims[0]};
    const int box[2] = {64, g.b_mn ? 64 : bn};
    if ((r = make_tiled_map(&mb, g.b, g.dtype, 2, dims, str, box, 128))) return r;
  }
  int splits = 1;
  if (g.out_kind == 2) {
    // split the reduction so that every SM has work once (each split adds its tile to the output through memory), but keep
    // slices of at least four slabs
    splits = sms / (p.m_tiles * p.n_tiles);
    const int cap = p.slabs_total / 4;
    if (splits > cap) splits = cap;
    if (splits < 1) splits = 1;
  }
  p.slabs_per_split = (p.slabs_total + splits - 1) / splits;
  p.k_splits = (p.slabs_total + p.slabs_per_split - 1) / p.slabs_per_split;
  p.n_cols = (int)g.N; p.n_rows = g.M;
  p.a_mn = g.a_mn; p.b_mn = g.b_mn; p.b_panels = g.b_panels; p.out_kind = g.out_kind;
  p.ab_fmt = g.dtype == MF_BF16 ? 1u : 0u;
  p.mean = g.ln_mean; p.rstd = g.ln_rstd; p.gain = g.ln_gain; p.shift = g.ln_shift; p.m_total = (int)g.M; p.r_total = g.R;
  MF_REQUIRE(!g.ln_gain || g.a_mn, MF_ERR_UNSUPPORTED, "gemm_tc: LayerNorm is applied along the rows of an MN-major A");
  p.status = status_word();
  MF_REQUIRE(p.status, MF_ERR_CUDA, "could not allocate the device status word");
  MF_REQUIRE(tc_async_status() == 0, MF_ERR_CUDA, "an earlier tensor-core kernel gave up on a bounded wait; results are invalid");
  if (g.out_kind == 2 && !g.accumulate) MF_CUDA(cudaMemsetAsync(g.c, 0, sizeof(float) * (size_t)g.M * g.N, st));
  const int n_items = p.m_tiles * p.n_tiles * p.k_splits;
  const int grid = sms < n_items ? sms : n_items;
  auto launch = [&](auto type, auto ln, auto width) -> int {
    constexpr bool LN = decltype(ln)::value;
    constexpr int BN = decltype(width)::value;
    constexpr auto kern = gemm_tc_kernel<decltype(type), LN, BN>;
    if (int e = opt_in_smem<kern>(Geo<BN>::kSmem)) return e;
    kern<<<grid, kThreads + (LN ? kLnThreads : 0), Geo<BN>::kSmem, st>>>(ma, mb, mc, p);
    return MF_OK;
  };
  auto with_width = [&](auto type, auto ln) {
    return bn == 64 ? launch(type, ln, std::integral_constant<int, 64>{}) : bn == 128 ? launch(type, ln, std::integral_constant<int, 128>{})
                                                                                     : launch(type, ln, std::integral_constant<int, 256>{});
  };
  auto with_ln = [&](auto type) { return g.ln_gain ? with_width(type, std::true_type{}) : with_width(type, std::false_type{}); };
  r = g.dtype == MF_BF16 ? with_ln(__nv_bfloat16{}) : with_ln(__half{});
  if (r) return r;
  MF_LAUNCHED("gemm_tc_kernel");
  return MF_OK;
}

}  // namespace mf
