// Pair-biased masked attention backward on the tensor cores (tcgen05 + TMEM + TMA), head sizes up to 64 (as one or two
// halves of 32 columns, template parameter NH).
//
// Two kernels share the transposed-score scheme (keys on the TMEM lanes):
//
//   S''^T = K_j Q_i^T + sqrt(D) * bias^T + terms        dP''^T = V_j dO_i^T - delta_i      (tcgen05.mma into TMEM; the bias
//   P^T   = 2^(c1 * S''^T)                              dS^T   = P^T dP''^T                 term is itself a product with
//   alpha * I, and the key mask, the log-sum-exp and delta enter through one more K = 16 product: evo_tc_common.cuh)
//
// evo_bwd_ws_kernel (dQ, dK, dV).  A persistent CTA (768 threads) owns a (b, n, h) - or a range of its key tiles - and walks the
// key tiles j and, inside, the query tiles i in HALF blocks of [128 keys x 64 queries].  Two teams of eight compute
// warps take alternate half blocks, each with its own score buffers in TMEM, so that the tensor pipe works on one
// team's products while the other team exponentiates.  A thread (key row, 32 query columns) writes packed 16-bit
// P^T and dS^T back over the scores it has just read: they are the TMEM A operands of  dV_j += P^T dO_i  and
// dK_j += dS^T Q_i.  dS^T also goes to a shared-memory tile, read MN-major as the A operand of  dQ_i += dS K_j.
// dK_j / dV_j accumulate in TMEM over the query tiles and dQ_i over the key tiles (or, for long rows and split
// items, leave block by block through fp32 adds in global memory).
//
// evo_dbias_ws_kernel (dBias = sum of dS over the N rows that share the bias).  A CTA keeps ONE (b, h, i tile,
// j tile) and walks a range of rows n: scores and dP for row n+1 are produced while the 16 compute warps turn row n
// into dS and add it to register accumulators; nothing is reduced through memory until the range is done.  Ranges
// are summed in a fixed order afterwards, so dBias is bit-reproducible.  With one row per bias (N = 1) the kernel is not
// run: dS is the answer and evo_bwd_ws_kernel stores it.
//
// delta_i = rowsum(dO_i * O_i) and the term tiles come from a small pre-kernel.  The bias tile of a half block is the A
// operand [128 keys x 16 queries] of the products that add it: the caller's bias ([queries][keys]) is exactly that in
// MN-major form and is loaded in place when TMA can address it; otherwise a 16-bit copy with a 16-byte pitch is made
// first (copy_bias_rows: [4, 32, 384, 384] fp32 in 20 us, where the transposed copy made before took 38).  All waits are bounded
// (tc.cuh); on expiry the CTA runs dry without touching global memory and the host sees mf_async_status() != 0.
#include <type_traits>

#include "evo_tc_common.cuh"

namespace mf {
namespace {
using namespace tcx;

constexpr int kT = 128;             // tile edge (keys and queries)
constexpr int kHalf = 64;           // queries per half block
constexpr int kComputeWarps = 16;
constexpr int kThreads = (kComputeWarps + 4) * 32;
constexpr int kTileB = 128 * 64;    // [128 x 32] 16-bit operand tile, 64-byte rows, 64B swizzle
constexpr int kAtomB = 128 * 128;   // [128 x 64] 16-bit tile, 128-byte rows, 128B swizzle (bias atoms, dS^T atoms)
constexpr int kDP = 32;             // padded head size
// Head sizes up to 64 are handled as NH = 1 or 2 halves of 32 columns: every operand is loaded as NH tiles of [128 x 32]
// (the same layout whatever the head size), the score products run over 2 * NH slices of 16, and each half has its own
// 32 columns in the dK, dV and dQ accumulators.  With two halves the stages are twice as large, so there are fewer:
template <int NH> struct Geo {
  static constexpr int kStageB = 2 * NH * kTileB + 4096;            // main kernel: a (K, V, XK) or (Q, dO, XQ) stage
  static constexpr int kDbStageB = 4 * NH * kTileB + 2 * 4096;      // dBias kernel: one row's Q, dO, K, V tiles and its two term tiles
  static constexpr int NQ = NH == 1 ? 3 : 2;       // (Q, dO, XQ) stages
  static constexpr int NKV = NH == 1 ? 2 : 1;      // (K, V, XK) stages
  static constexpr int NB = NH == 1 ? 3 : 2;       // bias atoms
  static constexpr int NS = NH == 1 ? 3 : 2;       // dBias kernel: operand stages
  static constexpr size_t kMainSmem = 1024 + 4 * (size_t)kAtomB + NB * (size_t)kAtomB + (NQ + NKV) * (size_t)kStageB + 2048 + kXTileB;
  static constexpr size_t kDbSmem = 1024 + 2 * (size_t)kAtomB + NS * (size_t)kDbStageB + 2048 + kXTileB;
};
static_assert(Geo<2>::kMainSmem + 1024 <= 227 * 1024 && Geo<1>::kMainSmem + 1024 <= 227 * 1024, "shared memory of the main kernel");
static_assert(Geo<2>::kDbSmem + 1024 <= 227 * 1024 && Geo<1>::kDbSmem + 1024 <= 227 * 1024, "shared memory of the dBias kernel");
constexpr int kMainThreads = kThreads + 128;      // the main kernel has four write-out warps besides
// registers per thread: at launch / compute warps / helper (and write-out) warps after setmaxnreg.  The raise of the
// compute warps can only draw on what the others release inside the CTA - otherwise it never returns.
constexpr int kLaunchRegs = 96, kComputeRegs = 104, kHelperRegs = 64;
static_assert(kComputeWarps * 32 * kComputeRegs + 128 * kHelperRegs <= kThreads * kLaunchRegs, "setmaxnreg budget");
constexpr int kMainLaunchRegs = 80, kMainComputeRegs = 96, kMainHelperRegs = 48;
static_assert(kComputeWarps * 32 * kMainComputeRegs + 256 * kMainHelperRegs <= kMainThreads * kMainLaunchRegs, "setmaxnreg budget");

struct BwdWsP {
  int B, N, L, H, D;
  int n_t, n_items, lpad;
  int ksplit;            // work items per (b, n, h): the key tiles are split into this many ranges
  int step[4];           // the grid size as (range, h, n, b) digits: from one item of a CTA to its next
  int dq_stream;         // dQ leaves the SM block by block (more query tiles than TMEM holds)
  int dbuf;              // dK/dV accumulators double-buffered over the key tiles
  float* dq_acc;         // fp32 [B,N,L,H,D] accumulator of dQ when ksplit > 1 or dq_stream
  float c1, scale, inv_L;
  uint32_t fmt, bfmt;
  int n_alpha; float alpha[2];
  int bias_b_mul;
  const uint8_t* xq; const uint8_t* xk;     // rank-one term tiles (evo_extras_ws_kernel)
  const int* flags;                         // per (b, n, h): every key of the row is masked
  void* dbias_direct;                       // N == 1 and a 16-bit d_pair_bias: dS is the answer, written by this kernel
  void *dq, *dk, *dv; TokenStrides gs;
  int* status;
};

// Work item of a CTA: a range of the key tiles of (b, n, h).  The first one is taken apart by divisions, the others are
// stepped to: six divisions per item and role, executed once in 30000 cycles and so each time from a cold instruction cache,
// took 1000 cycles.
struct Item {
  int sp, h, n, b;
  __device__ __forceinline__ Item(int item, const BwdWsP& p) {
    sp = item % p.ksplit;
    const int bnh = item / p.ksplit, bn = bnh / p.H;
    h = bnh - bn * p.H; b = bn / p.N; n = bn - b * p.N;
  }
  __device__ __forceinline__ void step(const BwdWsP& p) {
    sp += p.step[0]; h += p.step[1]; n += p.step[2]; b += p.step[3];
    if (sp >= p.ksplit) { sp -= p.ksplit; ++h; }
    if (h >= p.H) { h -= p.H; ++n; }
    if (n >= p.N) { n -= p.N; ++b; }
  }
  __device__ __forceinline__ int bn(const BwdWsP& p) const { return b * p.N + n; }
  __device__ __forceinline__ int bnh(const BwdWsP& p) const { return bn(p) * p.H + h; }
  __device__ __forceinline__ int jt0(const BwdWsP& p) const { return p.ksplit == 1 ? 0 : sp * p.n_t / p.ksplit; }
  __device__ __forceinline__ int jt1(const BwdWsP& p) const { return p.ksplit == 1 ? p.n_t : (sp + 1) * p.n_t / p.ksplit; }
};

// Every role waits for each phase of a barrier in turn (see tc.cuh).  That is why dQ on chip has a barrier of its own, item_dq: the
// write-out warps would use one phase of dq_done an item, and nothing that they wait for says how far the dQ products have
// come (the compute warps hand P and dS over before they wait for the product of two blocks ago).  The issuer starts an item's dQ
// behind item_done of the item before, so that item_dq cannot run ahead.
struct Bars {
  uint64_t kv_full[2], kv_empty[2], qd_full[3], qd_empty[3], bt_full[3], bt_empty[3];
  uint64_t sd_ready[2], written[2], buf_free[2];
  uint64_t ds_written[2], dq_done[2];        // per block parity: dS^T tile complete in shared memory / its dQ product complete
  uint64_t kv_done[2], kv_drained[2];        // by parity: the dK / dV accumulation of a key tile is complete / has been read out
  uint64_t item_dq, item_done[2];            // the item's on-chip dQ accumulators are complete / have been read out
  uint64_t dq_drained[2];
};

// 1-D bulk copy global -> shared, completion counted in bytes on `bar` (addresses and size multiples of 16 bytes)
__device__ __forceinline__ void bulk_load_1d(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// One thread per (b, n, i < lpad, h): delta = sum_d dO * O (D is a multiple of 8), the XQ row of query i and, for h == 0,
// the XK row of key i.  Consecutive threads take the heads of one token, then the next token: a warp's pieces of o and dO
// are contiguous, token by token.  A block stays in one row (b, n), so that indexes are taken apart in 32 bits (21.8 -> 20.5 us
// for [1, 384, 384, 4, 32], 14.4 of them the bytes).  Above 32 columns (DP = 64) a warp fetches its pieces together and hands
// them out through shared memory: with every thread reading its own 2 D bytes each load instruction touched 32 lines
// ([4, 1, 384, 32, 64]: 13.7 -> 8.3 us; at 32 columns the detour costs 1 us more than it gives).
// flags[bnh]: the row (b, n) has every key masked (lse = -FLT_MAX, for all of its queries alike).  The fp32 accumulator of
// dQ, where one is used, is cleared here as well: each memset in front of the kernels cost 2 us of GPU time and as much of
// the host's.
constexpr int kXWarps = 4;
template <typename T, int DP>
__global__ void __launch_bounds__(kXWarps * 32) evo_extras_ws_kernel(const T* __restrict__ o, TokenStrides os, const T* __restrict__ d_o, TokenStrides ds, const float* __restrict__ lse,
                                     const void* __restrict__ mask, int64_t ms_b, int64_t ms_n, int64_t ms_l, int mask_dtype,
                                     uint8_t* __restrict__ xq, uint8_t* __restrict__ xk, int* __restrict__ flags,
                                     float* __restrict__ dq_acc, int row_blocks, int N, int L, int lpad, int H, int D) {
  constexpr bool kShared = DP > 32;
  __shared__ uint4 piece_s[kShared ? kXWarps : 1][2][32 * (DP / 8 + 1)];
  const int bn = (int)(blockIdx.x / (unsigned)row_blocks), b = bn / N, n = bn - b * N;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned first = ((blockIdx.x - (unsigned)bn * row_blocks) * kXWarps + warp) * 32, total = (unsigned)lpad * H, real = (unsigned)L * H;
  const int per_row = D / 8, pitch = per_row | 1;        // 16-byte pieces; odd: no bank conflicts
#pragma unroll
  for (int k0 = 0; kShared && k0 < DP / 8; k0 += 4) {
    uint4 a[4], g[4];
    int at[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int f = (k0 + k) * 32 + lane, pr = f / per_row, c = f - pr * per_row;
      const unsigned idx = first + pr;
      at[k] = pr < 32 && idx < real ? pr * pitch + c : -1;
      if (at[k] >= 0) {
        const int i = (int)(idx / (unsigned)H), h = (int)(idx - (unsigned)i * H);
        a[k] = __ldg(reinterpret_cast<const uint4*>(o + os.at(b, n, i) + h * D) + c);
        g[k] = __ldg(reinterpret_cast<const uint4*>(d_o + ds.at(b, n, i) + h * D) + c);
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (at[k] >= 0) { piece_s[warp][0][at[k]] = a[k]; piece_s[warp][1][at[k]] = g[k]; }
  }
  if (dq_acc && first < real) {
    float4* z = reinterpret_cast<float4*>(dq_acc + ((int64_t)bn * real + first) * D);
    const int n_z = (int)(real - first < 32u ? real - first : 32u) * (D / 4);
    for (int f = lane; f < n_z; f += 32) z[f] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (kShared) __syncwarp();
  const unsigned idx = first + lane;
  if (idx >= total) return;
  const int i = (int)(idx / (unsigned)H), h = (int)(idx - (unsigned)i * H);
  const float sqrt_d = sqrtf((float)D);
  const __nv_bfloat16 one = __float2bfloat16_rn(1.f), zero = __float2bfloat16_rn(0.f);
  const int nt = lpad / 128, tile = i >> 7, r = i & 127;
  {
    const int64_t bnh = (int64_t)bn * H + h;
    float nl = kMinusBig, nd = 0.f;
    if (i < L) {
      float dl = 0.f;
      const uint4* po = reinterpret_cast<const uint4*>(o + os.at(b, n, i) + h * D);
      const uint4* pg = reinterpret_cast<const uint4*>(d_o + ds.at(b, n, i) + h * D);
#pragma unroll 4
      for (int c = 0; c < per_row; ++c) {
        const uint4 a = kShared ? piece_s[warp][0][lane * pitch + c] : __ldg(po + c), g = kShared ? piece_s[warp][1][lane * pitch + c] : __ldg(pg + c);
        const uint32_t av[4] = {a.x, a.y, a.z, a.w}, gv[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 x = Pack2<T>::unpack(av[e]), y = Pack2<T>::unpack(gv[e]);
          dl = fmaf(x.x, y.x, dl); dl = fmaf(x.y, y.y, dl);
        }
      }
      nd = -dl;
      const float lv = lse[bnh * L + i];
      const bool masked = lv <= -3e38f;
      if (!masked) nl = -lv * sqrt_d;
      if (i == 0) flags[bnh] = masked;
    }
    __nv_bfloat16 a[3], b[3];
    split3(nl, a); split3(nd, b);
    uint8_t* base = xq + ((int64_t)bnh * nt + tile) * kXTileB;
    *reinterpret_cast<uint4*>(base + swz_offset(r, 0, 32)) = make_uint4(pack_bf(one, one), pack_bf(one, a[0]), pack_bf(a[1], a[2]), pack_bf(b[0], b[1]));
    *reinterpret_cast<uint4*>(base + swz_offset(r, 1, 32)) = make_uint4(pack_bf(b[2], zero), 0u, 0u, 0u);
  }
  if (h == 0) {
    float mv = kMinusBig;
    if (i < L) {
      const int64_t mi = b * ms_b + n * ms_n + (int64_t)i * ms_l;
      mv = mask_dtype == MF_U8 ? (static_cast<const uint8_t*>(mask)[mi] ? 0.f : kMinusBig) : fmaxf(load_rt(mask, mi, mask_dtype) * sqrt_d, kMinusBig);
    }
    __nv_bfloat16 m[3];
    split3(mv, m);
    uint8_t* base = xk + ((int64_t)bn * nt + tile) * kXTileB;
    *reinterpret_cast<uint4*>(base + swz_offset(r, 0, 32)) = make_uint4(pack_bf(m[0], m[1]), pack_bf(m[2], one), pack_bf(one, one), 0u);
    *reinterpret_cast<uint4*>(base + swz_offset(r, 1, 32)) = make_uint4(0u, 0u, 0u, 0u);
  }
}

// P^T and dS^T of one thread for 16 query columns.  sr: scores S''^T with the bias, mask and log-sum-exp terms already
// inside (see the rank-one terms above), dr: dP^T - delta.  Results packed two queries per word.  `careful`: the row (b, n)
// has every key masked - P is uniform over the keys of the row and no gradient passes through the (masked) logits.
template <typename T>
__device__ __forceinline__ void p_and_ds(const uint32_t (&sr)[16], const uint32_t (&dr)[16], float c1, bool careful,
                                         float p_uniform, uint32_t* __restrict__ pp, uint32_t* __restrict__ dd) {
  const float2 c1c1 = make_float2(c1, c1);
  if (careful) {
    const uint32_t pu = Pack2<T>::pack(p_uniform, p_uniform);
#pragma unroll
    for (int c = 0; c < 8; ++c) { pp[c] = pu; dd[c] = 0u; }
    return;
  }
#pragma unroll
  for (int c2 = 0; c2 < 8; ++c2) {
    const float2 xx = mul2(make_float2(__uint_as_float(sr[c2 * 2]), __uint_as_float(sr[c2 * 2 + 1])), c1c1);
    const float2 pr = make_float2(ex2f(xx.x), ex2f(xx.y));
    const float2 ds = mul2(pr, make_float2(__uint_as_float(dr[c2 * 2]), __uint_as_float(dr[c2 * 2 + 1])));
    pp[c2] = Pack2<T>::pack(pr.x, pr.y);
    dd[c2] = Pack2<T>::pack(ds.x, ds.y);
  }
}

template <typename T, typename TB, bool DQS, int NH>      // DQS: dQ streamed block by block through global memory
__global__ void __launch_bounds__(kMainThreads, 1)
evo_bwd_ws_kernel(const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mk,
                  const __grid_constant__ CUtensorMap mv, const __grid_constant__ CUtensorMap mg,
                  const __grid_constant__ CUtensorMap mbt, const BwdWsP p MF_TRACE_PARAM) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  constexpr int kStageB = Geo<NH>::kStageB, NQ = Geo<NH>::NQ, NKV = Geo<NH>::NKV, NB = Geo<NH>::NB;
  uint8_t* sDS = smem;                          // [2 blocks][2 atoms]: dS^T tiles for the dQ product
  uint8_t* sBT = sDS + 4 * kAtomB;              // bias atoms, ring of NB
  uint8_t* sKV = sBT + NB * kAtomB;             // [NKV stages][K halves, V halves, XK]
  uint8_t* sQD = sKV + NKV * kStageB;           // [NQ stages][Q halves, dO halves, XQ]
  uint8_t* sI = sQD + NQ * kStageB;             // alpha * I, two terms
  uint8_t* sXC = sI + 2048;                     // constant tile of the -delta term

  __shared__ Bars bar;
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;

  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  if (tid == 0) {
    abort_s = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bar.kv_full[i], 1); mbar_init(&bar.kv_empty[i], 1);
      mbar_init(&bar.sd_ready[i], 1); mbar_init(&bar.written[i], kComputeWarps / 2);
      mbar_init(&bar.buf_free[i], 1);
      mbar_init(&bar.ds_written[i], kComputeWarps); mbar_init(&bar.dq_done[i], 1);
      mbar_init(&bar.item_done[i], 4);
      mbar_init(&bar.dq_drained[i], 4);
      mbar_init(&bar.kv_done[i], 1); mbar_init(&bar.kv_drained[i], 4);
    }
    mbar_init(&bar.item_dq, 1);
    for (int i = 0; i < 3; ++i) {
      mbar_init(&bar.qd_full[i], 1); mbar_init(&bar.qd_empty[i], 1); mbar_init(&bar.bt_full[i], 1); mbar_init(&bar.bt_empty[i], 1);
    }
    mbar_fence_init();
    prefetch_tmap(&mq); prefetch_tmap(&mk); prefetch_tmap(&mv); prefetch_tmap(&mg); prefetch_tmap(&mbt);
  }
  write_alpha_identity<TB>(sI, p.alpha[0], tid, kMainThreads);
  write_alpha_identity<TB>(sI + 1024, p.alpha[1], tid, kMainThreads);
  write_xc_tile(sXC, tid, kMainThreads);
  fence_async_smem();
  if (warp == 0) { tmem_alloc(&tmem_base_s, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  volatile int* abort_flag = &abort_s;
  const uint32_t tm0 = uniform(tmem_base_s);
  const int nt = p.n_t;
  const bool dbuf = p.dbuf != 0;
  // TMEM: team t's scores S''^T at t*128 + [0,64), dP^T at t*128 + [64,128) (P^T / dS^T are packed over them);
  // dK | dV accumulators (one or two sets); dQ accumulators (one per query tile, or two used in turn when streaming)
  // (each accumulator has 32 columns per head half: dK = [0, 32 NH), dV = [32 NH, 64 NH) of a set)
  const uint32_t tKV = tm0 + 256, tDQ = tm0 + 256 + (dbuf ? 128 : 64) * NH;
  const uint32_t kv_set = dbuf ? 64 * NH : 0;    // column distance between the two dK|dV accumulator sets

  if (warp < kComputeWarps) {
    // ============================================================================ compute warps
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kMainComputeRegs));
    const int team = warp >> 3;                       // takes the half blocks with (half == team)
    const int ch = (warp >> 2) & 1;                   // which 32 of the half block's 64 query columns
    const int r = (warp & 3) * 32 + lane;             // TMEM lane = key row inside the tile
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tST = tm0 + team * 128 + ch * 32 + lane_addr, tDP = tST + 64;
    MF_TRACE_DECL(tr, team, blockIdx.x == 0 && (warp == 0 || warp == 8) && lane == 0);

    uint32_t g = 0;                 // full blocks seen by this CTA (both teams count every block)
    Item at(blockIdx.x, p);
    int special_next = p.flags[at.bnh(p)];
    for (int item = blockIdx.x; item < p.n_items; item += gridDim.x) {
      const int h = at.h, b = at.b, jt0 = at.jt0(p), jt1 = at.jt1(p);
      const bool special = special_next != 0;      // every key of the row is masked: the item takes the careful path
      at.step(p);
      if (item + (int)gridDim.x < p.n_items) special_next = p.flags[at.bnh(p)];
      for (int jt = jt0; jt < jt1; ++jt) {
        const int j = jt * kT + r;
        const float p_uniform = j < p.L ? p.inv_L : 0.f;       // careful path: P of a fully masked row
        for (int it = 0; it < nt; ++it, ++g) {
          // ---- S''^T, dP^T of my half block -> registers
          tr(1);
          wait_or_flag(&bar.sd_ready[team], g & 1, abort_flag);
          tc_fence_after();
          tr(2);
          uint32_t pp[16], dd[16];
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {        // 16 query columns at a time keeps the live registers down
            uint32_t sr[16], dr[16];
            tmem_ld16(tST + hf * 16, sr);
            tmem_ld16(tDP + hf * 16, dr);
            tmem_ld_wait();
            if (hf == 0) tr(3);
            p_and_ds<T>(sr, dr, p.c1, special, p_uniform, pp + hf * 8, dd + hf * 8);
          }
          tr(4);
          // ---- packed P^T / dS^T over the scores just read (A operands of the dV / dK products)
          tmem_st16(tST, pp);
          tmem_st16(tDP, dd);
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar.written[team]);
          // ---- a bias that only this row uses (N = 1): d_pair_bias[b, h, i, j] = dS[i, j], no sum over rows; lanes hold
          // consecutive keys j, so every store instruction writes 64 contiguous bytes
          if (p.dbias_direct && j < p.L) {
            const int i0 = it * kT + team * kHalf + ch * 32;
            T* dst = static_cast<T*>(p.dbias_direct) + (((int64_t)b * p.H + h) * p.L + i0) * p.L + j;
#pragma unroll
            for (int c = 0; c < 16; ++c) {
              if (i0 + 2 * c < p.L) *reinterpret_cast<unsigned short*>(dst) = (unsigned short)(dd[c] & 0xffffu);
              if (i0 + 2 * c + 1 < p.L) *reinterpret_cast<unsigned short*>(dst + p.L) = (unsigned short)(dd[c] >> 16);
              dst += 2 * (int64_t)p.L;
            }
          }
          // ---- dS^T also to the shared-memory tile of this block (A operand of the dQ product), once the dQ
          // product that read this buffer two blocks ago is complete
          if (g >= 2) wait_or_flag(&bar.dq_done[g & 1], ((g >> 1) - 1) & 1, abort_flag);
          tr(5);
          {
            uint8_t* atom = sDS + (g & 1) * 2 * kAtomB + team * kAtomB;
#pragma unroll
            for (int c = 0; c < 4; ++c)
              *reinterpret_cast<uint4*>(atom + swz_offset(r, ch * 4 + c, 128)) = make_uint4(dd[c * 4], dd[c * 4 + 1], dd[c * 4 + 2], dd[c * 4 + 3]);
          }
          fence_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar.ds_written[g & 1]);
          tr(6);
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kMainHelperRegs));
    // The helper roles are run by whole warps (one elected lane issues: see mma_ss_el); every exit decision is a warp vote.
    auto dead = [&] { return __any_sync(0xffffffffu, *abort_flag) != 0; };
    constexpr uint32_t hi64 = desc_hi(512, kSw64), hi128 = desc_hi(1024, kSw128);
    constexpr uint32_t kTile16 = kTileB / 16, kAtom16 = kAtomB / 16;      // descriptor address units
    constexpr uint32_t hi32 = desc_hi(256, kSw32), kStage16 = kStageB / 16, kX16 = kXTileB / 16;
    // inside a stage: the NH halves of the first operand (K or Q), the NH halves of the second (V or dO), the term tile
    constexpr uint32_t kOp2 = NH * kTile16, kTerm16 = 2 * NH * kTile16;
    const uint32_t kv_base = desc_lo(smem_u32(sKV), 16), qd_base = desc_lo(smem_u32(sQD), 16);
    if (warp == kComputeWarps) {
      // ========================================================================== dV / dK issuer: per half block
      //   dV_j += P^T dO_i,  dK_j += dS^T Q_i   (A = packed P^T / dS^T in TMEM, B = the dO / Q rows of the half, MN-major;
      //   one group of four products per head half, into that half's 32 accumulator columns)
      const uint32_t id_kv = idesc_f16(128, 32, p.fmt, 0, 1);
      const uint32_t n_set = dbuf ? 2 : 1;
      MF_TRACE_DECL(tr, 2, blockIdx.x == 0 && lane == 0);
      uint32_t g = 0, kv = 0, qslot = 0;
      Item at(blockIdx.x, p);
      for (int item = blockIdx.x; item < p.n_items; item += gridDim.x, at.step(p)) {
        for (int jt = at.jt0(p), jt1 = at.jt1(p); jt < jt1; ++jt, ++kv) {
          // the accumulators have been read out since their last key tile (the one before, or with two sets the one before that)
          if (kv >= n_set) wait_or_flag(&bar.kv_drained[(kv - n_set) & 1], ((kv - n_set) >> 1) & 1, abort_flag);
          const uint32_t tdk = tKV + (kv & 1) * kv_set, tdv = tdk + 32 * NH;
          for (int it = 0; it < nt && !dead(); ++it, ++g) {
            const uint32_t q_lo = qd_base + qslot * kStage16, do_lo = q_lo + kOp2;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              tr(20);
              wait_or_flag(&bar.written[half], g & 1, abort_flag);
              tc_fence_after();
              tr(21);
              const uint32_t tPt = tm0 + half * 128, tDSt = tPt + 64;
              const bool first = it == 0 && half == 0;
#pragma unroll
              for (int hh = 0; hh < NH; ++hh) {
                const uint32_t b_do = do_lo + hh * kTile16 + half * 256, b_q = q_lo + hh * kTile16 + half * 256;
                mma_ts_el(tdv + hh * 32, tPt, b_do, hi64, id_kv, !first);
                mma_ts_el(tdv + hh * 32, tPt + 8, b_do + 64, hi64, id_kv, true);
                mma_ts_el(tdv + hh * 32, tPt + 32, b_do + 128, hi64, id_kv, true);
                mma_ts_el(tdv + hh * 32, tPt + 40, b_do + 192, hi64, id_kv, true);
                mma_ts_el(tdk + hh * 32, tDSt, b_q, hi64, id_kv, !first);
                mma_ts_el(tdk + hh * 32, tDSt + 8, b_q + 64, hi64, id_kv, true);
                mma_ts_el(tdk + hh * 32, tDSt + 32, b_q + 128, hi64, id_kv, true);
                mma_ts_el(tdk + hh * 32, tDSt + 40, b_q + 192, hi64, id_kv, true);
              }
              tc_commit_el(&bar.buf_free[half]);
              tr(22);
            }
            tc_commit_el(&bar.qd_empty[qslot]);
            if (it == nt - 1) tc_commit_el(&bar.kv_done[kv & 1]);
            if (++qslot == NQ) qslot = 0;
          }
        }
      }
    } else if (warp >= kComputeWarps + 4) {
      // ========================================================================== write-out warps: accumulators to global memory
      // The compute warps did this beside their blocks: a fifth of their time, with the wait for the last products at each
      // item's end (forward + backward [1, 384, 384, 4, 32] 359 us, 338 now; at 768 2577 and 2508).
      const int r = (warp & 3) * 32 + lane;             // TMEM lane: key row (dK, dV) or query row (dQ) inside the tile
      const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
      MF_TRACE_DECL(tr, 4, blockIdx.x == 0 && warp == kComputeWarps + 4 && lane == 0);
      uint32_t g = 0, kv = 0;
      int item_no = 0;
      Item at(blockIdx.x, p);
      for (int item = blockIdx.x; item < p.n_items; item += gridDim.x, ++item_no, at.step(p)) {
        // rows of a dQ accumulator added, scaled, to the fp32 dQ rows in global memory
        auto add_dq = [&](uint32_t tacc, int it2, int hh) {
          uint32_t o32[32];
          tmem_ld32(tacc + hh * 32 + lane_addr, o32);
          tmem_ld_wait();
          const int i = it2 * kT + r;
          if (i < p.L && !*abort_flag) {
            float* arow = p.dq_acc + (((int64_t)at.bn(p) * p.L + i) * p.H + at.h) * p.D + hh * 32;
#pragma unroll
            for (int d4 = 0; d4 < 8; ++d4)
              if (hh * 32 + d4 * 4 < p.D)
                asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(arow + d4 * 4),
                             "f"(__uint_as_float(o32[d4 * 4]) * p.scale), "f"(__uint_as_float(o32[d4 * 4 + 1]) * p.scale),
                             "f"(__uint_as_float(o32[d4 * 4 + 2]) * p.scale), "f"(__uint_as_float(o32[d4 * 4 + 3]) * p.scale) : "memory");
          }
        };
        for (int jt = at.jt0(p), jt1 = at.jt1(p); jt < jt1; ++jt, ++kv) {
          for (int it = 0; DQS && it < nt; ++it, ++g) {               // streamed dQ: the product of every block
            wait_or_flag(&bar.dq_done[g & 1], (g >> 1) & 1, abort_flag);
            tc_fence_after();
#pragma unroll 1
            for (int hh = 0; hh < NH; ++hh) add_dq(tDQ + (g & 1) * 32 * NH, it, hh);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar.dq_drained[g & 1]);
          }
          // dK_j (scaled) and dV_j
          wait_or_flag(&bar.kv_done[kv & 1], (kv >> 1) & 1, abort_flag);
          tc_fence_after();
          const int j = jt * kT + r;
          const int64_t row = p.gs.at(at.b, at.n, j) + at.h * p.D;
#pragma unroll 1
          for (int u = 0; u < 2 * NH; ++u) {            // (dK or dV, head half)
            const int hh = u & (NH - 1);
            const bool is_dk = u < NH;
            store_rows(tKV + (kv & 1) * kv_set + u * 32 + lane_addr, is_dk ? p.scale : 1.f, static_cast<T*>(is_dk ? p.dk : p.dv) + row + hh * 32,
                       p.gs.l, j, *abort_flag ? 0 : p.L, p.D - hh * 32);
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar.kv_drained[kv & 1]);
        }
        if constexpr (!DQS) {                           // every query tile's dQ
          wait_or_flag(&bar.item_dq, item_no & 1, abort_flag);
          tc_fence_after();
#pragma unroll 1
          for (int u = 0; u < nt * NH; ++u) {           // (query tile, head half)
            const int it = NH == 1 ? u : u >> 1, hh = u & (NH - 1), i = it * kT + r;
            if (p.ksplit > 1) add_dq(tDQ + it * 32 * NH, it, hh);
            else
              store_rows(tDQ + u * 32 + lane_addr, p.scale, static_cast<T*>(p.dq) + p.gs.at(at.b, at.n, i) + at.h * p.D + hh * 32, p.gs.l, i,
                         *abort_flag ? 0 : p.L, p.D - hh * 32);
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar.item_done[item_no & 1]);
        }
      }
    } else if (warp == kComputeWarps + 3) {
      // ========================================================================== dQ issuer: per block
      //   dQ_i += dS K_j   (A = the dS^T tile in shared memory read MN-major: M = queries; B = K_j, MN-major)
      const uint32_t id_q = idesc_f16(128, 32, p.fmt, 1, 1);
      const uint32_t ds_base = desc_lo(smem_u32(sDS), kAtomB);
      uint32_t g = 0, kv = 0;
      int item_no = 0;
      Item at(blockIdx.x, p);
      for (int item = blockIdx.x; item < p.n_items; item += gridDim.x, ++item_no, at.step(p)) {
        const int jt0 = at.jt0(p), jt1 = at.jt1(p);
        // the on-chip dQ accumulators of the previous item must have been read out before they start afresh
        if (!DQS && item_no > 0) wait_or_flag(&bar.item_done[(item_no - 1) & 1], ((item_no - 1) >> 1) & 1, abort_flag);
        for (int jt = jt0; jt < jt1; ++jt, ++kv) {
          const uint32_t k_lo = kv_base + (kv % NKV) * kStage16;
          for (int it = 0; it < nt && !dead(); ++it, ++g) {
            wait_or_flag(&bar.ds_written[g & 1], (g >> 1) & 1, abort_flag);
            if constexpr (DQS) { if (g >= 2) wait_or_flag(&bar.dq_drained[g & 1], ((g >> 1) - 1) & 1, abort_flag); }
            tc_fence_after();
            const uint32_t a_lo = ds_base + (g & 1) * 2 * kAtom16;
            const uint32_t tacc = tDQ + (DQS ? (g & 1) : it) * 32 * NH;
#pragma unroll
            for (int hh = 0; hh < NH; ++hh) {          // one group of eight products per head half
              const uint32_t kh = k_lo + hh * kTile16;
              mma_ss_el(tacc + hh * 32, a_lo, hi128, kh, hi64, id_q, DQS ? false : jt > jt0);
#pragma unroll
              for (int ks = 1; ks < 8; ++ks) mma_ss_el(tacc + hh * 32, a_lo + ks * (2048 / 16), hi128, kh + ks * 64, hi64, id_q, true);
            }
            if (!DQS && jt == jt1 - 1 && it == nt - 1) tc_commit_el(&bar.item_dq);
            tc_commit_el(&bar.dq_done[g & 1]);
            if (it == nt - 1) tc_commit_el(&bar.kv_empty[kv % NKV]);
          }
        }
      }
    } else if (warp == kComputeWarps + 2) {
      // ========================================================================== score issuer: per half block
      //   S''^T = K_j Q_i^T + alpha * bias^T,  dP^T = V_j dO_i^T
      const uint32_t id_s = idesc_f16(128, kHalf, p.fmt, 0, 0);
      // The bias atom of a half block is the A operand [128 keys x 64 queries] of four K = 16 products: two pieces
      // [64 queries x 64 keys] of the bias as it is, read MN-major (keys contiguous).
      const uint32_t id_b = idesc_f16(128, 16, p.bfmt, 1, 0);
      const uint32_t id_x = idesc_f16(128, kHalf, 1u, 0, 0);        // the rank-one term tiles are bf16 whatever q/k/v are
      const uint32_t xc_lo = desc_lo(smem_u32(sXC), 16);
      const uint32_t bt_base = desc_lo(smem_u32(sBT), 8192);
      constexpr uint32_t bstep = 2048 / 16;                        // 16 queries further: 16 rows of 128 bytes
      const uint32_t i_lo0 = desc_lo(smem_u32(sI), 16), i_lo1 = i_lo0 + 1024 / 16;
      const bool two_terms = p.n_alpha > 1;
      MF_TRACE_DECL(tr, 3, blockIdx.x == 0 && lane == 0);
      uint32_t g = 0, kv = 0, bslot = 0, buse = 0, qslot = 0, quse = 0;
      Item at(blockIdx.x, p);
      for (int item = blockIdx.x; item < p.n_items; item += gridDim.x, at.step(p)) {
        for (int jt = at.jt0(p), jt1 = at.jt1(p); jt < jt1; ++jt, ++kv) {
          wait_or_flag(&bar.kv_full[kv % NKV], (kv / NKV) & 1, abort_flag);
          const uint32_t k_lo = kv_base + (kv % NKV) * kStage16, v_lo = k_lo + kOp2, xk_lo = k_lo + kTerm16;
          for (int it = 0; it < nt && !dead(); ++it, ++g) {
            wait_or_flag(&bar.qd_full[qslot], quse & 1, abort_flag);
            const uint32_t q_blk = qd_base + qslot * kStage16;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              tr(30);
              wait_or_flag(&bar.bt_full[bslot], buse & 1, abort_flag);
              if (g >= 1) wait_or_flag(&bar.buf_free[half], (g - 1) & 1, abort_flag);
              tc_fence_after();
              tr(31);
              const uint32_t tS = tm0 + half * 128, tD = tS + 64;
              const uint32_t q_lo = q_blk + half * 256, g_lo = q_lo + kOp2, xq_lo = q_blk + kTerm16 + half * (kX16 / 2);
#pragma unroll
              for (int hh = 0; hh < NH; ++hh) {
                mma_ss_el(tS, k_lo + hh * kTile16, hi64, q_lo + hh * kTile16, hi64, id_s, hh > 0);
                mma_ss_el(tS, k_lo + hh * kTile16 + 2, hi64, q_lo + hh * kTile16 + 2, hi64, id_s, true);
              }
              mma_ss_el(tS, xk_lo, hi32, xq_lo, hi32, id_x, true);               // + mask_j - lse_i
              const uint32_t a_lo = bt_base + bslot * kAtom16;
#pragma unroll
              for (int c = 0; c < 4; ++c) mma_ss_el(tS + c * 16, a_lo + c * bstep, hi128, i_lo0, hi64, id_b, true);
              if (two_terms) {
#pragma unroll
                for (int c = 0; c < 4; ++c) mma_ss_el(tS + c * 16, a_lo + c * bstep, hi128, i_lo1, hi64, id_b, true);
              }
#pragma unroll
              for (int hh = 0; hh < NH; ++hh) {
                mma_ss_el(tD, v_lo + hh * kTile16, hi64, g_lo + hh * kTile16, hi64, id_s, hh > 0);
                mma_ss_el(tD, v_lo + hh * kTile16 + 2, hi64, g_lo + hh * kTile16 + 2, hi64, id_s, true);
              }
              mma_ss_el(tD, xc_lo, hi32, xq_lo, hi32, id_x, true);               // - delta_i
              tc_commit_el(&bar.sd_ready[half]);
              tc_commit_el(&bar.bt_empty[bslot]);
              if (++bslot == NB) { bslot = 0; ++buse; }
              tr(32);
            }
            if (++qslot == NQ) { qslot = 0; ++quse; }
          }
        }
      }
    } else if (warp == kComputeWarps + 1) {
      // ========================================================================== TMA producer, in order of need
      uint32_t g = 0, kv = 0, bslot = 0, buse = 0, nbt = 0, qslot = 0, quse = 0;
      Item at(blockIdx.x, p);
      for (int item = blockIdx.x; item < p.n_items && !dead(); item += gridDim.x, at.step(p)) {
        const int h = at.h, n = at.n, b = at.b, bn = at.bn(p), bnh = at.bnh(p);
        for (int jt = at.jt0(p), jt1 = at.jt1(p); jt < jt1 && !dead(); ++jt, ++kv) {
          if (kv >= (uint32_t)NKV) wait_or_flag(&bar.kv_empty[kv % NKV], ((kv / NKV) - 1) & 1, abort_flag);
          if (dead()) break;
          if (elect_one()) {
            uint64_t* fb = &bar.kv_full[kv % NKV];
            uint8_t* st = sKV + (kv % NKV) * kStageB;
            mbar_expect_tx(fb, kStageB);
#pragma unroll
            for (int hh = 0; hh < NH; ++hh) {
              tma_load_5d(st + hh * kTileB, &mk, fb, hh * kDP, h, jt * kT, n, b);
              tma_load_5d(st + (NH + hh) * kTileB, &mv, fb, hh * kDP, h, jt * kT, n, b);
            }
            bulk_load_1d(st + 2 * NH * kTileB, p.xk + ((int64_t)bn * nt + jt) * kXTileB, kXTileB, fb);
          }
          for (int it = 0; it < nt; ++it, ++g) {
            if (quse >= 1) wait_or_flag(&bar.qd_empty[qslot], (quse - 1) & 1, abort_flag);
            if (dead()) break;
            if (elect_one()) {
              uint64_t* fb = &bar.qd_full[qslot];
              uint8_t* st = sQD + qslot * kStageB;
              mbar_expect_tx(fb, kStageB);
#pragma unroll
              for (int hh = 0; hh < NH; ++hh) {
                tma_load_5d(st + hh * kTileB, &mq, fb, hh * kDP, h, it * kT, n, b);
                tma_load_5d(st + (NH + hh) * kTileB, &mg, fb, hh * kDP, h, it * kT, n, b);
              }
              bulk_load_1d(st + 2 * NH * kTileB, p.xq + ((int64_t)bnh * nt + it) * kXTileB, kXTileB, fb);
            }
            if (++qslot == NQ) { qslot = 0; ++quse; }
            for (int half = 0; half < 2; ++half) {
              if (buse >= 1) wait_or_flag(&bar.bt_empty[bslot], (buse - 1) & 1, abort_flag);
              if (dead()) break;
              if (elect_one()) {
                mbar_expect_tx(&bar.bt_full[bslot], kAtomB);
                // [64 queries x 64 keys] pieces of the bias: keys 0-63 | 64-127 of the tile
                tma_load_4d(sBT + bslot * kAtomB, &mbt, &bar.bt_full[bslot], jt * kT, it * kT + half * kHalf, h, b * p.bias_b_mul);
                tma_load_4d(sBT + bslot * kAtomB + 8192, &mbt, &bar.bt_full[bslot], jt * kT + 64, it * kT + half * kHalf, h, b * p.bias_b_mul);
              }
              ++nbt;
              if (++bslot == NB) { bslot = 0; ++buse; }
            }
          }
        }
      }
      if (dead() && lane == 0) {
        // the copies already requested must land before the CTA's shared memory is given back (bounded)
        for (uint32_t back = 0; back < (uint32_t)NKV && back < kv; ++back) { const uint32_t c = kv - 1 - back; mbar_wait(&bar.kv_full[c % NKV], (c / NKV) & 1); }
        for (uint32_t back = 0; back < (uint32_t)NQ && back < g; ++back) { const uint32_t c = g - 1 - back; mbar_wait(&bar.qd_full[c % NQ], (c / NQ) & 1); }
        for (uint32_t back = 0; back < (uint32_t)NB && back < nbt; ++back) { const uint32_t c = nbt - 1 - back; mbar_wait(&bar.bt_full[c % NB], (c / NB) & 1); }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && abort_s) *reinterpret_cast<volatile int*>(p.status) = 1;
  if (warp == 0) tmem_dealloc(tmem_base_s, 512);
}

// ------------------------------------------------------------------------------------------------ dBias
struct DbP {
  int B, N, L, H, D;
  int n_t, lpad, nsplit, n_units;
  float c1;
  uint32_t fmt, bfmt;
  int n_alpha; float alpha[2];
  int bias_b_mul;
  const uint8_t* xq; const uint8_t* xk;      // rank-one term tiles (evo_extras_ws_kernel)
  float* part;            // fp32 [nsplit][B][H][L][L] partial sums
  void* out16;            // with a single row range and a 16-bit d_bias: the result itself, [B][H][L][L] in the q/k/v type
  int* status;
};

struct DbBars {                              // every role waits for each phase of a barrier in turn (see tc.cuh)
  uint64_t op_full[3], op_empty[3];          // Q, dO, K, V, XQ, XK of one row n
  uint64_t bt_full, bt_free;                 // the unit's two bias atoms
  uint64_t sd_ready[2], loaded[2];
};

template <typename T, typename TB, int NH>
__global__ void __launch_bounds__(kThreads, 1)
evo_dbias_ws_kernel(const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mk,
                    const __grid_constant__ CUtensorMap mv, const __grid_constant__ CUtensorMap mg,
                    const __grid_constant__ CUtensorMap mbt, const DbP p MF_TRACE_PARAM) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sBT = smem;                          // two bias atoms (queries 0-63 | 64-127 of the tile)
  constexpr int kDbStageB = Geo<NH>::kDbStageB, NS = Geo<NH>::NS;
  uint8_t* sOP = sBT + 2 * kAtomB;              // [NS stages][Q halves, dO halves, K halves, V halves, XQ, XK]
  uint8_t* sI = sOP + NS * kDbStageB;
  uint8_t* sXC = sI + 2048;                     // constant tile of the -delta term

  __shared__ DbBars bar;
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;

  // With one head half uniform operands only make the compute warps spill more (24 bytes stored, 16 without): [1, 384, 384, 4, 32] 73.2 us
  // for this kernel, 71.9 without, at 512 183.5 and 180.0 (at 96 8.1 and 8.3); with two halves [4, 1, 384, 32, 64] 34.2 and 36.1.
  constexpr bool kUniform = NH > 1;
  const int tid = threadIdx.x, warp = kUniform ? uniform(tid >> 5) : tid >> 5, lane = tid & 31;
  if (tid == 0) {
    abort_s = 0;
    for (int i = 0; i < 3; ++i) {
      mbar_init(&bar.op_full[i], 1); mbar_init(&bar.op_empty[i], 2);      // two issuers commit
    }
    mbar_init(&bar.bt_full, 1); mbar_init(&bar.bt_free, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(&bar.sd_ready[i], 2); mbar_init(&bar.loaded[i], kComputeWarps); }
    mbar_fence_init();
    prefetch_tmap(&mq); prefetch_tmap(&mk); prefetch_tmap(&mv); prefetch_tmap(&mg); prefetch_tmap(&mbt);
  }
  write_alpha_identity<TB>(sI, p.alpha[0], tid, kThreads);
  write_alpha_identity<TB>(sI + 1024, p.alpha[1], tid, kThreads);
  write_xc_tile(sXC, tid, kThreads);
  fence_async_smem();
  if (warp == 0) { tmem_alloc(&tmem_base_s, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  volatile int* abort_flag = &abort_s;
  const uint32_t tm0 = kUniform ? uniform(tmem_base_s) : tmem_base_s;
  const int nt = p.n_t;
  // unit = ((b * H + h) * nt + jt) * nt + it, split `sp` of the rows
  struct Unit { int b, h, jt, it, n0, n1; };
  auto unit_of = [&](int u) {
    Unit x;
    const int sp = u % p.nsplit; int c = u / p.nsplit;
    x.it = c % nt; c /= nt; x.jt = c % nt; c /= nt; x.h = c % p.H; x.b = c / p.H;
    x.n0 = (int)((int64_t)sp * p.N / p.nsplit); x.n1 = (int)((int64_t)(sp + 1) * p.N / p.nsplit);
    return x;
  };

  if (warp < kComputeWarps) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kComputeRegs));
    const int w = warp >> 2;                          // query quarter (32 columns) handled by this thread
    const int r = (warp & 3) * 32 + lane;             // TMEM lane = key row inside the tile
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    uint32_t g = 0;                                   // rows processed by this CTA (TMEM buffer g & 1)
    const float2 c1c1 = make_float2(p.c1, p.c1);
    MF_TRACE_DECL(tr, 0, blockIdx.x == 0 && tid == 0);
    for (int u = blockIdx.x; u < p.n_units; u += gridDim.x) {
      const Unit x = unit_of(u);
      const int j = x.jt * kT + r;
      float2 acc[16];
#pragma unroll
      for (int c = 0; c < 16; ++c) acc[c] = make_float2(0.f, 0.f);
      for (int n = x.n0; n < x.n1; ++n, ++g) {
        const uint32_t tST = tm0 + (g & 1) * 256 + w * 32 + lane_addr, tDP = tST + 128;
        tr(1);
        wait_or_flag(&bar.sd_ready[g & 1], (g >> 1) & 1, abort_flag);
        tc_fence_after();
        tr(2);
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {          // 16 query columns at a time keeps the live registers down
          uint32_t sr[16], dr[16];
          tmem_ld16(tST + hf * 16, sr);
          tmem_ld16(tDP + hf * 16, dr);
          tmem_ld_wait();
          if (hf == 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar.loaded[g & 1]);
            tr(3);
          }
          // mask, lse and delta are already inside the accumulators: P = 2^(c1 S''), dS = P dP''
#pragma unroll
          for (int c2 = 0; c2 < 8; ++c2) {
            const float2 xx = mul2(make_float2(__uint_as_float(sr[c2 * 2]), __uint_as_float(sr[c2 * 2 + 1])), c1c1);
            const float2 pr = make_float2(ex2f(xx.x), ex2f(xx.y));
            acc[hf * 8 + c2] = fma2(pr, make_float2(__uint_as_float(dr[c2 * 2]), __uint_as_float(dr[c2 * 2 + 1])), acc[hf * 8 + c2]);
          }
        }
        tr(4);
      }
      // the unit's partial sum: part[sp][b][h][i][j], lanes = consecutive keys
      if (j < p.L && !*abort_flag) {
        const int sp = u % p.nsplit;
        const int64_t at = ((((int64_t)sp * p.B + x.b) * p.H + x.h) * p.L) * (int64_t)p.L + j;
        const int i0 = x.it * kT + w * 32;
        if (p.out16) {
          T* dst = static_cast<T*>(p.out16) + at;
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            if (i0 + 2 * c < p.L) dst[(int64_t)(i0 + 2 * c) * p.L] = from_f<T>(acc[c].x);
            if (i0 + 2 * c + 1 < p.L) dst[(int64_t)(i0 + 2 * c + 1) * p.L] = from_f<T>(acc[c].y);
          }
        } else {
          float* dst = p.part + at;
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            if (i0 + 2 * c < p.L) dst[(int64_t)(i0 + 2 * c) * p.L] = acc[c].x;
            if (i0 + 2 * c + 1 < p.L) dst[(int64_t)(i0 + 2 * c + 1) * p.L] = acc[c].y;
          }
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kHelperRegs));
    // The helper roles are run by whole warps (one elected lane issues: see mma_ss_el); every exit decision is a warp vote.
    auto dead = [&] { return __any_sync(0xffffffffu, *abort_flag) != 0; };
    constexpr uint32_t hi64 = desc_hi(512, kSw64), hi128 = desc_hi(1024, kSw128);
    constexpr uint32_t kTile16 = kTileB / 16, kAtom16 = kAtomB / 16;
    constexpr uint32_t hi32 = desc_hi(256, kSw32), kStage16 = kDbStageB / 16;
    const uint32_t op_base = desc_lo(smem_u32(sOP), 16);
    const uint32_t id_s = idesc_f16(128, 128, p.fmt, 0, 0);
    const uint32_t id_x = idesc_f16(128, 128, 1u, 0, 0);          // the rank-one term tiles are bf16 whatever q/k/v are
    if (warp == kComputeWarps) {
      // ========================================================================== score issuer: S''^T = K Q^T + alpha * bias^T
      const uint32_t id_b = idesc_f16(128, 16, p.bfmt, 1, 0);      // see the main kernel's score issuer
      const uint32_t bt_lo = desc_lo(smem_u32(sBT), 8192);
      constexpr uint32_t bstep = 2048 / 16;
      const uint32_t i_lo0 = desc_lo(smem_u32(sI), 16), i_lo1 = i_lo0 + 1024 / 16;
      const bool two_terms = p.n_alpha > 1;
      MF_TRACE_DECL(tr, 2, blockIdx.x == 0 && lane == 0);
      uint32_t g = 0, un = 0, stage = 0, suse = 0;
      for (int u = blockIdx.x; u < p.n_units && !dead(); u += gridDim.x, ++un) {
        const Unit x = unit_of(u);
        wait_or_flag(&bar.bt_full, un & 1, abort_flag);
        for (int n = x.n0; n < x.n1 && !dead(); ++n, ++g) {
          tr(20);
          wait_or_flag(&bar.op_full[stage], suse & 1, abort_flag);
          if (g >= 2) wait_or_flag(&bar.loaded[g & 1], ((g >> 1) - 1) & 1, abort_flag);
          tc_fence_after();
          tr(21);
          const uint32_t q_lo = op_base + stage * kStage16, k_lo = q_lo + 2 * NH * kTile16;
          const uint32_t xq_lo = q_lo + 4 * NH * kTile16, xk_lo = xq_lo + kXTileB / 16;
          const uint32_t tST = tm0 + (g & 1) * 256;
#pragma unroll
          for (int hh = 0; hh < NH; ++hh) {
            mma_ss_el(tST, k_lo + hh * kTile16, hi64, q_lo + hh * kTile16, hi64, id_s, hh > 0);
            mma_ss_el(tST, k_lo + hh * kTile16 + 2, hi64, q_lo + hh * kTile16 + 2, hi64, id_s, true);
          }
          mma_ss_el(tST, xk_lo, hi32, xq_lo, hi32, id_x, true);                 // + mask_j - lse_i
#pragma unroll
          for (int c = 0; c < 8; ++c) mma_ss_el(tST + c * 16, bt_lo + (c >> 2) * kAtom16 + (c & 3) * bstep, hi128, i_lo0, hi64, id_b, true);
          if (two_terms) {
#pragma unroll
            for (int c = 0; c < 8; ++c) mma_ss_el(tST + c * 16, bt_lo + (c >> 2) * kAtom16 + (c & 3) * bstep, hi128, i_lo1, hi64, id_b, true);
          }
          tc_commit_el(&bar.sd_ready[g & 1]);
          tc_commit_el(&bar.op_empty[stage]);
          if (++stage == NS) { stage = 0; ++suse; }
          tr(22);
        }
        tc_commit_el(&bar.bt_free);       // every product that reads this unit's bias atoms is complete
      }
    } else if (warp == kComputeWarps + 2) {
      // ========================================================================== dP issuer: dP^T = V dO^T
      uint32_t g = 0, stage = 0, suse = 0;
      for (int u = blockIdx.x; u < p.n_units && !dead(); u += gridDim.x) {
        const Unit x = unit_of(u);
        for (int n = x.n0; n < x.n1 && !dead(); ++n, ++g) {
          wait_or_flag(&bar.op_full[stage], suse & 1, abort_flag);
          if (g >= 2) wait_or_flag(&bar.loaded[g & 1], ((g >> 1) - 1) & 1, abort_flag);
          tc_fence_after();
          const uint32_t g_lo = op_base + stage * kStage16 + NH * kTile16, v_lo = g_lo + 2 * NH * kTile16;
          const uint32_t xq_lo = op_base + stage * kStage16 + 4 * NH * kTile16;
          const uint32_t tDP = tm0 + (g & 1) * 256 + 128;
#pragma unroll
          for (int hh = 0; hh < NH; ++hh) {
            mma_ss_el(tDP, v_lo + hh * kTile16, hi64, g_lo + hh * kTile16, hi64, id_s, hh > 0);
            mma_ss_el(tDP, v_lo + hh * kTile16 + 2, hi64, g_lo + hh * kTile16 + 2, hi64, id_s, true);
          }
          mma_ss_el(tDP, desc_lo(smem_u32(sXC), 16), hi32, xq_lo, hi32, id_x, true);      // - delta_i
          tc_commit_el(&bar.sd_ready[g & 1]);
          tc_commit_el(&bar.op_empty[stage]);
          if (++stage == NS) { stage = 0; ++suse; }
        }
      }
    } else if (warp == kComputeWarps + 1) {
      // ========================================================================== TMA producer
      uint32_t g = 0, un = 0, stage = 0, suse = 0;
      for (int u = blockIdx.x; u < p.n_units && !dead(); u += gridDim.x, ++un) {
        const Unit x = unit_of(u);
        if (un >= 1) wait_or_flag(&bar.bt_free, (un - 1) & 1, abort_flag);
        if (dead()) break;
        if (elect_one()) {
          mbar_expect_tx(&bar.bt_full, 2 * kAtomB);
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4)       // (query half, key half) pieces of [64 x 64]
            tma_load_4d(sBT + (q4 >> 1) * kAtomB + (q4 & 1) * 8192, &mbt, &bar.bt_full, x.jt * kT + (q4 & 1) * 64,
                        x.it * kT + (q4 >> 1) * kHalf, x.h, x.b * p.bias_b_mul);
        }
        for (int n = x.n0; n < x.n1; ++n, ++g) {
          if (suse >= 1) wait_or_flag(&bar.op_empty[stage], (suse - 1) & 1, abort_flag);
          if (dead()) break;
          if (elect_one()) {
            uint64_t* fb = &bar.op_full[stage];
            uint8_t* st = sOP + stage * kDbStageB;
            mbar_expect_tx(fb, kDbStageB);
#pragma unroll
            for (int hh = 0; hh < NH; ++hh) {
              tma_load_5d(st + hh * kTileB, &mq, fb, hh * kDP, x.h, x.it * kT, n, x.b);
              tma_load_5d(st + (NH + hh) * kTileB, &mg, fb, hh * kDP, x.h, x.it * kT, n, x.b);
              tma_load_5d(st + (2 * NH + hh) * kTileB, &mk, fb, hh * kDP, x.h, x.jt * kT, n, x.b);
              tma_load_5d(st + (3 * NH + hh) * kTileB, &mv, fb, hh * kDP, x.h, x.jt * kT, n, x.b);
            }
            const int64_t bn = (int64_t)x.b * p.N + n;
            bulk_load_1d(st + 4 * NH * kTileB, p.xq + ((bn * p.H + x.h) * nt + x.it) * kXTileB, kXTileB, fb);
            bulk_load_1d(st + 4 * NH * kTileB + kXTileB, p.xk + (bn * nt + x.jt) * kXTileB, kXTileB, fb);
          }
          if (++stage == NS) { stage = 0; ++suse; }
        }
      }
      if (dead() && lane == 0) {
        for (uint32_t back = 0; back < (uint32_t)NS && back < g; ++back) { const uint32_t c = g - 1 - back; mbar_wait(&bar.op_full[c % NS], (c / NS) & 1); }
        if (un > 0) mbar_wait(&bar.bt_full, (un - 1) & 1);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && abort_s) *reinterpret_cast<volatile int*>(p.status) = 1;
  if (warp == 0) tmem_dealloc(tmem_base_s, 512);
}

// d_bias[b][h][i][j] = sum over the row ranges, in order, cast to the output type
template <typename TO>
__global__ void dbias_finish_kernel(const float* __restrict__ part, TO* __restrict__ out, int64_t n, int nsplit) {
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (i >= n) return;
  if (i + 4 <= n && (n & 3) == 0) {            // four entries per thread; every range starts on a 16-byte boundary
    float4 s = *reinterpret_cast<const float4*>(part + i);
    for (int k = 1; k < nsplit; ++k) {
      const float4 t = *reinterpret_cast<const float4*>(part + (int64_t)k * n + i);
      s.x += t.x; s.y += t.y; s.z += t.z; s.w += t.w;
    }
    out[i] = from_f<TO>(s.x); out[i + 1] = from_f<TO>(s.y); out[i + 2] = from_f<TO>(s.z); out[i + 3] = from_f<TO>(s.w);
    return;
  }
  for (int64_t e = i; e < n && e < i + 4; ++e) {
    float s = part[e];
    for (int k = 1; k < nsplit; ++k) s += part[(int64_t)k * n + e];
    out[e] = from_f<TO>(s);
  }
}

// the fp32 accumulator of dQ ([B, N, L, H, D], D a multiple of 8) to its 16-bit place, eight elements per thread
template <typename T>
__global__ void __launch_bounds__(256) cast_dq_kernel(const float* __restrict__ src, T* __restrict__ dst, TokenStrides gs, int64_t n8, int HD, int L, int N) {
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= n8) return;
  const int64_t tok = i * 8 / HD;
  const int e = (int)(i * 8 - tok * HD);
  const int l = (int)(tok % L); const int64_t bn = tok / L;
  const float4 x = reinterpret_cast<const float4*>(src)[2 * i], y = reinterpret_cast<const float4*>(src)[2 * i + 1];
  uint4 v;
  v.x = Pack2<T>::pack(x.x, x.y); v.y = Pack2<T>::pack(x.z, x.w); v.z = Pack2<T>::pack(y.x, y.y); v.w = Pack2<T>::pack(y.z, y.w);
  *reinterpret_cast<uint4*>(dst + gs.at((int)(bn / N), (int)(bn % N), l) + e) = v;
}

// With few (b, n, h) triples (single-representation attention: N = 1) the key tiles of each are spread over several
// CTAs so that the whole GPU works; the partial dQ rows then meet in an fp32 accumulator.
int bwd_ksplit(int64_t bnh, int nt, int sms) {
  if (bnh >= sms || nt < 2) return 1;
  int64_t k = sms / bnh;                 // as many ranges as keep every CTA at one work item
  if (k > nt) k = nt;
  return k < 1 ? 1 : (int)k;
}

struct BwdPlan {
  int nt, lpad, ksplit, dq_stream, dbuf, nsplit;
  bool dq_fp32, part_direct, bias_direct;
  size_t off_flags, off_xq, off_xk, off_part, off_dq, off_bias, total;
};

BwdPlan plan_bwd(const mf_evo_bwd_args& a) {
  BwdPlan pl{};
  const int sms = sm_count();
  pl.nt = (a.L + kT - 1) / kT;
  pl.lpad = pl.nt * kT;
  pl.ksplit = bwd_ksplit((int64_t)a.B * a.N * a.H, pl.nt, sms);
  // dQ accumulators of all query tiles next to one set (up to six tiles) or two sets (up to four) of dK/dV accumulators;
  // longer rows stream dQ
  if (a.D <= kDP) {
    pl.dq_stream = pl.nt > 6;
    pl.dbuf = pl.dq_stream || pl.nt <= 4;
  } else {
    // two head halves: one set of dK|dV accumulators (128 columns) leaves room for two dQ accumulators of 64 columns
    pl.dq_stream = pl.nt > 2;
    pl.dbuf = 0;
  }
  pl.dq_fp32 = pl.ksplit > 1 || pl.dq_stream;
  const int64_t combos = (int64_t)a.B * a.H * pl.nt * pl.nt;
  int64_t ns = sms / combos;
  if (ns < 1) ns = 1;
  if (ns > a.N) ns = a.N;
  pl.nsplit = (int)ns;
  pl.part_direct = pl.nsplit == 1;      // a single range writes d_bias itself, in its own type
  size_t off = 0;
  pl.off_flags = off; off += align_up(sizeof(int) * (size_t)a.B * a.N * a.H, 256);
  pl.off_xq = off; off += (size_t)a.B * a.N * a.H * pl.nt * kXTileB;
  pl.off_xk = off; off += (size_t)a.B * a.N * pl.nt * kXTileB;
  pl.off_part = off; if (!pl.part_direct) off += align_up(sizeof(float) * (size_t)pl.nsplit * a.B * a.H * a.L * a.L, 256);
  pl.off_dq = off; if (pl.dq_fp32) off += align_up(sizeof(float) * (size_t)a.B * a.N * a.L * a.H * a.D, 256);
  pl.bias_direct = bias_tma_ok(a.bias, a.bias_dtype, a.bias_strides, a.B, a.H);
  pl.off_bias = off; if (!pl.bias_direct) off += bias_copy_bytes(a.bias_strides, a.B, a.H, a.L);
  pl.total = off;
  return pl;
}

template <typename T, typename TB, int NH>
int launch_bwd_ws(const mf_evo_bwd_args& a, const mf_evo_layout& lay, cudaStream_t st) {
  const BwdPlan pl = plan_bwd(a);
  CUtensorMap mq, mk, mv, mg, mbt;
  int r;
  const int64_t cs[5] = {lay.d_o[0], lay.d_o[1], lay.d_o[2], a.D, 1};
  if ((r = make_qkv_map(&mq, a.q, a.dtype, a.B, a.N, a.L, a.H, a.D, a.q_strides, kDP, kT))) return r;
  if ((r = make_qkv_map(&mk, a.k, a.dtype, a.B, a.N, a.L, a.H, a.D, a.k_strides, kDP, kT))) return r;
  if ((r = make_qkv_map(&mv, a.v, a.dtype, a.B, a.N, a.L, a.H, a.D, a.v_strides, kDP, kT))) return r;
  if ((r = make_qkv_map(&mg, a.d_o, a.dtype, a.B, a.N, a.L, a.H, a.D, cs, kDP, kT))) return r;
  int* status = status_word();
  MF_REQUIRE(status, MF_ERR_CUDA, "could not allocate the device status word");
  MF_REQUIRE(tc_async_status() == 0, MF_ERR_CUDA, "an earlier tensor-core kernel gave up on a bounded wait; results are invalid");
  char* ws = static_cast<char*>(a.workspace);
  int* flags = reinterpret_cast<int*>(ws + pl.off_flags);
  uint8_t* xq = reinterpret_cast<uint8_t*>(ws + pl.off_xq);
  uint8_t* xk = reinterpret_cast<uint8_t*>(ws + pl.off_xk);
  float* part = !pl.part_direct ? reinterpret_cast<float*>(ws + pl.off_part) : (a.dbias_dtype == MF_F32 ? static_cast<float*>(a.d_bias) : nullptr);
  float* dq_acc = reinterpret_cast<float*>(ws + pl.off_dq);
  // a bias that TMA cannot address is copied in a 16-bit type: the bias dtype when that is one, else the q/k/v dtype
  using TT = typename std::conditional<sizeof(TB) == 2, TB, T>::type;
  const int bt_dtype = sizeof(TB) == 2 ? a.bias_dtype : a.dtype;
  const int lpad = pl.lpad;
  const int bias_b_mul = a.bias_strides[0] == 0 ? 0 : 1;
  {
    const void* bias = a.bias;
    int64_t str[4] = {1, a.bias_strides[2], a.bias_strides[1], a.bias_strides[0]};
    if (!pl.bias_direct) {
      void* copy = ws + pl.off_bias;
      if ((r = copy_bias_rows(a.bias, a.bias_dtype, a.bias_strides, copy, bt_dtype, a.B, a.H, a.L, st))) return r;
      bias = copy;
      str[1] = bias_pitch(a.L); str[2] = str[1] * a.L; str[3] = str[2] * a.H;
    }
    const int64_t dims[4] = {a.L, a.L, a.H, bias_b_mul ? a.B : 1};
    const int box[4] = {64, 64, 1, 1};
    if ((r = make_tiled_map(&mbt, bias, bt_dtype, 4, dims, str, box, 128))) return r;
  }
  {
    const int row_blocks = (int)(((int64_t)lpad * a.H + kXWarps * 32 - 1) / (kXWarps * 32));
    auto kern = a.D <= 32 ? evo_extras_ws_kernel<T, 32> : evo_extras_ws_kernel<T, 64>;
    kern<<<(unsigned)((int64_t)a.B * a.N * row_blocks), kXWarps * 32, 0, st>>>(static_cast<const T*>(a.o), token_strides(lay.o), static_cast<const T*>(a.d_o), token_strides(lay.d_o), a.lse,
                                                                             a.mask, a.mask_strides[0], a.mask_strides[1], a.mask_strides[2], a.mask_dtype,
                                                                             xq, xk, flags, pl.dq_fp32 ? dq_acc : nullptr, row_blocks, a.N, a.L, lpad, a.H, a.D);
  }
  MF_LAUNCHED("evo_extras_ws_kernel");
  const int64_t n_dq = (int64_t)a.B * a.N * a.L * a.H * a.D;

  float alpha[2];
  const int n_alpha = split_alpha(a.D, bt_dtype, alpha, false);
  // With one row per bias (N = 1, single-representation attention) and d_pair_bias in the q/k/v type, dS is the answer:
  // the dQ/dK/dV kernel writes it and the d_pair_bias kernel is not needed.
  const bool dbias_direct = a.N == 1 && a.dbias_dtype == a.dtype;
  // ---- dBias first: a caller that all-reduces it over row shards can start while dQ / dK / dV are computed
  if (!dbias_direct) {
    DbP p{};
    p.B = a.B; p.N = a.N; p.L = a.L; p.H = a.H; p.D = a.D;
    p.n_t = pl.nt; p.lpad = lpad; p.nsplit = pl.nsplit;
    p.n_units = a.B * a.H * pl.nt * pl.nt * pl.nsplit;
    p.c1 = kLog2e / sqrtf((float)a.D);
    p.fmt = a.dtype == MF_BF16 ? 1u : 0u; p.bfmt = bt_dtype == MF_BF16 ? 1u : 0u;
    p.n_alpha = n_alpha; p.alpha[0] = alpha[0]; p.alpha[1] = alpha[1];
    p.bias_b_mul = bias_b_mul;
    p.xq = xq; p.xk = xk;
    p.part = part;
    p.out16 = pl.part_direct && a.dbias_dtype != MF_F32 ? a.d_bias : nullptr;
    p.status = status;
    const size_t smem = Geo<NH>::kDbSmem;
    int grid = sm_count();
    if (grid > p.n_units) grid = p.n_units;
    constexpr auto kern = evo_dbias_ws_kernel<T, TT, NH>;
    if (int e = opt_in_smem<kern>(smem, kLaunchRegs)) return e;
    kern<<<grid, kThreads, smem, st>>>(mq, mk, mv, mg, mbt, p MF_TRACE_ARG);
    MF_LAUNCHED("evo_dbias_ws_kernel");
    if (!pl.part_direct) {
      const int64_t n_out = (int64_t)a.B * a.H * a.L * a.L;
      if (a.dbias_dtype == MF_F32)
        dbias_finish_kernel<float><<<(unsigned)((n_out + 1023) / 1024), 256, 0, st>>>(part, static_cast<float*>(a.d_bias), n_out, pl.nsplit);
      else
        dbias_finish_kernel<T><<<(unsigned)((n_out + 1023) / 1024), 256, 0, st>>>(part, static_cast<T*>(a.d_bias), n_out, pl.nsplit);
      MF_LAUNCHED("dbias_finish_kernel");
    }
  }
  if (a.dbias_ready_event && !dbias_direct) MF_CUDA(cudaEventRecord(static_cast<cudaEvent_t>(a.dbias_ready_event), st));
  // ---- dQ, dK, dV
  {
    BwdWsP p{};
    p.B = a.B; p.N = a.N; p.L = a.L; p.H = a.H; p.D = a.D;
    p.n_t = pl.nt; p.lpad = lpad; p.ksplit = pl.ksplit; p.dq_stream = pl.dq_stream; p.dbuf = pl.dbuf;
    p.n_items = a.B * a.N * a.H * pl.ksplit;
    int grid = sm_count();
    if (grid > p.n_items) grid = p.n_items;
    p.step[0] = grid % pl.ksplit; p.step[1] = grid / pl.ksplit % a.H; p.step[2] = grid / pl.ksplit / a.H % a.N; p.step[3] = grid / pl.ksplit / a.H / a.N;
    p.dq_acc = dq_acc;
    p.scale = 1.0f / sqrtf((float)a.D); p.c1 = kLog2e * p.scale; p.inv_L = 1.0f / a.L;
    p.fmt = a.dtype == MF_BF16 ? 1u : 0u; p.bfmt = bt_dtype == MF_BF16 ? 1u : 0u;
    p.n_alpha = n_alpha; p.alpha[0] = alpha[0]; p.alpha[1] = alpha[1];
    p.bias_b_mul = bias_b_mul;
    p.xq = xq; p.xk = xk; p.flags = flags;
    p.dbias_direct = dbias_direct ? a.d_bias : nullptr;
    p.dq = a.dq; p.dk = a.dk; p.dv = a.dv; p.gs = token_strides(lay.d_qkv);
    p.status = status;
    const size_t smem = Geo<NH>::kMainSmem;
    if (pl.dq_stream) {
      constexpr auto kern = evo_bwd_ws_kernel<T, TT, true, NH>;
      if (int e = opt_in_smem<kern>(smem, kMainLaunchRegs)) return e;
      kern<<<grid, kMainThreads, smem, st>>>(mq, mk, mv, mg, mbt, p MF_TRACE_ARG);
    } else {
      constexpr auto kern = evo_bwd_ws_kernel<T, TT, false, NH>;
      if (int e = opt_in_smem<kern>(smem, kMainLaunchRegs)) return e;
      kern<<<grid, kMainThreads, smem, st>>>(mq, mk, mv, mg, mbt, p MF_TRACE_ARG);
    }
    MF_LAUNCHED("evo_bwd_ws_kernel");
    if (a.dbias_ready_event && dbias_direct) MF_CUDA(cudaEventRecord(static_cast<cudaEvent_t>(a.dbias_ready_event), st));
  }
  if (pl.dq_fp32) {
    const int64_t n8 = n_dq / 8;
    cast_dq_kernel<T><<<(unsigned)((n8 + 255) / 256), 256, 0, st>>>(dq_acc, static_cast<T*>(a.dq), token_strides(lay.d_qkv), n8, a.H * a.D, a.L, a.N);
    MF_LAUNCHED("cast_dq_kernel");
  }
  return MF_OK;
}

}  // namespace

bool evo_bwd_ws_shape_ok(int L, int D) {
  // head sizes up to 64 (two halves of 32 columns); rows of more than six query tiles (two with a head size above 32)
  // stream dQ through an fp32 accumulator in global memory, which has been validated up to 2048 tokens
  return D <= 64 && L <= 2048;
}

size_t evo_bwd_ws_workspace(const mf_evo_bwd_args& a) { return plan_bwd(a).total; }

#define MF_DISPATCH_BIAS(dt, TB, ...)                                         \
  switch (dt) {                                                               \
    case MF_F32: { using TB = float; __VA_ARGS__; } break;                    \
    case MF_BF16: { using TB = __nv_bfloat16; __VA_ARGS__; } break;           \
    case MF_F16: { using TB = __half; __VA_ARGS__; } break;                   \
    default: return fail(MF_ERR_BAD_ARG, "unknown bias dtype %d", (int)(dt)); \
  }

int evo_bwd_ws(const mf_evo_bwd_args& a, const mf_evo_layout& lay, cudaStream_t st) {
  int r = MF_OK;
  if (a.dtype == MF_BF16) {
    MF_DISPATCH_BIAS(a.bias_dtype, TB, { r = a.D <= kDP ? launch_bwd_ws<__nv_bfloat16, TB, 1>(a, lay, st) : launch_bwd_ws<__nv_bfloat16, TB, 2>(a, lay, st); });
  } else {
    MF_DISPATCH_BIAS(a.bias_dtype, TB, { r = a.D <= kDP ? launch_bwd_ws<__half, TB, 1>(a, lay, st) : launch_bwd_ws<__half, TB, 2>(a, lay, st); });
  }
  return r;
}

}  // namespace mf
