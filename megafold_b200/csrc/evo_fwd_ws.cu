// Pair-biased masked attention forward, warp-specialised (tcgen05 + TMEM + TMA), head sizes up to 32.
//
// A persistent CTA (one per SM, 640 threads) runs THREE independent streams.  The CTA owns a contiguous range of work items
// (b, n, h, 128-query tile), which its streams share out; a stream walks, per item, the keys in blocks of 64.  Roles:
//
//   warps 0-3 / 4-7 / 8-11   softmax warpgroup of stream 0 / 1 / 2: one query row (= one TMEM lane) per thread
//   warp 12 / 13 / 14        MMA issuer of stream 0 / 1 / 2
//   warp 16 / 17 / 18        TMA producer of stream 0 / 1 / 2 (15 and 19 only fill their warpgroups)
//
// Per key block the issuer builds   S = Q K^T + sqrt(D) * bias   entirely on the tensor core: two MMAs for Q K^T and
// four [128 x 16] x [16 x 16] MMAs that add the bias tile (A operand, straight from the TMA-loaded tile) times
// alpha * I (B operand), plus, where the block has a masked key, one K = 16 step that adds the key-mask term (a [64 x 16]
// tile, written by the producer warp, times a constant tile) - see evo_tc_common.cuh.  The softmax thread takes the maximum
// of a pair of blocks with three-input max (the positive scale commutes with it), then reads the logits again and writes
// packed 16-bit P = 2^(x - m) over them in TMEM while adding up the row sum (packed adds that hide under the
// exponentials).  P V accumulates into O in TMEM over the key blocks; O and the sum are only multiplied by
// 2^(m_old - m_new) when the running maximum has grown by more than 8 (rare after the first pair; P then stays
// below 2^8, far inside the 16-bit range), or at all (kExactStep).  Only O and the log-sum-exp reach global memory.
//
// Bound: no single unit.  The exponentials, one per logit at 16 a clock and SM, are 50 of the 89 us that [1, 384, 384, 4, 32]
// bf16 takes (256 clocks a warp and 32 logits of its rows; one warp per scheduler needs 11.4 cycles an element in this loop
// with the unit free to it, two 9.3, three 8.9, where 8 saturate it), the issue slots are half used, and with either the
// exponentials or half of the products left out the time falls by 3 % only: what counts is how many softmax warps have work.
// So there are three streams, which leaves a thread 128 registers: the logits are read twice (a TMEM read of 128 columns
// takes 25 cycles).  A stream has two score buffers of 64 keys, so that the products of a block run under the other one's
// exponentials; P overwrites the scores, since TMEM has no room beside them (3 x (2 x 64 + 32) columns).  Step v of a stream's
// products is P V of block v - 2 and the scores of block v, one sequence into one buffer with one completion barrier: it
// says that the scores are there and that the operand buffers of that parity are free again.  The maximum is that of 128
// keys: with one per block of 64 the same call takes 90 us, but other last bits come out, on which the shift gradients of a
// block's pair-bias LayerNorms depend (they are 0 up to rounding), and rows that need rescaling at every new maximum
// (kExactStep) wait for the last product twice as often ([1, 467, 467, 4, 32]: 217 us where pairs take 203).  For the bits' sake the
// exponent stays a difference and a product as well: one fused step for both takes 85 instead of 90 us.
// Measured, [1, 384, 384, 4, 32] bf16 / [1, 467, 467, 4, 32] bf16 (copied bias): 135 / 294 us with two streams of 128-key tiles
// (208 registers a thread, every logit in a register), 115 / 254 with three streams and one score buffer each, 98 / 263 with
// two buffers of 64 keys, 90 / 217 with the operands of the products in uniform registers, 94 / 203 with pairs, 89 / 197 with 128 / 40 registers
// a softmax / helper thread instead of 120 / 56, as now.
// Taken back: loading the next block's logits between the exponentials (109), separate warps for the bias copies and the
// mask terms (108: more warps for the same issue slots), nanosleep in the waits of the helper warps (99), streams started
// a third of a block apart (100; all against 98).
//
// Every wait is bounded; on expiry the CTA raises a flag, all roles run dry without touching global memory, TMEM is
// freed and the host sees mf_async_status() != 0.
#include "evo_tc_common.cuh"

namespace mf {
namespace {
using namespace tcx;

constexpr int kT = 128;                      // queries of an item
constexpr int kB = 64;                       // keys of a block
constexpr int kStreams = 3;
constexpr int kThreads = (kStreams + 2) * 128;
constexpr int kQB = kT * 64;                 // Q tile: [128 x 32] 16-bit, 64-byte rows, 64B swizzle
constexpr int kKB = kB * 64;                 // K and V tiles: [64 x 32]
constexpr int kAtomB = kT * 128;             // bias tile: [128 rows x 64 columns] 16-bit, 128-byte rows, 128B swizzle
constexpr int kXB = kB * 32;                 // mask-term tile: [64 x 16] bf16
constexpr int kStreamBytes = 2 * (kQB + 2 * kKB + kAtomB + kXB);
constexpr int kStreamCols = 2 * kB + 32;     // TMEM columns of a stream: S [0,64) and [64,128), P packed over them, O [128,160)
static_assert(kStreams * kStreamCols <= 512, "TMEM");
constexpr float kRescaleStep = 8.f;          // O is rescaled only when the running maximum grows by more than this (base-2 logits)
// A bias that had to be copied belongs to a length whose calls ran the general kernel (evo_tc_fwd.cu), which takes every
// tile's probabilities relative to the running maximum and the bias as it is.  For them the step is 0 and sqrt(D) keeps its
// second term, so that they are as close to the exact result as there: the largest probability of a row is then exactly 1.
// Distance from 64 bits at [1, 200, 467, 4, 32] bf16: 2.25e-3 with the step of 8 (2.04e-3 the general kernel and now),
// fp16 at 323: 3.02e-4 with it, 2.81e-4 without but with one term, 2.54e-4 now.  It costs 8 % at [1, 467, 467, 4, 32] (182 -> 197 us);
// a template parameter, because a step read from the arguments cost the other lengths 1.5 %.
constexpr float kExactStep = 0.f;

struct FwdWsP {
  int B, N, L, H, D;
  int n_qt, n_kb, n_items, bias_b_mul;
  float c1;               // D^-1/2 * log2(e)
  uint32_t fmt, bfmt;     // tcgen05 operand formats of q/k/v and of the bias (1 = bf16, 0 = f16)
  int n_alpha; float alpha[2];
  const void* mask; int64_t ms[3]; int mask_dtype;
  void* o; TokenStrides os; float* lse; int* status;
};

// Every role waits for each phase of a barrier in turn (see tc.cuh).  The softmax warps need the second step of each pair of
// blocks: with an even number of blocks an item these are the steps of one parity, 1, 3, 5, ...; with an odd number (ODD) the parity
// changes from item to item and they wait for the first step of a pair as well.  A kernel of its own, since code for it in the loop
// cost the even numbers 1 %; [1, 448, 448, 4, 32] 161.5 -> 162.5 us, [1, 264, 264, 4, 32] 59.8 -> 60.3.  (Commits of one warp that arrive in the
// order in which they were issued would do too; that order is not promised.)
struct StreamBars {                      // [parity of the block; of the item for Q]
  uint64_t q_full[2], k_full[2], v_full[2];      // Q tile / K, bias and mask-term tiles / V tile
  uint64_t step_done[2];                 // step v: P V of block v - 2 and the scores of block v are complete
  uint64_t p_ready[2];                   // P is written (the scores, and an item's last O, have been read)
  int masked[2];                         // the block's mask-term tile has anything but zeros
};

// position of a stream's work item
struct ItemPos { int qt, h, n, b; };
__device__ __forceinline__ ItemPos item_pos(int it, const FwdWsP& p) {
  ItemPos x;
  x.qt = it % p.n_qt;
  const int r = it / p.n_qt, bn = r / p.H;
  x.h = r % p.H; x.n = bn % p.N; x.b = bn / p.N;
  return x;
}
__device__ __forceinline__ void step_item(ItemPos& x, const FwdWsP& p) {      // four divisions took 600 cycles each time
  if (++x.qt == p.n_qt) { x.qt = 0; if (++x.h == p.H) { x.h = 0; if (++x.n == p.N) { x.n = 0; ++x.b; } } }
}

constexpr int kLaunchRegs = 96, kSoftmaxRegs = 128, kHelperRegs = 40;      // registers per thread: at launch / after setmaxnreg
static_assert(kLaunchRegs * kThreads <= 65536, "register file");
static_assert(kStreams * 128 * kSoftmaxRegs + 256 * kHelperRegs <= kThreads * kLaunchRegs, "setmaxnreg budget");

template <typename T, typename TB, bool EXACT, bool ODD>      // EXACT: see kExactStep; ODD: an odd number of key blocks, see StreamBars
__global__ void __maxnreg__(kLaunchRegs)
evo_fwd_ws_kernel(const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mk,
                  const __grid_constant__ CUtensorMap mv, const __grid_constant__ CUtensorMap mb, const FwdWsP p MF_TRACE_PARAM) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sI = smem + kStreams * kStreamBytes;       // alpha * I tiles, 1 KB each
  uint8_t* sXO = sI + 2048;                           // constant partner tile of the mask term

  __shared__ StreamBars bars[kStreams];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;

  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  if (tid == 0) {
    abort_s = 0;
    for (int q = 0; q < kStreams; ++q)
      for (int i = 0; i < 2; ++i) {
        StreamBars& b = bars[q];
        mbar_init(&b.q_full[i], 1); mbar_init(&b.v_full[i], 1); mbar_init(&b.step_done[i], 1);
        mbar_init(&b.k_full[i], 2);       // the copies and the mask-term tile
        mbar_init(&b.p_ready[i], 4);      // one arrival per softmax warp
      }
    mbar_fence_init();
    prefetch_tmap(&mq); prefetch_tmap(&mk); prefetch_tmap(&mv); prefetch_tmap(&mb);
  }
  // constant MMA operand: alpha * I (bias)
  write_alpha_identity<TB>(sI, p.alpha[0], tid, kThreads);
  write_alpha_identity<TB>(sI + 1024, p.alpha[1], tid, kThreads);
  write_xo_tile(sXO, tid, kThreads);
  fence_async_smem();
  if (warp == 0) { tmem_alloc(&tmem_base_s, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  volatile int* abort_flag = &abort_s;

  const int s = warp < 4 * kStreams ? warp >> 2 : (warp & 3) % kStreams;      // stream of this warp
  StreamBars& bar = bars[s];
  uint8_t* sB = smem + s * kStreamBytes;                      // [2 parities] each
  uint8_t* sQ = sB + 2 * kAtomB;
  uint8_t* sK = sQ + 2 * kQB;
  uint8_t* sV = sK + 2 * kKB;
  uint8_t* sXK = sV + 2 * kKB;
  const uint32_t tbase = uniform(tmem_base_s) + s * kStreamCols;

  // items of this CTA, then of this stream: whole CTAs differ by one item at most, and so do the streams of one
  const int cta_begin = (int)((int64_t)blockIdx.x * p.n_items / gridDim.x), cta_n = (int)((int64_t)(blockIdx.x + 1) * p.n_items / gridDim.x) - cta_begin;
  const int item_begin = cta_begin + s * cta_n / kStreams;
  const int n_my = cta_begin + (s + 1) * cta_n / kStreams - item_begin;
  const int n_kb = p.n_kb;
  const uint32_t n_blk = (uint32_t)n_my * n_kb;               // key blocks of this stream

  if (warp < 4 * kStreams) {
    // =========================================================================== softmax warpgroup
    // Register re-partition: the CTA is launched with kLaunchRegs registers per thread; the helper warps drop to
    // kHelperRegs and the softmax warpgroups rise to kSoftmaxRegs.  The raise can only draw on what the drop releases
    // inside this CTA (otherwise it never returns): the launcher checks the launch figure.
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSoftmaxRegs));
    const int r = (warp & 3) * 32 + lane;
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tO = tbase + 2 * kB + lane_addr;
    const float2 c1c1 = make_float2(p.c1, p.c1);
    MF_TRACE_DECL(tr, s, blockIdx.x == 0 && (warp & 3) == 0 && lane == 0);
    ItemPos pos = item_pos(item_begin, p);
    float l_done = 1.f, m_done = 0.f;
    int i_done = 0;
    T* o_done = nullptr;
    float* lse_done = nullptr;
    auto wait_step = [&](uint32_t v) { wait_or_flag(&bar.step_done[v & 1], (v >> 1) & 1, abort_flag); tc_fence_after(); };
    // O / l and the log-sum-exp of the item before, whose last product is complete
    auto write_out = [&]() {
      const bool gone = *abort_flag;
      store_rows(tO, 1.f / l_done, o_done, p.os.l, i_done, gone ? 0 : p.L, p.D);
      if (gone) return;
      // a row whose keys are all masked has every logit at the mask term (about -1e30): uniform attention over its L
      // keys; its log-sum-exp is stored as -FLT_MAX, the value the backward kernels recognise
      if (i_done < p.L) *lse_done = m_done <= -1e28f ? -FLT_MAX : (m_done * p.c1 + lg2f(l_done)) * kLn2;
    };
    uint32_t u = 0;                                // block of the stream
    for (int il = 0; il < n_my; ++il) {
      const int i = pos.qt * kT + r;
      float m_used = 0.f;
      float2 lsum0 = make_float2(0.f, 0.f), lsum1 = lsum0;        // row sum of P relative to m_used (four partial sums)
      for (int t = 0; t < n_kb; t += 2) {          // a pair of blocks shares one maximum
        const uint32_t tS = tbase + (u & 1) * kB + lane_addr, tN = tbase + (~u & 1) * kB + lane_addr;
        const bool two = t + 1 < n_kb;
        tr(1);
        if (ODD) wait_step(u);
        wait_step(u + 1);                          // scores of both blocks, and every earlier product: O may be read and rescaled
        tr(2);
        // ---------------------------------------------------------------- pass 1: the maximum.  Bias and key mask are
        // already inside S (tensor core), and the scale c1 > 0 commutes with the maximum: nothing but three-input maxima.
        // The second block first: the first one is then in place for its exponentials.
        uint32_t sa[32], sc[32];
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        auto fold = [&](const uint32_t (&x)[32]) {
#pragma unroll
          for (int c4 = 0; c4 < 8; ++c4) {
            mx[c4 & 1 ? 2 : 0] = max3f(mx[c4 & 1 ? 2 : 0], __uint_as_float(x[c4 * 4]), __uint_as_float(x[c4 * 4 + 1]));
            mx[c4 & 1 ? 3 : 1] = max3f(mx[c4 & 1 ? 3 : 1], __uint_as_float(x[c4 * 4 + 2]), __uint_as_float(x[c4 * 4 + 3]));
          }
        };
        if (two) {
          tmem_ld32(tN, sa); tmem_ld32(tN + 32, sc);
          tmem_ld_wait(sa, sc);
          fold(sa); fold(sc);
        }
        tmem_ld32(tS, sa); tmem_ld32(tS + 32, sc);
        tmem_ld_wait(sa, sc);
        fold(sa); fold(sc);
        const float m_blk = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));      // in units of the unscaled scores
        tr(3);
        if (t == 0) {
          m_used = m_blk;
        } else {
          const bool grow = (m_blk - m_used) * p.c1 > (EXACT ? kExactStep : kRescaleStep);
          if (__any_sync(0xffffffffu, grow)) {
            // rare: bring O and the row sum of this warp's rows to the new maximum
            const float f = grow ? ex2f((m_used - m_blk) * p.c1) : 1.f;
            if (grow) m_used = m_blk;
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
              uint32_t o16[16];
              tmem_ld16(tO + hf * 16, o16);
              tmem_ld_wait();
#pragma unroll
              for (int d = 0; d < 16; ++d) o16[d] = __float_as_uint(__uint_as_float(o16[d]) * f);
              tmem_st16(tO + hf * 16, o16);
            }
            lsum0.x *= f; lsum0.y *= f; lsum1.x *= f; lsum1.y *= f;
          }
        }
        // ---------------------------------------------------------------- pass 2: P = 2^(x - m) as packed 16-bit
        // x = c1 * (s - m): the difference first, so that logits equal to the maximum give exactly 0 whatever their size
        // (a fully masked row sits at about -1e30, where a fused c1 * s - c1 * m would leave a huge rounding residue)
        const float2 mm = make_float2(m_used, m_used);
        auto exps = [&](const uint32_t (&x)[32], uint32_t tP) {
          uint32_t pk[16];
#pragma unroll
          for (int jj = 0; jj < 16; jj += 2) {
            const float2 xa = mul2(sub2(make_float2(__uint_as_float(x[2 * jj]), __uint_as_float(x[2 * jj + 1])), mm), c1c1);
            const float2 xb = mul2(sub2(make_float2(__uint_as_float(x[2 * jj + 2]), __uint_as_float(x[2 * jj + 3])), mm), c1c1);
            const float2 ea = make_float2(ex2f(xa.x), ex2f(xa.y)), eb = make_float2(ex2f(xb.x), ex2f(xb.y));
            lsum0 = add2(lsum0, ea); lsum1 = add2(lsum1, eb);
            pk[jj] = Pack2<T>::pack(ea.x, ea.y); pk[jj + 1] = Pack2<T>::pack(eb.x, eb.y);
          }
          tmem_st16(tP, pk);
        };
        auto hand_over = [&](uint32_t blk) {       // P of a block to the issuer
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar.p_ready[blk & 1]);
        };
        exps(sa, tS);
        if (two) tmem_ld32(tN, sa);
        exps(sc, tS + 16);
        tr(4);
        if (t == 0 && il > 0) write_out();         // before the first product of this item starts O afresh
        hand_over(u);
        ++u;
        if (two) {
          tmem_ld32(tN + 32, sc);
          tmem_ld_wait(sa, sc);
          exps(sa, tN);
          exps(sc, tN + 16);
          hand_over(u);
          ++u;
        }
        tr(5);
      }
      // the item's last product is under way: what its output needs is kept until the next item's first block
      l_done = (lsum0.x + lsum0.y) + (lsum1.x + lsum1.y); m_done = m_used; i_done = i;
      o_done = static_cast<T*>(p.o) + p.os.at(pos.b, pos.n, i) + pos.h * p.D;
      lse_done = p.lse + (((int64_t)pos.b * p.N + pos.n) * p.H + pos.h) * p.L + i;
      step_item(pos, p);
    }
    if (n_my > 0) {
      wait_step(u + 1);                            // the last block's product
      write_out();
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kHelperRegs));
    // The helper roles are run by whole warps (one elected lane issues: see mma_ss_el); every exit decision is a warp vote.
    auto dead = [&] { return __any_sync(0xffffffffu, *abort_flag) != 0; };
    if (warp < 4 * kStreams + kStreams) {
      // ========================================================================= MMA issuer of stream s
      const uint32_t id_s = idesc_f16(kT, kB, p.fmt, 0, 0);
      const uint32_t id_b = idesc_f16(kT, 16, p.bfmt, 0, 0);
      const uint32_t id_x = idesc_f16(kT, kB, 1u, 0, 0);           // the mask-term tiles are bf16 whatever q/k/v are
      const uint32_t id_o = idesc_f16(kT, 32, p.fmt, 0, 1);        // B (V) MN-major
      constexpr uint32_t hi64 = desc_hi(512, kSw64), hi128 = desc_hi(1024, kSw128), hi32 = desc_hi(256, kSw32);
      const uint32_t q_base = desc_lo(smem_u32(sQ), 16), k_base = desc_lo(smem_u32(sK), 16), v_base = desc_lo(smem_u32(sV), 16), b_base = desc_lo(smem_u32(sB), 16);
      const uint32_t i_lo0 = desc_lo(smem_u32(sI), 16), i_lo1 = i_lo0 + 1024 / 16, xo_lo = desc_lo(smem_u32(sXO), 16), xk_base = desc_lo(smem_u32(sXK), 16);
      const uint32_t tO = tbase + 2 * kB;
      const bool two_terms = p.n_alpha > 1;
      MF_TRACE_DECL(tr, 3 + s, blockIdx.x == 0 && lane == 0);
      int t = 0, il = 0;                                      // key block and item of block v
      int tp = 0;                                             // key block of block v - 2
      for (uint32_t v = 0; n_blk > 0 && v < n_blk + 2; ++v) {
        const uint32_t par = v & 1, phase = (v >> 1) & 1, tS = tbase + par * kB;
        tr(10);
        if (v < n_blk) {
          if (t == 0) wait_or_flag(&bar.q_full[il & 1], (il >> 1) & 1, abort_flag);
          wait_or_flag(&bar.k_full[par], phase, abort_flag);
        }
        tr(11);
        if (v >= 2) {
          wait_or_flag(&bar.v_full[par], phase ^ 1, abort_flag);
          wait_or_flag(&bar.p_ready[par], phase ^ 1, abort_flag);
        }
        tc_fence_after();
        tr(12);
        if (dead()) break;
        if (v >= 2) {                                         // O (+)= P V; the first product of an item starts O afresh
          const uint32_t v_lo = v_base + par * (kKB / 16);
          mma_ts_el(tO, tS, v_lo, hi64, id_o, tp > 0);
#pragma unroll
          for (int ks = 1; ks < kB / 16; ++ks) mma_ts_el(tO, tS + ks * 8, v_lo + ks * 64, hi64, id_o, true);
          if (++tp == n_kb) tp = 0;
        }
        tr(13);
        if (v < n_blk) {
          const uint32_t q_lo = q_base + (il & 1) * (kQB / 16), k_lo = k_base + par * (kKB / 16), b_lo = b_base + par * (kAtomB / 16);
          mma_ss_el(tS, q_lo, hi64, k_lo, hi64, id_s, false);
          mma_ss_el(tS, q_lo + 2, hi64, k_lo + 2, hi64, id_s, true);
          if (uniform(bar.masked[par])) mma_ss_el(tS, xo_lo, hi32, xk_base + par * (kXB / 16), hi32, id_x, true);        // + key mask
#pragma unroll
          for (int c = 0; c < 4; ++c) mma_ss_el(tS + c * 16, b_lo + c * 2, hi128, i_lo0, hi64, id_b, true);      // 16 key columns each
          if (two_terms) {
#pragma unroll
            for (int c = 0; c < 4; ++c) mma_ss_el(tS + c * 16, b_lo + c * 2, hi128, i_lo1, hi64, id_b, true);
          }
          if (++t == n_kb) { t = 0; ++il; }
        }
        tc_commit_el(&bar.step_done[par]);
        tr(14);
      }
    } else if (warp >= 4 * kStreams + 4 && warp < 5 * kStreams + 4) {
      // ========================================================================= TMA producer of stream s
      // Mask term of key j of row (b, n), in units of the unscaled scores (x sqrt(D)): 0 / -1e30 for a keep-mask, the value
      // for an additive mask; keys beyond L get -2e30 so that even a fully masked row (all its keys at -1e30) excludes them.
      // The mask values of a block are fetched one block ahead as raw bits (two independent loads) and converted when the
      // tile is written, so that their latency is never waited for.
      const float sqrt_d = sqrtf((float)p.D);
      uint32_t raw[kB / 32] = {};
      auto fetch = [&](const ItemPos& x, int j0) {
        const int64_t row = x.b * p.ms[0] + x.n * p.ms[1];
#pragma unroll
        for (int k = 0; k < kB / 32; ++k) {
          int j = j0 + k * 32 + lane;
          if (j >= p.L) j = p.L - 1;
          const int64_t mi = row + j * p.ms[2];
          raw[k] = p.mask_dtype == MF_U8 ? static_cast<const uint8_t*>(p.mask)[mi]
                   : p.mask_dtype == MF_F32 ? static_cast<const uint32_t*>(p.mask)[mi] : static_cast<const uint16_t*>(p.mask)[mi];
        }
      };
      auto term = [&](uint32_t bits, int j) {
        float v;
        if (p.mask_dtype == MF_U8) v = bits ? 0.f : kMinusBig;
        else {
          const float x = p.mask_dtype == MF_F32 ? __uint_as_float(bits)
                          : p.mask_dtype == MF_BF16 ? __uint_as_float(bits << 16) : __half2float(__ushort_as_half((unsigned short)bits));
          v = fmaxf(x * sqrt_d, kMinusBig);
        }
        return j < p.L ? v : 2.f * kMinusBig;
      };
      // The block's mask-term tile XK (rows = keys; columns 0..2 = split3 of the term), written by the whole warp unless
      // every term is 0: then nothing need be added.
      auto write_xk = [&](int j0, uint32_t par) {
        float v[kB / 32];
        bool any = false;
#pragma unroll
        for (int k = 0; k < kB / 32; ++k) { v[k] = term(raw[k], j0 + k * 32 + lane); any |= v[k] != 0.f; }
        any = __any_sync(0xffffffffu, any);
        if (any) {
          uint8_t* xt = sXK + par * kXB;
#pragma unroll
          for (int k = 0; k < kB / 32; ++k) {
            __nv_bfloat16 m3[3];
            const int r = k * 32 + lane;
            split3(v[k], m3);
            *reinterpret_cast<uint4*>(xt + swz_offset(r, 0, 32)) = make_uint4(pack_bf(m3[0], m3[1]), pack_bf(m3[2], __float2bfloat16_rn(0.f)), 0u, 0u);
            *reinterpret_cast<uint4*>(xt + swz_offset(r, 1, 32)) = make_uint4(0u, 0u, 0u, 0u);
          }
          fence_async_smem();
        }
        if (lane == 0) bar.masked[par] = any;
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar.k_full[par]);
      };
      MF_TRACE_DECL(tr, 6, blockIdx.x == 0 && s == 0 && lane == 0);
      // A bulk-tensor copy keeps the thread that issues it busy for a few hundred cycles whatever its size; several lanes of
      // one warp issuing in the same instruction cost little more than one.  So lanes 0 to 3 request the K and bias tiles of
      // block v, the V tile of block v - 2 and, at an item's first block, its Q tile together.
      const CUtensorMap* my_map = lane == 0 ? &mk : lane == 1 ? &mb : lane == 2 ? &mv : &mq;
      ItemPos pos = item_pos(item_begin, p), vpos = pos;      // items of blocks v and v - 2
      int t = 0, tv = 0, il = 0;
      uint32_t v = 0;                                         // blocks requested so far
      if (n_blk > 0) fetch(pos, 0);
      for (; n_blk > 0 && v < n_blk + 2; ++v) {
        const uint32_t par = v & 1;
        tr(20);
        if (v >= 2) wait_or_flag(&bar.step_done[par], ((v >> 1) & 1) ^ 1, abort_flag);
        tr(21);
        if (dead()) break;
        const bool more = v < n_blk;
        if (lane == 0 && more) mbar_expect_tx(&bar.k_full[par], kKB + kAtomB);
        if (lane == 2 && v >= 2) mbar_expect_tx(&bar.v_full[par], kKB);
        if (lane == 3 && more && t == 0) mbar_expect_tx(&bar.q_full[il & 1], kQB);
        __syncwarp();
        if (lane < 4 && (lane == 2 ? v >= 2 : more && (lane != 3 || t == 0))) {
          uint64_t* full = lane < 2 ? &bar.k_full[par] : lane == 2 ? &bar.v_full[par] : &bar.q_full[il & 1];
          uint8_t* dst = lane == 0 ? sK + par * kKB : lane == 1 ? sB + par * kAtomB : lane == 2 ? sV + par * kKB : sQ + (il & 1) * kQB;
          int c0 = 0, c1 = pos.h, c2 = t * kB, c3 = pos.n, c4 = pos.b;
          if (lane == 1) { c0 = t * kB; c1 = pos.qt * kT; c2 = pos.h; c3 = pos.b * p.bias_b_mul; c4 = 0; }
          if (lane == 2) { c1 = vpos.h; c2 = tv * kB; c3 = vpos.n; c4 = vpos.b; }
          if (lane == 3) c2 = pos.qt * kT;
          tma_load_5d(dst, my_map, full, c0, c1, c2, c3, c4);
        }
        __syncwarp();
        tr(22);
        if (v >= 2 && ++tv == n_kb) { tv = 0; step_item(vpos, p); }
        if (more) {
          write_xk(t * kB, par);
          if (++t == n_kb) { t = 0; ++il; step_item(pos, p); }
          if (v + 1 < n_blk) fetch(pos, t * kB);
        }
        tr(23);
      }
      if (dead() && lane == 0) {
        // the copies already requested must land before the CTA's shared memory is given back (bounded)
        const uint32_t nk = v < n_blk ? v : n_blk, nv = v > 2 ? v - 2 : 0, nq = il + (t > 0);
        drain_ring(bar.q_full, nq, 2); drain_ring(bar.k_full, nk, 2); drain_ring(bar.v_full, nv, 2);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && abort_s) *reinterpret_cast<volatile int*>(p.status) = 1;
  if (warp == 0) tmem_dealloc(tmem_base_s, 512);
}

template <typename T, typename TB, bool EXACT, bool ODD>
int launch_fwd_ws(const mf_evo_fwd_args& a, const mf_evo_layout& lay, cudaStream_t st) {
  CUtensorMap mq, mk, mv, mb;
  int r;
  if ((r = make_qkv_map(&mq, a.q, a.dtype, a.B, a.N, a.L, a.H, a.D, a.q_strides, 32, kT))) return r;
  if ((r = make_qkv_map(&mk, a.k, a.dtype, a.B, a.N, a.L, a.H, a.D, a.k_strides, 32, kB))) return r;
  if ((r = make_qkv_map(&mv, a.v, a.dtype, a.B, a.N, a.L, a.H, a.D, a.v_strides, 32, kB))) return r;
  FwdWsP p{};
  p.B = a.B; p.N = a.N; p.L = a.L; p.H = a.H; p.D = a.D;
  p.n_qt = (a.L + kT - 1) / kT; p.n_kb = (a.L + kB - 1) / kB;
  p.n_items = a.B * a.N * a.H * p.n_qt;
  p.c1 = kLog2e / sqrtf((float)a.D);
  p.fmt = a.dtype == MF_BF16 ? 1u : 0u;
  p.bfmt = a.bias_dtype == MF_BF16 ? 1u : 0u;
  p.n_alpha = split_alpha(a.D, a.bias_dtype, p.alpha, EXACT);
  p.mask = a.mask; for (int i = 0; i < 3; ++i) p.ms[i] = a.mask_strides[i];
  p.mask_dtype = a.mask_dtype;
  p.o = a.o; p.os = token_strides(lay.o); p.lse = a.lse;
  p.status = status_word();
  MF_REQUIRE(p.status, MF_ERR_CUDA, "could not allocate the device status word");
  MF_REQUIRE(tc_async_status() == 0, MF_ERR_CUDA, "an earlier tensor-core kernel gave up on a bounded wait; results are invalid");
  p.bias_b_mul = a.bias_strides[0] == 0 ? 0 : 1;
  {
    // five dimensions (the last one a dummy) so that one instruction, issued by several lanes, loads K and bias tiles alike
    const int64_t dims[5] = {a.L, a.L, a.H, p.bias_b_mul ? a.B : 1, 1};
    const int64_t str[5] = {1, a.bias_strides[2], a.bias_strides[1], a.bias_strides[0], 0};
    const int box[5] = {kB, kT, 1, 1, 1};
    if ((r = make_tiled_map(&mb, a.bias, a.bias_dtype, 5, dims, str, box, 128))) return r;
  }
  int grid = sm_count();
  if (grid > p.n_items) grid = p.n_items;
  const size_t smem = 1024 + kStreams * (size_t)kStreamBytes + 2048 + kXTileB;
  constexpr auto kern = evo_fwd_ws_kernel<T, TB, EXACT, ODD>;
  if (int e = opt_in_smem<kern>(smem, kLaunchRegs)) return e;
  kern<<<grid, kThreads, smem, st>>>(mq, mk, mv, mb, p MF_TRACE_ARG);
  MF_LAUNCHED("evo_fwd_ws_kernel");
  return MF_OK;
}

template <bool EXACT, bool ODD>
int dispatch(const mf_evo_fwd_args& a, const mf_evo_layout& lay, cudaStream_t st) {
  if (a.dtype == MF_BF16)
    return a.bias_dtype == MF_BF16 ? launch_fwd_ws<__nv_bfloat16, __nv_bfloat16, EXACT, ODD>(a, lay, st) : launch_fwd_ws<__nv_bfloat16, __half, EXACT, ODD>(a, lay, st);
  return a.bias_dtype == MF_BF16 ? launch_fwd_ws<__half, __nv_bfloat16, EXACT, ODD>(a, lay, st) : launch_fwd_ws<__half, __half, EXACT, ODD>(a, lay, st);
}

}  // namespace

// The warp-specialised kernel covers head sizes up to 32, rows up to 2048 tokens and a 16-bit pair bias; other calls use
// the general kernel.
static bool shape_ok(const mf_evo_fwd_args& a) { return a.D <= 32 && a.L <= 2048 && (a.bias_dtype == MF_BF16 || a.bias_dtype == MF_F16); }

// A bias whose rows TMA cannot address (a chain of odd length) is copied to a 16-byte pitch when the caller gives the
// scratch for it: an exact copy in 3 us.  At [1, 467, 467, 4, 32] the call takes 197 us, where the general kernel that reads
// such a bias in place takes 1263, and the same kernel on the copied bias 457.
size_t evo_fwd_ws_workspace(const mf_evo_fwd_args& a) {
  if (!shape_ok(a) || bias_tma_ok(a.bias, a.bias_dtype, a.bias_strides, a.B, a.H)) return 0;
  return bias_copy_bytes(a.bias_strides, a.B, a.H, a.L);
}
bool evo_fwd_ws_supported(const mf_evo_fwd_args& a, size_t workspace_bytes) {
  return shape_ok(a) && workspace_bytes >= evo_fwd_ws_workspace(a);
}

int evo_fwd_ws(const mf_evo_fwd_args& args, const mf_evo_layout& lay, void* workspace, cudaStream_t st) {
  mf_evo_fwd_args a = args;
  const bool copied = evo_fwd_ws_workspace(args) != 0;
  if (copied) {
    int r = copy_bias_rows(a.bias, a.bias_dtype, a.bias_strides, workspace, a.bias_dtype, a.B, a.H, a.L, st);
    if (r) return r;
    const int64_t row = bias_pitch(a.L);
    a.bias = workspace;
    a.bias_strides[3] = 1; a.bias_strides[2] = row; a.bias_strides[1] = row * a.L;
    a.bias_strides[0] = args.bias_strides[0] == 0 ? 0 : row * a.L * a.H;
  }
  const bool odd = (a.L + kB - 1) / kB % 2 != 0;
  if (copied) return odd ? dispatch<true, true>(a, lay, st) : dispatch<true, false>(a, lay, st);
  return odd ? dispatch<false, true>(a, lay, st) : dispatch<false, false>(a, lay, st);
}

}  // namespace mf
