// Pair-biased masked attention forward on the tensor cores (tcgen05 + TMEM + TMA): the GENERAL kernel, for the calls
// the warp-specialised kernel (evo_fwd_ws.cu) does not take - head sizes 33..64, an fp32 or unaligned pair bias,
// rows longer than 2048 tokens.
//
// A persistent CTA (one per SM, 256 threads) runs TWO independent streams, one per warpgroup.  A stream walks a
// contiguous range of work items (b, n, h, 128-query tile) and, per item, the key tiles (128 keys, 64 for DP = 64).  Inside a stream every
// thread owns one query row (= one TMEM lane); "officers" of the warpgroup also issue the stream's
// tcgen05.mma instructions (warp 0, through an elected lane), its Q/K/V TMA loads (thread 32) and its bias TMA loads (thread 64):
//
//   wait S(t) in TMEM -> tcgen05.ld the whole row of the tile into registers -> group barrier ->
//   S(t+1) = Q K(t+1)^T is issued at once (the S buffer is free again: registers double-buffer it)
//   -> row thread: logits in base 2 (scale, bias from shared memory, key mask), running max, exp2,
//   row sum, packed 16-bit P -> fold O_tile(t-1) from TMEM into the register accumulator ->
//   tcgen05.st P -> group barrier -> O_tile(t) = P V(t) is issued (P as TMEM A operand, V as
//   MN-major B operand) and the TMA rings are topped up.
//
// Operand tiles are [128 rows x DP] (DP = 32: 64-byte rows, 64B swizzle; DP = 64: 128-byte rows) fetched
// from the strided [B, N, L, H, D] tensors by 5-D tensor maps; smaller head sizes are zero-filled by TMA.
// A 16-bit pair bias with TMA-addressable rows is staged as [128 rows x 64 columns] chunks (128-byte rows, 128B
// swizzle, DP = 32 only).  Other aligned biases (fp32, or DP = 64 whose operand tiles leave less room) go through a ring per
// warp of [32 rows x 64 bytes] chunks, filled by cp.async six chunks ahead: the row threads' own loads from global memory,
// 128 bytes of a row at a time with their latency in the open, made the fp32 bias of [4, 1, 384, 32, 64] cost 72 us where
// this takes 48.  Unaligned or strided biases, and DP = 64 beyond 2176 keys (the mask rows need the room), are still read
// by the row thread.
//
// Every wait is bounded; on expiry the CTA raises a flag that all threads honour at their next group
// barrier, TMEM is freed and the host sees mf_async_status() != 0.
#include "evo_tc_common.cuh"

namespace mf {
namespace {
using namespace tcx;

constexpr int kQT = 128;
constexpr int kThreads = 256;
constexpr int kVS = 2;        // V ring stages per stream
constexpr int kBC = 3;        // bias chunk ring per stream (2 chunks per key tile: every TMA issue costs the
                              // issuing thread, a lane of a compute warp, some hundreds of cycles)
constexpr int kBCW = 64;      // columns per bias chunk (128-byte rows)
constexpr int kBChunkBytes = 128 * kBCW * 2;
constexpr size_t kSmemLimit = 232448 - 1024;       // of a block, less the static arrays
constexpr int kWChunkBytes = 32 * 64;      // staged bias: ring per warp
enum BiasMode { kDirect, kTma, kStaged };

template <int DP> struct Cfg {
  static constexpr int ROWB = DP * 2;
  // keys per tile: a row thread holds its scores and its DP outputs in registers; 128 + 64 spilled 100 registers to L2
  static constexpr int KT = DP == 32 ? 128 : 64;
  static constexpr int QB = kQT * ROWB, TILEB = KT * ROWB;
  static constexpr int KS = 3;                    // K ring stages per stream
  static constexpr int WC = 6;                    // staged bias: chunks in the ring of a warp
  static constexpr Swizzle SW = DP == 32 ? kSw64 : kSw128;
  static constexpr int SBO = 8 * ROWB;
  static constexpr int STREAM_BYTES(int mode) {
    return QB + TILEB * (KS + kVS) + (mode == kTma ? kBC * kBChunkBytes : mode == kStaged ? 4 * WC * kWChunkBytes : 0);
  }
};

struct FwdP {
  int B, N, L, H, D;
  int n_qt, n_kt, n_items, lpad, items_per_stream, bias_b_mul;
  float c1;               // D^-1/2 * log2(e)
  uint32_t ab_fmt;        // 1 = bf16, 0 = f16
  const void* bias; int64_t bs[4]; int bias_fast;
  const void* mask; int64_t ms[3]; int mask_dtype;
  void* o; TokenStrides os; float* lse; int* status;
};

struct StreamBars {
  uint64_t q_full, k_full[3], v_full[kVS], b_full[kBC], b_empty[kBC], s_ready, pv_done;
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src, int bytes) {      // the rest of the 16 is zero
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// 32 consecutive bias values of one row as fp32 from global memory; `p` 16-byte aligned, in bounds.
template <typename TB>
__device__ __forceinline__ void load_bias32_fast(const TB* p, float (&out)[32]) {
  if constexpr (sizeof(TB) == 4) {
    const float4* v = reinterpret_cast<const float4*>(p);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float4 x = __ldg(v + i);
      out[4 * i] = x.x; out[4 * i + 1] = x.y; out[4 * i + 2] = x.z; out[4 * i + 3] = x.w;
    }
  } else {
    const uint4* v = reinterpret_cast<const uint4*>(p);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint4 x = __ldg(v + i);
      float2 a = Pack2<TB>::unpack(x.x), b = Pack2<TB>::unpack(x.y), c = Pack2<TB>::unpack(x.z), d = Pack2<TB>::unpack(x.w);
      out[8 * i] = a.x; out[8 * i + 1] = a.y; out[8 * i + 2] = b.x; out[8 * i + 3] = b.y;
      out[8 * i + 4] = c.x; out[8 * i + 5] = c.y; out[8 * i + 6] = d.x; out[8 * i + 7] = d.y;
    }
  }
}
template <typename TB>
__device__ __forceinline__ void load_bias32_slow(const TB* row, int64_t sj, int j0, int L, float (&out)[32]) {
#pragma unroll
  for (int i = 0; i < 32; ++i) out[i] = (j0 + i < L) ? to_f(row[(int64_t)(j0 + i) * sj]) : 0.f;
}

template <int DP, typename T, typename TB, int BM>
__global__ void __launch_bounds__(kThreads, 1)
evo_fwd_tc_kernel(const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mk,
                  const __grid_constant__ CUtensorMap mv, const __grid_constant__ CUtensorMap mb, const FwdP p) {
  using C = Cfg<DP>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  constexpr int kKT = C::KT, kWC = C::WC, kStreamBytes = C::STREAM_BYTES(BM);

  __shared__ StreamBars bars[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;

  // A 16-bit bias read element by element is the one form that is slower with uniform operands (the compiler then spills three times as much in the
  // loop over its columns: [4, 1, 322, 8, 48] 38 -> 42 us; staged and TMA forms [4, 1, 384, 32, 64] 48 -> 44 and 43 -> 39).
  constexpr bool kUniform = BM != kDirect || sizeof(TB) != 2;
  const int tid = threadIdx.x, warp = kUniform ? uniform(tid >> 5) : tid >> 5, lane = tid & 31;
  const int s = warp >> 2;                    // stream = warpgroup
  const int wg_tid = tid & 127;
  const bool leader = (warp & 3) == 0;
  if (tid == 0) {
    abort_s = 0;
    for (int q = 0; q < 2; ++q) {
      StreamBars& b = bars[q];
      mbar_init(&b.q_full, 1);
      for (int i = 0; i < 3; ++i) mbar_init(&b.k_full[i], 1);
      for (int i = 0; i < kVS; ++i) mbar_init(&b.v_full[i], 1);
      for (int i = 0; i < kBC; ++i) { mbar_init(&b.b_full[i], 1); mbar_init(&b.b_empty[i], 128); }
      mbar_init(&b.s_ready, 1);
      mbar_init(&b.pv_done, 1);
    }
    mbar_fence_init();
    prefetch_tmap(&mq); prefetch_tmap(&mk); prefetch_tmap(&mv);
    if (BM == kTma) prefetch_tmap(&mb);
  }
  if (warp == 0) { tmem_alloc(&tmem_base_s, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  volatile int* abort_flag = &abort_s;
  StreamBars& bar = bars[s];
  uint8_t* sb = smem + s * kStreamBytes;
  uint8_t* sQ = sb;
  uint8_t* sK = sQ + C::QB;
  uint8_t* sV = sK + C::KS * C::TILEB;
  uint8_t* sB = sV + kVS * C::TILEB;
  float* mask2 = reinterpret_cast<float*>(smem + 2 * kStreamBytes) + s * p.lpad;

  const int r = (warp & 3) * 32 + lane;                              // TMEM lane = query row in the tile
  const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
  const uint32_t tS = tmem_base_s + s * 256 + lane_addr, tP = tS + 128, tO = tS + 192;
  const uint32_t tS0 = (kUniform ? uniform(tmem_base_s) : tmem_base_s) + s * 256;                      // lane 0 addresses for the MMA issuer
  const uint32_t id_s = idesc_f16(128, kKT, p.ab_fmt, 0, 0);
  const uint32_t id_o = idesc_f16(128, DP, p.ab_fmt, 0, 1);

  // first streams of all SMs before the second ones: where there are fewer items than streams, or one and a bit per stream,
  // most SMs then run one stream undisturbed
  const int stream = s * gridDim.x + blockIdx.x;
  const int item_begin = stream * p.items_per_stream;
  int item_end = item_begin + p.items_per_stream;
  if (item_end > p.n_items) item_end = p.n_items;
  const int n_my = item_end > item_begin ? item_end - item_begin : 0;
  const int g_total = n_my * p.n_kt;
  const int per_bn = p.H * p.n_qt;

  // ---- TMA bookkeeping.  Three "officers" per stream share the issue work so that none of it piles up on
  // one warp: warp 0 issues the MMAs, thread 32 the Q/K/V loads, thread 64 the bias loads.
  // A cursor walks (item, key tile) incrementally: no divisions on the hot path.
  struct Cursor {
    int qt, h, n, b, t, item_local;
  };
  auto cursor_init = [&](Cursor& c) {
    const int it = item_begin;
    c.qt = it % p.n_qt; c.h = (it / p.n_qt) % p.H;
    const int bn = it / per_bn;
    c.n = bn % p.N; c.b = bn / p.N; c.t = 0; c.item_local = 0;
  };
  auto cursor_next_item = [&](Cursor& c) {
    c.t = 0; ++c.item_local;
    if (++c.qt == p.n_qt) { c.qt = 0; if (++c.h == p.H) { c.h = 0; if (++c.n == p.N) { c.n = 0; ++c.b; } } }
  };
  auto cursor_next_tile = [&](Cursor& c) { if (++c.t == p.n_kt) cursor_next_item(c); };
  const bool officer_kv = wg_tid == 32, officer_b = wg_tid == 64;
  Cursor ck, cv, cq, cbias;
  cursor_init(ck); cursor_init(cv); cursor_init(cq); cursor_init(cbias);
  int gk = 0, gv = 0, cb_next = 0, cb_quarter = 0;
  uint32_t kslot = 0, vslot = 0, pslot = 0, puse = 0;
  auto issue_q = [&]() {      // Q of the cursor's item, then advance to the next item
    mbar_expect_tx(&bar.q_full, C::QB);
    tma_load_5d(sQ, &mq, &bar.q_full, 0, cq.h, cq.qt * kQT, cq.n, cq.b);
    cursor_next_item(cq);
  };
  // K tiles may be requested up to KS ahead of the last S that is known to be complete (s_done tiles)
  auto pump_k = [&](int s_done) {
    while (gk < g_total && gk < s_done + C::KS) {
      mbar_expect_tx(&bar.k_full[kslot], C::TILEB);
      tma_load_5d(sK + kslot * C::TILEB, &mk, &bar.k_full[kslot], 0, ck.h, ck.t * kKT, ck.n, ck.b);
      cursor_next_tile(ck); ++gk;
      if (++kslot == C::KS) kslot = 0;
    }
  };
  auto pump_v = [&](int pv_done_cnt) {
    while (gv < g_total && gv < pv_done_cnt + kVS) {
      mbar_expect_tx(&bar.v_full[vslot], C::TILEB);
      tma_load_5d(sV + vslot * C::TILEB, &mv, &bar.v_full[vslot], 0, cv.h, cv.t * kKT, cv.n, cv.b);
      cursor_next_tile(cv); ++gv;
      if (++vslot == kVS) vslot = 0;
    }
  };
  auto pump_b = [&]() {
    if (BM != kTma) return;
    while (cb_next < g_total * (kKT / kBCW)) {
      if (puse > 0 && !mbar_test(&bar.b_empty[pslot], (puse - 1) & 1)) break;
      mbar_expect_tx(&bar.b_full[pslot], kBChunkBytes);
      tma_load_4d(sB + pslot * kBChunkBytes, &mb, &bar.b_full[pslot], cbias.t * kKT + cb_quarter * kBCW, cbias.qt * kQT,
                  cbias.h, cbias.b * p.bias_b_mul);
      ++cb_next;
      if (++cb_quarter == kKT / kBCW) { cb_quarter = 0; cursor_next_tile(cbias); }
      if (++pslot == kBC) { pslot = 0; ++puse; }
    }
  };
  // staged bias: my warp's next chunk, four lanes a row; always one cp.async group
  constexpr int kWCols = 64 / sizeof(TB), kWChunks = kKT / kWCols;      // per chunk / chunks per key tile
  uint8_t* const ring = sB + (warp & 3) * (kWC * kWChunkBytes);
  auto stage_bias = [&]() {
    if (cb_next < g_total * kWChunks) {
      const int col = cbias.t * kKT + cb_quarter * kWCols + (lane & 3) * (16 / (int)sizeof(TB));
      int bytes = (p.L - col) * (int)sizeof(TB);
      bytes = bytes < 0 ? 0 : bytes > 16 ? 16 : bytes;                  // zeros beyond the last key
      const TB* base = static_cast<const TB*>(p.bias) + cbias.b * p.bs[0] + cbias.h * p.bs[1] + (bytes > 0 ? col : 0);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int rl = k * 8 + (lane >> 2), row = cbias.qt * kQT + (warp & 3) * 32 + rl;
        cp_async16(ring + pslot * kWChunkBytes + swz_offset(rl, lane & 3, 64), base + (int64_t)(row < p.L ? row : p.L - 1) * p.bs[2], bytes);
      }
      ++cb_next;
      if (++cb_quarter == kWChunks) { cb_quarter = 0; cursor_next_tile(cbias); }
      if (++pslot == kWC) pslot = 0;
    }
    cp_async_commit();
  };
  auto issue_s = [&](int g) {     // S(g) = Q K(g)^T
    const uint32_t q_lo = desc_lo(smem_u32(sQ), 16), k_lo = desc_lo(smem_u32(sK + (g % C::KS) * C::TILEB), 16);
#pragma unroll
    for (int ks = 0; ks < DP / 16; ++ks)
      mma_ss_el(tS0, q_lo + ks * 2, desc_hi(C::SBO, C::SW), k_lo + ks * 2, desc_hi(C::SBO, C::SW), id_s, ks > 0);
    tc_commit_el(&bar.s_ready);
  };
  auto issue_pv = [&](int g) {    // O_tile(g) = P V(g)
    const uint32_t v_lo = desc_lo(smem_u32(sV + (g % kVS) * C::TILEB), 16);
#pragma unroll
    for (int ks = 0; ks < kKT / 16; ++ks)
      mma_ts_el(tS0 + 192, tS0 + 128 + ks * 8, v_lo + ks * (16 * C::ROWB / 16), desc_hi(C::SBO, C::SW), id_o, ks > 0);
    tc_commit_el(&bar.pv_done);
  };

  if (g_total > 0) {
    if (officer_kv) { issue_q(); pump_k(0); pump_v(0); }
    if (officer_b) pump_b();
    if (BM == kStaged)
      for (int i = 0; i < kWC; ++i) stage_bias();
  }

  const TB* bias = static_cast<const TB*>(p.bias);
  int prev_bn = -1;
  int t = 0, item_local = 0;
  int b = 0, n = 0, h = 0, i = 0;
  bool row_ok = false;
  const TB* brow = bias;
  float m = -INFINITY, l = 0.f, corr_prev = 0.f;
  float acc[DP];
  uint32_t bslot = 0, bphase = 0;          // bias chunk ring position of the consumer

  auto fold = [&]() {   // acc = acc * corr_prev + O_tile
    tc_fence_after();
#pragma unroll
    for (int cb = 0; cb < DP / 32; ++cb) {
      uint32_t o32[32];
      tmem_ld32(tO + cb * 32, o32);
      tmem_ld_wait();
#pragma unroll
      for (int d = 0; d < 32; ++d) acc[cb * 32 + d] = fmaf(acc[cb * 32 + d], corr_prev, __uint_as_float(o32[d]));
    }
  };

  for (int g = 0; g < g_total; ++g) {
    if (t == 0) {
      // ---------------------------------------------------------------- new item
      const int it = item_begin + item_local;
      const int qt = it % p.n_qt, bn = it / per_bn;
      h = (it / p.n_qt) % p.H; n = bn % p.N; b = bn / p.N;
      i = qt * kQT + r;
      row_ok = i < p.L;
      brow = bias + b * p.bs[0] + h * p.bs[1] + (int64_t)(row_ok ? i : p.L - 1) * p.bs[2];
      if (bn != prev_bn) {
        // additive key terms of row (b, n) in the base-2 domain; columns beyond L are -inf
        named_sync(1 + s, 128);
        for (int j = wg_tid; j < p.lpad; j += 128) {
          float v = -INFINITY;
          if (j < p.L) {
            const int64_t mi = b * p.ms[0] + n * p.ms[1] + j * p.ms[2];
            v = p.mask_dtype == MF_U8 ? (static_cast<const uint8_t*>(p.mask)[mi] ? 0.f : -FLT_MAX)
                                      : load_rt(p.mask, mi, p.mask_dtype) * kLog2e;
          }
          mask2[j] = v;
        }
        named_sync(1 + s, 128);
        prev_bn = bn;
      }
      m = -INFINITY; l = 0.f; corr_prev = 0.f;
#pragma unroll
      for (int d = 0; d < DP; ++d) acc[d] = 0.f;
      if (leader) {
        wait_or_flag(&bar.q_full, item_local & 1, abort_flag);
        wait_or_flag(&bar.k_full[g % C::KS], (g / C::KS) & 1, abort_flag);
        tc_fence_after();
        if (!__any_sync(0xffffffffu, *abort_flag)) issue_s(g);
      }
    }
    // ------------------------------------------------------------------ S(g) -> registers
    wait_or_flag(&bar.s_ready, g & 1, abort_flag);
    tc_fence_after();
    uint32_t sr[kKT];
    {
      uint32_t (*s4)[32] = reinterpret_cast<uint32_t (*)[32]>(sr);
#pragma unroll
      for (int c = 0; c < kKT / 32; ++c) tmem_ld32(tS + c * 32, s4[c]);
      tmem_ld_wait();
    }
    tc_fence_before();
    if (named_sync_or(1 + s, 128, *abort_flag)) break;
    if (leader) {
      // the S buffer is free: start the next tile's scores right away
      if (t + 1 < p.n_kt) {
        wait_or_flag(&bar.k_full[(g + 1) % C::KS], ((g + 1) / C::KS) & 1, abort_flag);
        tc_fence_after();
        if (!__any_sync(0xffffffffu, *abort_flag)) issue_s(g + 1);
      }
    }
    if (officer_kv) {
      if (t + 1 == p.n_kt && item_local + 1 < n_my) issue_q();   // every S of this item is complete: Q is free
      pump_k(g + 1);
    }
    if (officer_b) pump_b();
    // ------------------------------------------------------------------ pass 1: base-2 logits, row max
    const int j0 = t * kKT;
    constexpr int kW = BM == kStaged ? kWCols : 32;      // columns at a time
    float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int cb = 0; cb < kKT / kW; ++cb) {
      float bv[kW];
      if constexpr (BM == kTma) {
        // a chunk holds 64 columns: two passes of this loop read its two halves
        if ((cb & 1) == 0) wait_or_flag(&bar.b_full[bslot], bphase, abort_flag);
        const uint8_t* chunk = sB + bslot * kBChunkBytes;
#pragma unroll
        for (int pc = 0; pc < 4; ++pc) {
          const uint4 x = *reinterpret_cast<const uint4*>(chunk + swz_offset(r, (cb & 1) * 4 + pc, 128));
          float2 a = Pack2<TB>::unpack(x.x), b2 = Pack2<TB>::unpack(x.y), c2 = Pack2<TB>::unpack(x.z), d2 = Pack2<TB>::unpack(x.w);
          bv[8 * pc] = a.x; bv[8 * pc + 1] = a.y; bv[8 * pc + 2] = b2.x; bv[8 * pc + 3] = b2.y;
          bv[8 * pc + 4] = c2.x; bv[8 * pc + 5] = c2.y; bv[8 * pc + 6] = d2.x; bv[8 * pc + 7] = d2.y;
        }
        if (cb & 1) {
          mbar_arrive(&bar.b_empty[bslot]);
          if (++bslot == kBC) { bslot = 0; bphase ^= 1; }
        }
      } else if constexpr (BM == kStaged) {
        cp_async_wait<kWC - 1>();
        __syncwarp();
#pragma unroll
        for (int pc = 0; pc < 4; ++pc) {
          const uint4 x = *reinterpret_cast<const uint4*>(ring + bslot * kWChunkBytes + swz_offset(lane, pc, 64));
          const uint32_t u[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if constexpr (sizeof(TB) == 4) {
              bv[pc * 4 + e] = __uint_as_float(u[e]);
            } else {
              const float2 v = Pack2<TB>::unpack(u[e]);
              bv[pc * 8 + e * 2] = v.x; bv[pc * 8 + e * 2 + 1] = v.y;
            }
          }
        }
        __syncwarp();                         // everybody has read: the slot may be filled again
        if (++bslot == kWC) bslot = 0;
        stage_bias();
      } else {
        if (p.bias_fast && (j0 + kKT <= p.L)) load_bias32_fast<TB>(brow + j0 + cb * 32, bv);
        else load_bias32_slow<TB>(brow, p.bs[3], j0 + cb * 32, p.L, bv);
      }
#pragma unroll
      for (int q4 = 0; q4 < kW / 4; ++q4) {
        const float4 mk4 = *reinterpret_cast<const float4*>(mask2 + j0 + cb * kW + q4 * 4);
        const float mk[4] = {mk4.x, mk4.y, mk4.z, mk4.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int jj = cb * kW + q4 * 4 + e;
          const float v = fmaf(__uint_as_float(sr[jj]), p.c1, fmaf(bv[q4 * 4 + e], kLog2e, mk[e]));
          sr[jj] = __float_as_uint(v);
          mx4[e] = fmaxf(mx4[e], v);
        }
      }
    }
    const float m_new = fmaxf(fmaxf(m, fmaxf(mx4[0], mx4[1])), fmaxf(mx4[2], mx4[3]));
    const float m_ref = m_new == -INFINITY ? 0.f : m_new;      // every logit so far is -inf (a mask or bias of -inf): no NaN yet
    const float corr = ex2f(m - m_ref);
    // ------------------------------------------------------------------ fold O_tile(g-1), then P(g)
    if (t > 0) {
      wait_or_flag(&bar.pv_done, (g - 1) & 1, abort_flag);
      fold();
    }
    float rs4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int cb = 0; cb < kKT / 64; ++cb) {
      uint32_t pk[32];
#pragma unroll
      for (int jj = 0; jj < 32; ++jj) {
        const float p0 = ex2f(__uint_as_float(sr[cb * 64 + 2 * jj]) - m_ref);
        const float p1 = ex2f(__uint_as_float(sr[cb * 64 + 2 * jj + 1]) - m_ref);
        rs4[jj & 3] += p0 + p1;
        pk[jj] = Pack2<T>::pack(p0, p1);
      }
      tmem_st32(tP + cb * 32, pk);
    }
    l = fmaf(l, corr, (rs4[0] + rs4[1]) + (rs4[2] + rs4[3]));
    m = m_new;
    corr_prev = corr;
    tmem_st_wait();
    tc_fence_before();
    if (named_sync_or(1 + s, 128, *abort_flag)) break;
    if (leader) {
      wait_or_flag(&bar.v_full[g % kVS], (g / kVS) & 1, abort_flag);
      tc_fence_after();
      if (!__any_sync(0xffffffffu, *abort_flag)) issue_pv(g);
    }
    if (officer_kv) pump_v(g);          // P V(g-1) and earlier are known complete
    if (officer_b) pump_b();
    if (++t == p.n_kt) {
      // ---------------------------------------------------------------- item done
      wait_or_flag(&bar.pv_done, g & 1, abort_flag);
      fold();
      if (row_ok && !*abort_flag) {
        const float inv = 1.f / l;
        T* orow = static_cast<T*>(p.o) + p.os.at(b, n, i) + h * p.D;
#pragma unroll
        for (int d8 = 0; d8 < DP / 8; ++d8) {
          if (d8 * 8 < p.D) {
            uint4 v;
            v.x = Pack2<T>::pack(acc[d8 * 8] * inv, acc[d8 * 8 + 1] * inv);
            v.y = Pack2<T>::pack(acc[d8 * 8 + 2] * inv, acc[d8 * 8 + 3] * inv);
            v.z = Pack2<T>::pack(acc[d8 * 8 + 4] * inv, acc[d8 * 8 + 5] * inv);
            v.w = Pack2<T>::pack(acc[d8 * 8 + 6] * inv, acc[d8 * 8 + 7] * inv);
            *reinterpret_cast<uint4*>(orow + d8 * 8) = v;
          }
        }
        // a row whose keys are all masked keeps m = -FLT_MAX: its log-sum-exp is stored as -FLT_MAX, the value the
        // backward kernels recognise
        p.lse[(((int64_t)b * p.N + n) * p.H + h) * p.L + i] = m <= -1e38f ? -FLT_MAX : (m + lg2f(l)) * kLn2;
      }
      t = 0;
      ++item_local;
    }
  }
  if (*abort_flag) {
    if (officer_kv) { drain_ring(&bar.q_full, cq.item_local, 1); drain_ring(bar.k_full, gk, C::KS); drain_ring(bar.v_full, gv, kVS); }
    if (BM == kTma && officer_b) drain_ring(bar.b_full, cb_next, kBC);
  }
  if (BM == kStaged) cp_async_wait<0>();

  tc_fence_before();
  __syncthreads();
  if (tid == 0 && abort_s) *reinterpret_cast<volatile int*>(p.status) = 1;
  if (warp == 0) tmem_dealloc(tmem_base_s, 512);
}

template <int DP, typename T, typename TB>
int launch_fwd(const mf_evo_fwd_args& a, const mf_evo_layout& lay, cudaStream_t st) {
  using C = Cfg<DP>;
  constexpr int kKT = C::KT;
  CUtensorMap mq, mk, mv, mb;
  int r;
  if ((r = make_qkv_map(&mq, a.q, a.dtype, a.B, a.N, a.L, a.H, a.D, a.q_strides, DP, kQT))) return r;
  if ((r = make_qkv_map(&mk, a.k, a.dtype, a.B, a.N, a.L, a.H, a.D, a.k_strides, DP, kKT))) return r;
  if ((r = make_qkv_map(&mv, a.v, a.dtype, a.B, a.N, a.L, a.H, a.D, a.v_strides, DP, kKT))) return r;
  FwdP p{};
  p.B = a.B; p.N = a.N; p.L = a.L; p.H = a.H; p.D = a.D;
  p.n_qt = (a.L + kQT - 1) / kQT; p.n_kt = (a.L + kKT - 1) / kKT;
  p.n_items = a.B * a.N * a.H * p.n_qt;
  p.lpad = p.n_kt * kKT;
  p.c1 = kLog2e / sqrtf((float)a.D);
  p.ab_fmt = a.dtype == MF_BF16 ? 1u : 0u;
  p.bias = a.bias; for (int i = 0; i < 4; ++i) p.bs[i] = a.bias_strides[i];
  const size_t bes = sizeof(TB);
  p.bias_fast = a.bias_strides[3] == 1 && (reinterpret_cast<uintptr_t>(a.bias) & 15) == 0 &&
                (a.bias_strides[0] * bes) % 16 == 0 && (a.bias_strides[1] * bes) % 16 == 0 && (a.bias_strides[2] * bes) % 16 == 0;
  p.mask = a.mask; for (int i = 0; i < 3; ++i) p.ms[i] = a.mask_strides[i];
  p.mask_dtype = a.mask_dtype;
  p.o = a.o; p.os = token_strides(lay.o); p.lse = a.lse;
  p.status = status_word();
  MF_REQUIRE(p.status, MF_ERR_CUDA, "could not allocate the device status word");
  MF_REQUIRE(tc_async_status() == 0, MF_ERR_CUDA, "an earlier tensor-core kernel gave up on a bounded wait; results are invalid");

  // bias through shared memory: unit inner stride, 16-byte aligned rows, and room; by TMA for a 16-bit dtype and DP = 32
  constexpr int kModeFast = DP == 32 && sizeof(TB) == 2 ? kTma : kStaged;
  const auto smem_of = [&](int mode) { return 1024 + 2 * ((size_t)C::STREAM_BYTES(mode) + sizeof(float) * p.lpad); };
  const bool fast = p.bias_fast && smem_of(kModeFast) <= kSmemLimit;
  mb = mq;
  if (fast && kModeFast == kTma) {
    p.bias_b_mul = a.bias_strides[0] == 0 ? 0 : 1;
    const int64_t dims[4] = {a.L, a.L, a.H, p.bias_b_mul ? a.B : 1};
    const int64_t str[4] = {1, a.bias_strides[2], a.bias_strides[1], a.bias_strides[0]};
    const int box[4] = {kBCW, 128, 1, 1};
    if ((r = make_tiled_map(&mb, a.bias, a.bias_dtype, 4, dims, str, box, kBCW * 2))) return r;
  }
  int grid = sm_count();
  if (grid > p.n_items) grid = p.n_items;
  p.items_per_stream = (p.n_items + 2 * grid - 1) / (2 * grid);
  const size_t smem = smem_of(fast ? kModeFast : kDirect);
  if (fast) {
    constexpr auto kern = evo_fwd_tc_kernel<DP, T, TB, kModeFast>;
    if (int e = opt_in_smem<kern>(smem)) return e;
    kern<<<grid, kThreads, smem, st>>>(mq, mk, mv, mb, p);
  } else {
    constexpr auto kern = evo_fwd_tc_kernel<DP, T, TB, kDirect>;
    if (int e = opt_in_smem<kern>(smem)) return e;
    kern<<<grid, kThreads, smem, st>>>(mq, mk, mv, mb, p);
  }
  MF_LAUNCHED("evo_fwd_tc_kernel");
  return MF_OK;
}

}  // namespace

#define MF_DISPATCH_BIAS(dt, TB, ...)                                         \
  switch (dt) {                                                               \
    case MF_F32: { using TB = float; __VA_ARGS__; } break;                    \
    case MF_BF16: { using TB = __nv_bfloat16; __VA_ARGS__; } break;           \
    case MF_F16: { using TB = __half; __VA_ARGS__; } break;                   \
    default: return fail(MF_ERR_BAD_ARG, "unknown bias dtype %d", (int)(dt)); \
  }

int evo_fwd_tc(const mf_evo_fwd_args& a, const mf_evo_layout& lay, cudaStream_t st) {
  int r = MF_OK;
  if (a.dtype == MF_BF16) {
    MF_DISPATCH_BIAS(a.bias_dtype, TB, {
      r = a.D <= 32 ? launch_fwd<32, __nv_bfloat16, TB>(a, lay, st) : launch_fwd<64, __nv_bfloat16, TB>(a, lay, st);
    });
  } else {
    MF_DISPATCH_BIAS(a.bias_dtype, TB, {
      r = a.D <= 32 ? launch_fwd<32, __half, TB>(a, lay, st) : launch_fwd<64, __half, TB>(a, lay, st);
    });
  }
  return r;
}

}  // namespace mf
