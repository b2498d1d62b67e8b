// Pair-biased masked attention on CUDA cores, fp32 arithmetic throughout.
//
// This family serves fp32 storage (where tensor-core input rounding would break the 1e-4 bound),
// head sizes and strides the tcgen05 kernels do not take, and acts as the on-device cross-check of
// the tensor-core kernels.
//
// All kernels work on tiles of 64 rows x 64 columns of the logits with 256 threads; thread (ty, tx) owns the rows
// ty + 16 a and the columns tx + 16 b (a, b = 0..3).  Operands are staged as fp32 rows of pitch DP + 4 floats, so that the
// 16-byte reads of neighbouring rows touch different banks, and a step of four head columns costs eight of them for 64
// multiply-adds.  Probabilities pass through shared memory to the products that sum over columns.
//
// Bound: FP32 issue where there are enough tiles; at the sizes fp32 is used for (parity runs, tens of tokens) the number of
// tiles.  The backward therefore puts its three kinds of work - dK/dV per key tile, dQ per query tile, d_pair_bias per
// tile of it and range of rows - side by side in ONE launch; each recomputes the logits it needs and none adds into
// another's sums, so every result is a sum in a fixed order.  At [1,64,64,4,32] the backward takes 56 us instead of 472 and the forward 12 instead of 30: one
// warp per query used to walk all N rows for its row of d_pair_bias, on 32 blocks.
#include "common.cuh"

namespace mf {
namespace {

constexpr int kThreads = 256;
constexpr int kTile = 64;
constexpr int kPPitch = kTile + 4;

struct EvoP {
  int B, N, L, H, D;
  int bias_dtype, mask_dtype, dbias_dtype;
  float scale;
  const void *q, *k, *v;
  int64_t qs[5], ks[5], vs[5];
  bool q_vec, k_vec, v_vec, g_vec;       // rows can be read four elements at a time
  const void* mask; int64_t ms[3];
  const void* bias; int64_t bs[4];
  void* o; float* lse;
  // backward
  const void *d_o; const float* delta;
  void *dq, *dk, *dv; void* d_bias;
  TokenStrides os, gs;                   // of o / of dq, dk, dv
  int64_t ds[5];                         // of d_o
  int nt, nsplit;                        // tiles per sequence; ranges of the N rows that d_pair_bias is summed in
  float* part;                           // [nsplit][B][H][L][L] sums of the ranges, or NULL: one block sums all of them
};

// Rows [row0, row0 + 64) x [0, DP) of a [.., L, H, D] operand as fp32, zero outside L and D.
template <typename T, int DP>
__device__ __forceinline__ void load_tile(float* dst, const void* src, const int64_t* s, bool vec, int b, int n, int h, int row0, int L, int D) {
  constexpr int pitch = DP + 4;
  const T* base = static_cast<const T*>(src) + b * s[0] + n * s[1] + h * s[3];
#pragma unroll
  for (int it = 0; it < kTile * DP / 4 / kThreads; ++it) {
    const int idx = it * kThreads + threadIdx.x;
    const int r = idx / (DP / 4), d = (idx - r * (DP / 4)) * 4;
    const int l = row0 + r;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (l < L && d < D) {
      const T* p = base + l * s[2];
      if (vec) {
        __align__(16) T e[4];
        if constexpr (sizeof(T) == 4) *reinterpret_cast<uint4*>(e) = __ldg(reinterpret_cast<const uint4*>(p + d));
        else *reinterpret_cast<uint2*>(e) = __ldg(reinterpret_cast<const uint2*>(p + d));
        v = make_float4(to_f(e[0]), to_f(e[1]), to_f(e[2]), to_f(e[3]));
      } else {
        v.x = to_f(p[d * s[4]]);
        if (d + 1 < D) v.y = to_f(p[(d + 1) * s[4]]);
        if (d + 2 < D) v.z = to_f(p[(d + 2) * s[4]]);
        if (d + 3 < D) v.w = to_f(p[(d + 3) * s[4]]);
      }
    }
    *reinterpret_cast<float4*>(dst + r * pitch + d) = v;
  }
}

// acc[a][b] += sum_d A[ty + 16 a][d] B[tx + 16 b][d]
template <int DP>
__device__ __forceinline__ void dot_tile(const float* A, const float* B, int ty, int tx, float (&acc)[4][4]) {
  constexpr int pitch = DP + 4;
#pragma unroll 2
  for (int d = 0; d < DP; d += 4) {
    float4 x[4], y[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) x[a] = *reinterpret_cast<const float4*>(A + (ty + 16 * a) * pitch + d);
#pragma unroll
    for (int b = 0; b < 4; ++b) y[b] = *reinterpret_cast<const float4*>(B + (tx + 16 * b) * pitch + d);
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        acc[a][b] = fmaf(x[a].x, y[b].x, acc[a][b]);
        acc[a][b] = fmaf(x[a].y, y[b].y, acc[a][b]);
        acc[a][b] = fmaf(x[a].z, y[b].z, acc[a][b]);
        acc[a][b] = fmaf(x[a].w, y[b].w, acc[a][b]);
      }
  }
}

// acc[a][e] += sum_c P[ty + 16 a][c] V[c][d], the thread's DP / 16 head columns d = tx * DP / 16 + e
template <int DP>
__device__ __forceinline__ void sum_tile(const float* P, const float* V, int ty, int tx, float (&acc)[4][DP / 16]) {
  constexpr int pitch = DP + 4, E = DP / 16;
#pragma unroll 4
  for (int c = 0; c < kTile; c += 4) {
    float4 pr[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) pr[a] = *reinterpret_cast<const float4*>(P + (ty + 16 * a) * kPPitch + c);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float v[E];
      const float* row = V + (c + k) * pitch + tx * E;
      if constexpr (E == 2) { const float2 t = *reinterpret_cast<const float2*>(row); v[0] = t.x; v[1] = t.y; }
      else {
#pragma unroll
        for (int e = 0; e < E; e += 4) {
          const float4 t = *reinterpret_cast<const float4*>(row + e);
          v[e] = t.x; v[e + 1] = t.y; v[e + 2] = t.z; v[e + 3] = t.w;
        }
      }
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const float w = k == 0 ? pr[a].x : k == 1 ? pr[a].y : k == 2 ? pr[a].z : pr[a].w;
#pragma unroll
        for (int e = 0; e < E; ++e) acc[a][e] = fmaf(w, v[e], acc[a][e]);
      }
    }
  }
}

// reductions over the 16 threads that share a row
__device__ __forceinline__ float row_max(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float row_sum(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <typename T, int DP>
__device__ __forceinline__ void store_rows(void* out, const TokenStrides& s, const float (&acc)[4][DP / 16], const float (&f)[4], int b, int n, int h, int row0, int ty, int tx,
                                           const EvoP& p) {
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int l = row0 + ty + 16 * a;
    if (l >= p.L) continue;
    T* row = static_cast<T*>(out) + s.at(b, n, l) + h * p.D;
#pragma unroll
    for (int e = 0; e < DP / 16; ++e) {
      const int d = tx * (DP / 16) + e;
      if (d < p.D) row[d] = from_f<T>(acc[a][e] * f[a]);
    }
  }
}

__device__ __forceinline__ float bias_at(const EvoP& p, int b, int h, int i, int j) {
  return load_rt(p.bias, b * p.bs[0] + h * p.bs[1] + (int64_t)i * p.bs[2] + j * p.bs[3], p.bias_dtype);
}
__device__ __forceinline__ float mask_at(const EvoP& p, int b, int n, int j) {
  return mask_term(p.mask, b * p.ms[0] + n * p.ms[1] + j * p.ms[2], p.mask_dtype);
}

// ------------------------------------------------------------------------------------------
// forward: a block per (b, n, h, 64 queries), online softmax over the key tiles
// ------------------------------------------------------------------------------------------
template <typename T, int DP>
__global__ void __launch_bounds__(kThreads) evo_fwd_simt_kernel(const __grid_constant__ EvoP p) {
  extern __shared__ __align__(16) float smem[];
  constexpr int kOp = kTile * (DP + 4);
  float *Qs = smem, *Ks = Qs + kOp, *Vs = Ks + kOp, *Ps = Vs + kOp;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int h = blockIdx.y, bn = blockIdx.z, b = bn / p.N, n = bn - b * p.N, i0 = blockIdx.x * kTile;
  load_tile<T, DP>(Qs, p.q, p.qs, p.q_vec, b, n, h, i0, p.L, p.D);
  float acc[4][DP / 16], m[4], l[4];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    m[a] = -INFINITY; l[a] = 0.f;
#pragma unroll
    for (int e = 0; e < DP / 16; ++e) acc[a][e] = 0.f;
  }
  for (int j0 = 0; j0 < p.L; j0 += kTile) {
    __syncthreads();
    load_tile<T, DP>(Ks, p.k, p.ks, p.k_vec, b, n, h, j0, p.L, p.D);
    load_tile<T, DP>(Vs, p.v, p.vs, p.v_vec, b, n, h, j0, p.L, p.D);
    float bm[4][4];              // bias + mask of my logits, requested before the products
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int j = j0 + tx + 16 * c;
      const float mt = j < p.L ? mask_at(p, b, n, j) : 0.f;
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const int i = i0 + ty + 16 * a;
        bm[a][c] = j < p.L && i < p.L ? bias_at(p, b, h, i, j) + mt : -INFINITY;
      }
    }
    __syncthreads();
    float s[4][4] = {};
    dot_tile<DP>(Qs, Ks, ty, tx, s);
#pragma unroll
    for (int a = 0; a < 4; ++a) {
#pragma unroll
      for (int c = 0; c < 4; ++c) s[a][c] = fmaf(s[a][c], p.scale, bm[a][c]);
      const float m_new = fmaxf(m[a], row_max(fmaxf(fmaxf(s[a][0], s[a][1]), fmaxf(s[a][2], s[a][3]))));
      const float m_ref = m_new == -INFINITY ? 0.f : m_new;         // a row beyond L: every logit is -inf
      const float corr = expf(m[a] - m_ref);
      float sum = 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float pr = expf(s[a][c] - m_ref);
        sum += pr;
        Ps[(ty + 16 * a) * kPPitch + tx + 16 * c] = pr;
      }
      l[a] = l[a] * corr + row_sum(sum);
      m[a] = m_new;
#pragma unroll
      for (int e = 0; e < DP / 16; ++e) acc[a][e] *= corr;
    }
    __syncwarp();                // a row's probabilities are written and read by the same half warp
    sum_tile<DP>(Ps, Vs, ty, tx, acc);
  }
  float inv[4];
#pragma unroll
  for (int a = 0; a < 4; ++a) inv[a] = 1.f / l[a];
  store_rows<T, DP>(p.o, p.os, acc, inv, b, n, h, i0, ty, tx, p);
  if (tx == 0)
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int i = i0 + ty + 16 * a;
      if (i < p.L) p.lse[(((int64_t)b * p.N + n) * p.H + h) * p.L + i] = m[a] + logf(l[a]);
    }
}

// ------------------------------------------------------------------------------------------
// backward, step 0: delta[b,n,h,i] = sum_d dO * O      (eight threads per (b,n,i,h))
// ------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(kThreads) evo_delta_kernel(const T* __restrict__ o, TokenStrides os, const T* __restrict__ d_o, TokenStrides ds,
                                                             float* __restrict__ delta, int64_t rows, int N, int L, int H, int D) {
  const int64_t row = (int64_t)blockIdx.x * (kThreads / 8) + (threadIdx.x >> 3);
  // row = ((b*N+n)*L + i)*H + h  ->  delta index ((b*N+n)*H + h)*L + i
  const int h = row % H; const int64_t t = row / H; const int i = t % L; const int64_t bn = t / L;
  float s = 0.f;
  if (row < rows) {
    const T *po = o + os.at((int)(bn / N), (int)(bn % N), i) + h * D, *pg = d_o + ds.at((int)(bn / N), (int)(bn % N), i) + h * D;
    for (int d = threadIdx.x & 7; d < D; d += 8) s = fmaf(to_f(po[d]), to_f(pg[d]), s);
  }
#pragma unroll
  for (int k = 4; k > 0; k >>= 1) s += __shfl_xor_sync(0xffffffffu, s, k);
  if (row < rows && (threadIdx.x & 7) == 0) delta[(bn * H + h) * L + i] = s;
}

// P and dS of one logit from its product sums
__device__ __forceinline__ void p_ds(const EvoP& p, float s, float dp, float bias, float mt, float lse, float dl, float& pr, float& ds) {
  // a row whose keys are all masked has lse = -FLT_MAX (log l is absorbed): it is uniform over its L keys
  pr = lse <= -3e38f ? 1.f / p.L : expf(fmaf(s, p.scale, bias + mt) - lse);
  // a masked logit is a constant (masked_fill): no gradient flows into q, k or the bias through it,
  // which only matters for a row whose keys are ALL masked (elsewhere pr is exactly 0)
  ds = mt <= -FLT_MAX ? 0.f : pr * (dp - dl);
}

// dK and dV of 64 keys: rows of the tile are keys, columns queries
template <typename T, int DP>
__device__ __forceinline__ void bwd_dkv(const EvoP& p, float* smem, int b, int n, int h, int j0) {
  constexpr int kOp = kTile * (DP + 4);
  float *Ks = smem, *Vs = Ks + kOp, *Qs = Vs + kOp, *Gs = Qs + kOp, *Ps = Gs + kOp, *Ds = Ps + kTile * kPPitch;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  load_tile<T, DP>(Ks, p.k, p.ks, p.k_vec, b, n, h, j0, p.L, p.D);
  load_tile<T, DP>(Vs, p.v, p.vs, p.v_vec, b, n, h, j0, p.L, p.D);
  float dk[4][DP / 16] = {}, dv[4][DP / 16] = {}, mt[4];
#pragma unroll
  for (int a = 0; a < 4; ++a) mt[a] = j0 + ty + 16 * a < p.L ? mask_at(p, b, n, j0 + ty + 16 * a) : 0.f;
  for (int i0 = 0; i0 < p.L; i0 += kTile) {
    __syncthreads();
    load_tile<T, DP>(Qs, p.q, p.qs, p.q_vec, b, n, h, i0, p.L, p.D);
    load_tile<T, DP>(Gs, p.d_o, p.ds, p.g_vec, b, n, h, i0, p.L, p.D);
    float bias[4][4], lse[4], dl[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int i = i0 + tx + 16 * c;
      const int64_t srow = (((int64_t)b * p.N + n) * p.H + h) * p.L + i;
      lse[c] = i < p.L ? p.lse[srow] : 0.f; dl[c] = i < p.L ? p.delta[srow] : 0.f;
#pragma unroll
      for (int a = 0; a < 4; ++a) bias[a][c] = i < p.L && j0 + ty + 16 * a < p.L ? bias_at(p, b, h, i, j0 + ty + 16 * a) : 0.f;
    }
    __syncthreads();
    float s[4][4] = {}, dp[4][4] = {};
    dot_tile<DP>(Ks, Qs, ty, tx, s);
    dot_tile<DP>(Vs, Gs, ty, tx, dp);
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float pr = 0.f, ds = 0.f;
        if (i0 + tx + 16 * c < p.L) p_ds(p, s[a][c], dp[a][c], bias[a][c], mt[a], lse[c], dl[c], pr, ds);
        Ps[(ty + 16 * a) * kPPitch + tx + 16 * c] = pr;
        Ds[(ty + 16 * a) * kPPitch + tx + 16 * c] = ds;
      }
    __syncwarp();
    sum_tile<DP>(Ps, Gs, ty, tx, dv);
    sum_tile<DP>(Ds, Qs, ty, tx, dk);
  }
  const float one[4] = {1.f, 1.f, 1.f, 1.f}, sc[4] = {p.scale, p.scale, p.scale, p.scale};
  store_rows<T, DP>(p.dk, p.gs, dk, sc, b, n, h, j0, ty, tx, p);
  store_rows<T, DP>(p.dv, p.gs, dv, one, b, n, h, j0, ty, tx, p);
}

// S and dP of a (query tile, key tile) pair of row n turned into dS; rows are queries, columns keys
template <typename T, int DP>
__device__ __forceinline__ void ds_tile(const EvoP& p, const float* Qs, const float* Gs, const float* Ks, const float* Vs, int b, int n, int h, int i0, int j0,
                                        int ty, int tx, const float (&bias)[4][4], float (&ds)[4][4]) {
  float s[4][4] = {}, dp[4][4] = {}, lse[4], dl[4], mt[4];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int i = i0 + ty + 16 * a, j = j0 + tx + 16 * a;
    const int64_t srow = (((int64_t)b * p.N + n) * p.H + h) * p.L + i;
    lse[a] = i < p.L ? p.lse[srow] : 0.f; dl[a] = i < p.L ? p.delta[srow] : 0.f;
    mt[a] = j < p.L ? mask_at(p, b, n, j) : 0.f;
  }
  dot_tile<DP>(Qs, Ks, ty, tx, s);
  dot_tile<DP>(Gs, Vs, ty, tx, dp);
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      float pr;
      ds[a][c] = 0.f;
      if (j0 + tx + 16 * c < p.L && i0 + ty + 16 * a < p.L) p_ds(p, s[a][c], dp[a][c], bias[a][c], mt[c], lse[a], dl[a], pr, ds[a][c]);
    }
}
__device__ __forceinline__ void bias_tile(const EvoP& p, int b, int h, int i0, int j0, int ty, int tx, float (&bias)[4][4]) {
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int i = i0 + ty + 16 * a, j = j0 + tx + 16 * c;
      bias[a][c] = i < p.L && j < p.L ? bias_at(p, b, h, i, j) : 0.f;
    }
}

// dQ of 64 queries
template <typename T, int DP>
__device__ __forceinline__ void bwd_dq(const EvoP& p, float* smem, int b, int n, int h, int i0) {
  constexpr int kOp = kTile * (DP + 4);
  float *Ks = smem, *Vs = Ks + kOp, *Qs = Vs + kOp, *Gs = Qs + kOp, *Ds = Gs + kOp;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  load_tile<T, DP>(Qs, p.q, p.qs, p.q_vec, b, n, h, i0, p.L, p.D);
  load_tile<T, DP>(Gs, p.d_o, p.ds, p.g_vec, b, n, h, i0, p.L, p.D);
  float dq[4][DP / 16] = {};
  for (int j0 = 0; j0 < p.L; j0 += kTile) {
    __syncthreads();
    load_tile<T, DP>(Ks, p.k, p.ks, p.k_vec, b, n, h, j0, p.L, p.D);
    load_tile<T, DP>(Vs, p.v, p.vs, p.v_vec, b, n, h, j0, p.L, p.D);
    float bias[4][4], ds[4][4];
    bias_tile(p, b, h, i0, j0, ty, tx, bias);
    __syncthreads();
    ds_tile<T, DP>(p, Qs, Gs, Ks, Vs, b, n, h, i0, j0, ty, tx, bias, ds);
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int c = 0; c < 4; ++c) Ds[(ty + 16 * a) * kPPitch + tx + 16 * c] = ds[a][c];
    __syncwarp();
    sum_tile<DP>(Ds, Ks, ty, tx, dq);
  }
  const float sc[4] = {p.scale, p.scale, p.scale, p.scale};
  store_rows<T, DP>(p.dq, p.gs, dq, sc, b, n, h, i0, ty, tx, p);
}

// dBias of a 64 x 64 tile: the sum of dS over range `sp` of the N rows (or, without room for partial sums, over all ranges
// one after the other: the same sums in the same order)
template <typename T, int DP>
__device__ __forceinline__ void bwd_dbias(const EvoP& p, float* smem, int b, int h, int i0, int j0, int sp) {
  constexpr int kOp = kTile * (DP + 4);
  float *Ks = smem, *Vs = Ks + kOp, *Qs = Vs + kOp, *Gs = Qs + kOp;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float bias[4][4], total[4][4];
  bias_tile(p, b, h, i0, j0, ty, tx, bias);
  const int sp_end = p.part ? sp + 1 : p.nsplit;
  for (int r = sp; r < sp_end; ++r) {
    const int n0 = (int)((int64_t)r * p.N / p.nsplit), n1 = (int)((int64_t)(r + 1) * p.N / p.nsplit);
    float acc[4][4] = {};
    for (int n = n0; n < n1; ++n) {
      __syncthreads();
      load_tile<T, DP>(Qs, p.q, p.qs, p.q_vec, b, n, h, i0, p.L, p.D);
      load_tile<T, DP>(Gs, p.d_o, p.ds, p.g_vec, b, n, h, i0, p.L, p.D);
      load_tile<T, DP>(Ks, p.k, p.ks, p.k_vec, b, n, h, j0, p.L, p.D);
      load_tile<T, DP>(Vs, p.v, p.vs, p.v_vec, b, n, h, j0, p.L, p.D);
      __syncthreads();
      float ds[4][4];
      ds_tile<T, DP>(p, Qs, Gs, Ks, Vs, b, n, h, i0, j0, ty, tx, bias, ds);
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[a][c] += ds[a][c];
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int c = 0; c < 4; ++c) total[a][c] = r == sp ? acc[a][c] : total[a][c] + acc[a][c];
  }
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int i = i0 + ty + 16 * a, j = j0 + tx + 16 * c;
      if (i >= p.L || j >= p.L) continue;
      const int64_t at = (((int64_t)b * p.H + h) * p.L + i) * p.L + j;
      if (p.part && p.nsplit > 1) p.part[(int64_t)sp * p.B * p.H * p.L * p.L + at] = total[a][c];
      else store_rt(p.d_bias, at, p.dbias_dtype, total[a][c]);
    }
}

// backward, step 1: blocks [0, n_dkv) own key tiles, [n_dkv, 2 n_dkv) query tiles, the rest tiles of d_pair_bias
template <typename T, int DP>
__global__ void __launch_bounds__(kThreads, DP == 32 ? 2 : 1) evo_bwd_simt_kernel(const __grid_constant__ EvoP p, int64_t n_dkv) {
  extern __shared__ __align__(16) float smem[];
  int64_t u = blockIdx.x;
  if (u < 2 * n_dkv) {
    const bool dkv = u < n_dkv;
    if (!dkv) u -= n_dkv;
    const int t = (int)(u % p.nt); u /= p.nt;
    const int h = (int)(u % p.H); const int bn = (int)(u / p.H);
    if (dkv) bwd_dkv<T, DP>(p, smem, bn / p.N, bn % p.N, h, t * kTile);
    else bwd_dq<T, DP>(p, smem, bn / p.N, bn % p.N, h, t * kTile);
    return;
  }
  u -= 2 * n_dkv;
  int sp = 0;
  if (p.part) { sp = (int)(u % p.nsplit); u /= p.nsplit; }
  const int jt = (int)(u % p.nt); u /= p.nt;
  const int it = (int)(u % p.nt); u /= p.nt;
  bwd_dbias<T, DP>(p, smem, (int)(u / p.H), (int)(u % p.H), it * kTile, jt * kTile, sp);
}

// backward, step 2: d_pair_bias = the sums of the ranges, in order
__global__ void __launch_bounds__(kThreads) evo_dbias_sum_kernel(const float* __restrict__ part, void* __restrict__ out, int dtype, int64_t n, int nsplit) {
  const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  float s = part[i];
  for (int k = 1; k < nsplit; ++k) s += part[(int64_t)k * n + i];
  store_rt(out, i, dtype, s);
}

bool rows_vec(const void* p, const int64_t* s, int D, size_t es) {
  return s[4] == 1 && D % 4 == 0 && (reinterpret_cast<uintptr_t>(p) % (4 * es)) == 0 && s[0] % 4 == 0 && s[1] % 4 == 0 && s[2] % 4 == 0 && s[3] % 4 == 0;
}

template <typename A>
void fill_common(EvoP& p, const A& a) {
  p.B = a.B; p.N = a.N; p.L = a.L; p.H = a.H; p.D = a.D;
  p.bias_dtype = a.bias_dtype; p.mask_dtype = a.mask_dtype;
  p.scale = 1.0f / sqrtf((float)a.D);
  p.q = a.q; p.k = a.k; p.v = a.v;
  for (int i = 0; i < 5; ++i) { p.qs[i] = a.q_strides[i]; p.ks[i] = a.k_strides[i]; p.vs[i] = a.v_strides[i]; }
  const size_t es = dtype_size(a.dtype);
  p.q_vec = rows_vec(a.q, p.qs, a.D, es); p.k_vec = rows_vec(a.k, p.ks, a.D, es); p.v_vec = rows_vec(a.v, p.vs, a.D, es);
  p.mask = a.mask; for (int i = 0; i < 3; ++i) p.ms[i] = a.mask_strides[i];
  p.bias = a.bias; for (int i = 0; i < 4; ++i) p.bs[i] = a.bias_strides[i];
  p.nt = (a.L + kTile - 1) / kTile;
}

// Ranges of the N rows that a tile of d_pair_bias is summed in: enough blocks for four on each SM, at least two
// rows each (a block of one row would write its tile for less work than reading it back costs).
int bias_ranges(int B, int N, int L, int H) {
  const int64_t nt = (L + kTile - 1) / kTile, tiles = (int64_t)B * H * nt * nt;
  int64_t r = (4 * tcx::sm_count() + tiles - 1) / tiles;
  if (r > (N + 1) / 2) r = (N + 1) / 2;
  return (int)(r < 1 ? 1 : r);
}
size_t delta_bytes(const mf_evo_bwd_args& a) { return align_up(sizeof(float) * (size_t)a.B * a.N * a.H * a.L, 256); }

}  // namespace

#define MF_DISPATCH_DP(D, DP, ...)                             \
  if ((D) <= 32) { constexpr int DP = 32; __VA_ARGS__; }       \
  else if ((D) <= 64) { constexpr int DP = 64; __VA_ARGS__; }  \
  else if ((D) <= 128) { constexpr int DP = 128; __VA_ARGS__; } \
  else return fail(MF_ERR_UNSUPPORTED, "head size %d > 128 is not supported", (D));

int evo_fwd_simt(const mf_evo_fwd_args& a, const mf_evo_layout& lay, cudaStream_t st) {
  EvoP p{};
  fill_common(p, a);
  p.o = a.o; p.os = token_strides(lay.o); p.lse = a.lse;
  MF_DISPATCH_FLOAT(a.dtype, T, MF_DISPATCH_DP(a.D, DP, {
    constexpr size_t smem = sizeof(float) * (3 * kTile * (DP + 4) + kTile * kPPitch);
    constexpr auto kern = evo_fwd_simt_kernel<T, DP>;
    if (int e = opt_in_smem<kern>(smem)) return e;
    kern<<<dim3(p.nt, a.H, a.B * a.N), kThreads, smem, st>>>(p);
    MF_LAUNCHED("evo_fwd_simt_kernel");
  }));
  return MF_OK;
}

size_t evo_bwd_simt_workspace(const mf_evo_bwd_args& a) {
  const int r = bias_ranges(a.B, a.N, a.L, a.H);
  return delta_bytes(a) + (r > 1 ? align_up(sizeof(float) * (size_t)r * a.B * a.H * a.L * a.L, 256) : 0);
}

// partials: the workspace has room for the sums of the row ranges behind delta
static int bwd_simt(const mf_evo_bwd_args& a, const mf_evo_layout& lay, bool partials, cudaStream_t st) {
  EvoP p{};
  fill_common(p, a);
  p.lse = const_cast<float*>(a.lse);
  float* delta = static_cast<float*>(a.workspace);
  p.d_o = a.d_o; p.delta = delta;
  p.dq = a.dq; p.dk = a.dk; p.dv = a.dv; p.d_bias = a.d_bias; p.dbias_dtype = a.dbias_dtype;
  p.gs = token_strides(lay.d_qkv);
  p.ds[0] = lay.d_o[0]; p.ds[1] = lay.d_o[1]; p.ds[2] = lay.d_o[2]; p.ds[3] = a.D; p.ds[4] = 1;
  p.g_vec = rows_vec(a.d_o, p.ds, a.D, dtype_size(a.dtype));
  p.nsplit = bias_ranges(a.B, a.N, a.L, a.H);
  p.part = partials ? delta + delta_bytes(a) / sizeof(float) : nullptr;
  MF_DISPATCH_FLOAT(a.dtype, T, {
    const int64_t rows = (int64_t)a.B * a.N * a.L * a.H;
    evo_delta_kernel<T><<<(unsigned)((rows + kThreads / 8 - 1) / (kThreads / 8)), kThreads, 0, st>>>(
        static_cast<const T*>(a.o), token_strides(lay.o), static_cast<const T*>(a.d_o), token_strides(lay.d_o), delta, rows, a.N, a.L, a.H, a.D);
    MF_LAUNCHED("evo_delta_kernel");
    MF_DISPATCH_DP(a.D, DP, {
      constexpr size_t smem = sizeof(float) * (4 * kTile * (DP + 4) + 2 * kTile * kPPitch);
      constexpr auto kern = evo_bwd_simt_kernel<T, DP>;
      if (int e = opt_in_smem<kern>(smem)) return e;
      const int64_t n_dkv = (int64_t)a.B * a.N * a.H * p.nt;
      const int64_t blocks = 2 * n_dkv + (int64_t)a.B * a.H * p.nt * p.nt * (partials ? p.nsplit : 1);
      MF_REQUIRE(blocks <= INT32_MAX, MF_ERR_UNSUPPORTED, "too many tiles for the CUDA-core backward");
      kern<<<(unsigned)blocks, kThreads, smem, st>>>(p, n_dkv);
      MF_LAUNCHED("evo_bwd_simt_kernel");
    });
  });
  if (partials && p.nsplit > 1) {
    const int64_t n = (int64_t)a.B * a.H * a.L * a.L;
    evo_dbias_sum_kernel<<<(unsigned)((n + kThreads - 1) / kThreads), kThreads, 0, st>>>(p.part, a.d_bias, a.dbias_dtype, n, p.nsplit);
    MF_LAUNCHED("evo_dbias_sum_kernel");
  }
  return MF_OK;
}

int evo_bwd_simt(const mf_evo_bwd_args& a, const mf_evo_layout& lay, cudaStream_t st) { return bwd_simt(a, lay, true, st); }

// ---- backward without any allocation ------------------------------------------------------------------
// Scratch for the variant below: the per-query delta = rowsum(dO * O) values, B*N*H*L floats.  The array is part
// of the library image, so every GPU that loads the library holds these 4 MiB until the process exits.
constexpr size_t kNoAllocDeltaFloats = size_t(1) << 20;
static __device__ __align__(256) float g_noalloc_delta[kNoAllocDeltaFloats];

size_t evo_bwd_noalloc_max_rows() { return kNoAllocDeltaFloats; }

int evo_bwd_simt_noalloc(const mf_evo_bwd_args& a, const mf_evo_layout& lay, cudaStream_t st) {
  const size_t need = (size_t)a.B * a.N * a.H * a.L;
  MF_REQUIRE(need <= kNoAllocDeltaFloats, MF_ERR_UNSUPPORTED,
             "mf_evo_bwd_noalloc: B*N*H*L = %zu query rows exceed the built-in scratch of %zu rows; use mf_evo_bwd with a workspace",
             need, kNoAllocDeltaFloats);
  // In host code `g_noalloc_delta` is only a handle of the device array, not its address: the address is asked
  // for once per device (with that device current) and remembered.
  static float* dev_ptr[64] = {};
  int dev = 0;
  MF_CUDA(cudaGetDevice(&dev));
  MF_REQUIRE(dev >= 0 && dev < 64, MF_ERR_UNSUPPORTED, "device ordinal %d out of range", dev);
  float* scratch = __atomic_load_n(&dev_ptr[dev], __ATOMIC_ACQUIRE);
  if (!scratch) {
    MF_CUDA(cudaGetSymbolAddress(reinterpret_cast<void**>(&scratch), g_noalloc_delta));
    MF_REQUIRE(scratch != nullptr, MF_ERR_CUDA, "cudaGetSymbolAddress returned a null scratch address");
    __atomic_store_n(&dev_ptr[dev], scratch, __ATOMIC_RELEASE);
  }
  mf_evo_bwd_args b = a;
  b.workspace = scratch;
  b.workspace_bytes = kNoAllocDeltaFloats * sizeof(float);
  return bwd_simt(b, lay, false, st);     // delta is fully rewritten for the B*N*H*L rows in use: nothing to clear
}

}  // namespace mf
