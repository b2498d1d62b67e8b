// Element-wise pieces between the fused operators of a Pairformer block: the output gate of an attention and the re-layout of
// projected pair-bias rows.  Each direction of each is one pass over memory; torch's own kernels took six (sigmoid, two
// products, their gradients, packing copies of the strided gate) and three (slice, permute, zero-filled padding).
//
// Bound: HBM.  [768 * 768, 128] bf16: gate forward 3 x 151 MB in 89 us, backward 5 x 151 MB in 120 us.
#include <type_traits>

#include "common.cuh"

namespace mf {
namespace {

// Every step is rounded to T, as it is where each is an operation on tensors of its own: the values do not depend on which
// form a caller uses.
template <typename T> __device__ __forceinline__ float round_to(float v) { return to_f(from_f<T>(v)); }
template <typename T> __device__ __forceinline__ float sigmoid_(T x) { return round_to<T>(1.f / (1.f + expf(-to_f(x)))); }

template <typename T> struct Vec8 { __align__(16) T e[8]; };
template <typename T> __device__ __forceinline__ Vec8<T> ld8(const T* p) {
  Vec8<T> v;
#pragma unroll
  for (int i = 0; i < (int)sizeof(T) / 2; ++i) reinterpret_cast<uint4*>(v.e)[i] = __ldg(reinterpret_cast<const uint4*>(p) + i);
  return v;
}
template <typename T> __device__ __forceinline__ void st8(T* p, const Vec8<T>& v) {
#pragma unroll
  for (int i = 0; i < (int)sizeof(T) / 2; ++i) reinterpret_cast<uint4*>(p)[i] = reinterpret_cast<const uint4*>(v.e)[i];
}

// out[r, c] = o[r, c] * sigmoid(g[r * gs + c]); eight columns per thread
template <typename T>
__global__ void __launch_bounds__(256) gate_fwd_kernel(const T* __restrict__ o, const T* __restrict__ g, int64_t gs, T* __restrict__ out, int64_t n8, int c8) {
  const int64_t q = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (q >= n8) return;
  const int64_t r = q / c8;
  const int c = (int)(q - r * c8) * 8;
  const Vec8<T> a = ld8(o + q * 8), b = ld8(g + r * gs + c);
  Vec8<T> y;
#pragma unroll
  for (int i = 0; i < 8; ++i) y.e[i] = from_f<T>(to_f(a.e[i]) * sigmoid_<T>(b.e[i]));
  st8(out + q * 8, y);
}

// d_o = d * s, d_g = (d * o) * (1 - s) * s with s = sigmoid(g); d_g has the row stride of g's gradient array
template <typename T>
__global__ void __launch_bounds__(256) gate_bwd_kernel(const T* __restrict__ d, const T* __restrict__ o, const T* __restrict__ g, int64_t gs, T* __restrict__ d_o,
                                                       T* __restrict__ d_g, int64_t dgs, int64_t n8, int c8) {
  const int64_t q = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (q >= n8) return;
  const int64_t r = q / c8;
  const int c = (int)(q - r * c8) * 8;
  const Vec8<T> dv = ld8(d + q * 8), a = ld8(o + q * 8), b = ld8(g + r * gs + c);
  Vec8<T> x, y;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float s = sigmoid_<T>(b.e[i]), t = round_to<T>(to_f(dv.e[i]) * to_f(a.e[i]));
    x.e[i] = from_f<T>(to_f(dv.e[i]) * s);
    y.e[i] = from_f<T>(round_to<T>(t * round_to<T>(1.f - s)) * s);
  }
  st8(d_o + q * 8, x);
  st8(d_g + r * dgs + c, y);
}

// rows [L * L, np] <-> planes [H, L, L] (H <= np) in 32 x 32 tiles through shared memory, so that both sides are touched in
// whole lines; `swap`: plane element (i, j) belongs to row j * L + i.  To rows: columns H .. np - 1 become zero.
// VEC: rows of whole 16-byte pieces of 16-bit values are moved a piece at a time.  (A value at a time, with three divisions
// each: 28 us for [768, 768, 8] and four heads, 8 to planes and 16 to rows now; the bytes take 2.)
// A block takes a group of up to 32 columns, all of a projection but the widest: what the tile has room for in fp32.
constexpr int kHeadGroup = 32;
template <typename T, bool TO_ROWS, bool VEC>
__global__ void __launch_bounds__(256) bias_layout_kernel(T* __restrict__ rows, T* __restrict__ planes, int L, int np, int all_heads, bool swap) {
  extern __shared__ __align__(16) uint8_t raw[];
  const int first = blockIdx.z * kHeadGroup;
  const int cols = min(np - first, kHeadGroup), H = max(min(all_heads - first, kHeadGroup), 0);      // of my group
  rows += first;
  planes += (int64_t)first * L * L;
  T* tile = reinterpret_cast<T*>(raw);              // [H][32][33], plane order
  const int i0 = blockIdx.y * 32, j0 = blockIdx.x * 32;      // plane coordinates
  auto move_rows = [&] {
    if constexpr (VEC) {
      for (int e = threadIdx.x; e < 32 * 32; e += 256) {
        const int c = e % 32, r = e / 32, i = swap ? c : r, j = swap ? r : c;
        if (i0 + i >= L || j0 + j >= L) continue;
        uint4* p = reinterpret_cast<uint4*>(rows + ((int64_t)(swap ? j0 + j : i0 + i) * L + (swap ? i0 + i : j0 + j)) * np);
        for (int h0 = 0; h0 < cols; h0 += 8) {
          Vec8<T> v;
          if (!TO_ROWS) *reinterpret_cast<uint4*>(v.e) = p[h0 / 8];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            if (TO_ROWS) v.e[k] = h0 + k < H ? tile[((h0 + k) * 32 + i) * 33 + j] : from_f<T>(0.f);
            else if (h0 + k < H) tile[((h0 + k) * 32 + i) * 33 + j] = v.e[k];
          }
          if (TO_ROWS) p[h0 / 8] = *reinterpret_cast<const uint4*>(v.e);
        }
      }
      return;
    }
    for (int e = threadIdx.x; e < 32 * 32 * cols; e += 256) {
      const int h = e % cols, c = e / cols % 32, r = e / cols / 32;      // row block r, column c of it, in the order of memory
      const int i = swap ? c : r, j = swap ? r : c;
      if (i0 + i >= L || j0 + j >= L) continue;
      T* p = rows + ((int64_t)(swap ? j0 + j : i0 + i) * L + (swap ? i0 + i : j0 + j)) * np + h;
      if (TO_ROWS) *p = h < H ? tile[(h * 32 + i) * 33 + j] : from_f<T>(0.f);
      else if (h < H) tile[(h * 32 + i) * 33 + j] = *p;
    }
  };
  auto move_planes = [&] {
    for (int e = threadIdx.x; e < 32 * 32 * H; e += 256) {
      const int j = e % 32, i = e / 32 % 32, h = e / 1024;
      if (i0 + i >= L || j0 + j >= L) continue;
      T* p = planes + ((int64_t)h * L + i0 + i) * L + j0 + j;
      if (TO_ROWS) tile[(h * 32 + i) * 33 + j] = *p;
      else *p = tile[(h * 32 + i) * 33 + j];
    }
  };
  if (TO_ROWS) move_planes(); else move_rows();
  __syncthreads();
  if (TO_ROWS) move_rows(); else move_planes();
}

bool aligned16(std::initializer_list<const void*> ps) {
  for (const void* p : ps)
    if (reinterpret_cast<uintptr_t>(p) & 15) return false;
  return true;
}

}  // namespace

int gate_fwd(const void* o, const void* g, int64_t gs, void* out, int64_t rows, int cols, int dtype, cudaStream_t st) {
  MF_REQUIRE(cols % 8 == 0 && gs % 8 == 0 && aligned16({o, g, out}), MF_ERR_ALIGNMENT, "gate: rows must be multiples of 8 elements on 16-byte boundaries");
  const int64_t n8 = rows * (cols / 8);
  if (n8 == 0) return MF_OK;
  MF_DISPATCH_FLOAT(dtype, T, {
    gate_fwd_kernel<T><<<(unsigned)((n8 + 255) / 256), 256, 0, st>>>(static_cast<const T*>(o), static_cast<const T*>(g), gs, static_cast<T*>(out), n8, cols / 8);
    MF_LAUNCHED("gate_fwd_kernel");
  });
  return MF_OK;
}

int gate_bwd(const void* d, const void* o, const void* g, int64_t gs, void* d_o, void* d_g, int64_t dgs, int64_t rows, int cols, int dtype, cudaStream_t st) {
  MF_REQUIRE(cols % 8 == 0 && gs % 8 == 0 && dgs % 8 == 0 && aligned16({d, o, g, d_o, d_g}), MF_ERR_ALIGNMENT,
             "gate: rows must be multiples of 8 elements on 16-byte boundaries");
  const int64_t n8 = rows * (cols / 8);
  if (n8 == 0) return MF_OK;
  MF_DISPATCH_FLOAT(dtype, T, {
    gate_bwd_kernel<T><<<(unsigned)((n8 + 255) / 256), 256, 0, st>>>(static_cast<const T*>(d), static_cast<const T*>(o), static_cast<const T*>(g), gs,
                                                                     static_cast<T*>(d_o), static_cast<T*>(d_g), dgs, n8, cols / 8);
    MF_LAUNCHED("gate_bwd_kernel");
  });
  return MF_OK;
}

int bias_layout(void* rows, void* planes, int L, int np, int H, bool swap, bool to_rows, int dtype, cudaStream_t st) {
  MF_REQUIRE(H <= np, MF_ERR_UNSUPPORTED, "pair-bias rows of %d columns for %d heads", np, H);
  const dim3 grid((L + 31) / 32, (L + 31) / 32, (np + kHeadGroup - 1) / kHeadGroup);
  MF_DISPATCH_FLOAT(dtype, T, {
    const size_t smem = sizeof(T) * (size_t)(H < kHeadGroup ? H : kHeadGroup) * 32 * 33;
    auto launch = [&](auto to, auto vec) -> int {
      constexpr auto kern = bias_layout_kernel<T, decltype(to)::value, decltype(vec)::value>;
      if (int e = opt_in_smem<kern>(smem)) return e;
      kern<<<grid, 256, smem, st>>>(static_cast<T*>(rows), static_cast<T*>(planes), L, np, H, swap);
      return MF_OK;
    };
    using Yes = std::true_type; using No = std::false_type;
    constexpr bool can = sizeof(T) == 2;
    const bool vec = can && np % 8 == 0 && aligned16({rows});
    using Vec = std::bool_constant<can>;
    if (int e = vec ? (to_rows ? launch(Yes{}, Vec{}) : launch(No{}, Vec{})) : (to_rows ? launch(Yes{}, No{}) : launch(No{}, No{}))) return e;
    MF_LAUNCHED("bias_layout_kernel");
  });
  return MF_OK;
}

}  // namespace mf
