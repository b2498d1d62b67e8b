// Type conversion of several contiguous arrays in one launch.
//
// Bound: HBM for a large array, one launch for the usual four to six parameter-sized ones.  A block converts one chunk of
// 2048 elements (eight per thread, 16- or 32-byte accesses when both ends are aligned) of one array; the chunks of all
// arrays are numbered through and a block finds its array by comparing its number with at most seven prefix counts.
#include "common.cuh"

namespace mf {
namespace {

constexpr int kChunk = 2048;

struct CastP {
  const void* src[MF_CAST_MAX]; void* dst[MF_CAST_MAX];
  int64_t n[MF_CAST_MAX];
  unsigned first[MF_CAST_MAX + 1];      // number of the first chunk of each array
  int8_t src_dtype[MF_CAST_MAX], dst_dtype[MF_CAST_MAX];
  int n_items;
};

template <typename S, typename D>
__device__ __forceinline__ void cast_chunk(const S* src, D* dst, int64_t left) {
  const int e0 = threadIdx.x * 8;
  if (e0 >= left) return;
  const bool vec = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0 && e0 + 8 <= left;
  if (vec) {
    __align__(16) S in[8];
    __align__(16) D out[8];
#pragma unroll
    for (int i = 0; i < (int)(8 * sizeof(S) / 16); ++i) reinterpret_cast<uint4*>(in)[i] = reinterpret_cast<const uint4*>(src + e0)[i];
#pragma unroll
    for (int i = 0; i < 8; ++i) out[i] = from_f<D>(to_f(in[i]));
#pragma unroll
    for (int i = 0; i < (int)(8 * sizeof(D) / 16); ++i) reinterpret_cast<uint4*>(dst + e0)[i] = reinterpret_cast<const uint4*>(out)[i];
  } else {
    for (int i = e0; i < left && i < e0 + 8; ++i) dst[i] = from_f<D>(to_f(src[i]));
  }
}

template <typename S>
__device__ __forceinline__ void cast_to(const S* src, void* dst, int dst_dtype, int64_t at, int64_t left) {
  switch (dst_dtype) {
    case MF_F32: cast_chunk(src + at, static_cast<float*>(dst) + at, left); break;
    case MF_BF16: cast_chunk(src + at, static_cast<__nv_bfloat16*>(dst) + at, left); break;
    default: cast_chunk(src + at, static_cast<__half*>(dst) + at, left); break;
  }
}

__global__ void __launch_bounds__(256) cast_batch_kernel(const __grid_constant__ CastP p) {
  int k = 0;
  while (k + 1 < p.n_items && blockIdx.x >= p.first[k + 1]) ++k;
  const int64_t at = (int64_t)(blockIdx.x - p.first[k]) * kChunk, left = p.n[k] - at;
  switch (p.src_dtype[k]) {
    case MF_F32: cast_to(static_cast<const float*>(p.src[k]), p.dst[k], p.dst_dtype[k], at, left); break;
    case MF_BF16: cast_to(static_cast<const __nv_bfloat16*>(p.src[k]), p.dst[k], p.dst_dtype[k], at, left); break;
    default: cast_to(static_cast<const __half*>(p.src[k]), p.dst[k], p.dst_dtype[k], at, left); break;
  }
}

}  // namespace

int cast_batch(const mf_cast_item* items, int n_items, cudaStream_t st) {
  CastP p{};
  int64_t blocks = 0;
  for (int k = 0; k < n_items; ++k) {
    const mf_cast_item& it = items[k];
    if (it.n == 0) continue;
    const int j = p.n_items++;
    p.src[j] = it.src; p.dst[j] = it.dst; p.n[j] = it.n;
    p.src_dtype[j] = (int8_t)it.src_dtype; p.dst_dtype[j] = (int8_t)it.dst_dtype;
    p.first[j] = (unsigned)blocks;
    blocks += (it.n + kChunk - 1) / kChunk;
  }
  if (blocks == 0) return MF_OK;
  MF_REQUIRE(blocks <= INT32_MAX, MF_ERR_UNSUPPORTED, "mf_cast_batch: too many elements");
  cast_batch_kernel<<<(unsigned)blocks, 256, 0, st>>>(p);
  MF_LAUNCHED("cast_batch_kernel");
  return MF_OK;
}

}  // namespace mf
