// Interfaces of the tensor-core pieces that backward passes are composed of.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace mf {

// C[M, N] = sum_r A(m, r) B(n, r), fp32 accumulation, 16-bit operands of one dtype.
//   a_mn = 0: A stored [M, R] row-major;  a_mn = 1: stored [R, M].   Same for B with N.
//   out_kind 0: C stored in the operand dtype; 1: fp32; 2: fp32 with the reduction split over CTAs and summed by
//   TMA add-reductions (C is zeroed first unless `accumulate` is set - a caller that feeds the reduction in several row
//   ranges; summation order, and so the last bits, vary from run to run).
struct GemmTcArgs {
  const void* a; const void* b; void* c;
  int64_t M, N, R;
  int dtype, a_mn, b_mn, out_kind;
  int accumulate = 0;
  // A = LayerNorm of the array given (a_mn = 1: its rows are the reduction index), from saved row statistics; the normalised
  // matrix is formed in shared memory, rounded to the operand dtype, and never stored.
  const float *ln_mean = nullptr, *ln_rstd = nullptr;
  const void *ln_gain = nullptr, *ln_shift = nullptr;
  // b_mn = 1: B is stored in panels of 64 columns, [panel][R][64], so that every box of 64 rows is one run of 8 KB
  int b_panels = 0;
};
bool gemm_tc_ok(const GemmTcArgs& g);
int gemm_tc(const GemmTcArgs& g, cudaStream_t st);

// One pass over dy of the LayernormLinear backward (lnl_bwd_tc.cu): dx, and per block the column sums
// part [blocks][K] (gain gradient) and, with db_part, [blocks][N] (bias gradient).
struct LnlBwdRowsArgs {
  int64_t M; int K, N, dtype;
  const void *x, *gamma, *w, *dy;
  const float *mean, *rstd;
  const void *add1, *add2;   // NULL, or added to dx in this order, each sum rounded
  void* dx;
  float *part, *db_part;
};
bool lnl_bwd_rows_tc_ok(int64_t M, int K, int N);
int lnl_bwd_rows_tc_blocks(int64_t M);
int lnl_bwd_rows_tc(const LnlBwdRowsArgs& a, cudaStream_t st);

}  // namespace mf
