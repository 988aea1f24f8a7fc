// Host interface of the two-SM GEMM (gemm_pair.cu), called by the launchers of gemm_bf16.cu.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

struct PairPlan { int bn, S; };          // tile width (multiple of 32), pairs that share K (1, 2, 4 or 8)

struct PairOut {
  void* out;
  int64_t ldo;
  int f32;                               // 1: f32 result, 0: bf16
  int glu;                               // 0, or 1 + kind (common.cuh: glu_f)
  float glu_limit, alpha;
  int un_act, un_cols;                   // activation of the first un_cols output features
  const float* bias;
  int w_static;
  int group, pitch;                      // > 0: output columns in groups of `group` (a multiple of 32), `pitch` columns apart; TMA stores only
};

int mary_gemm_pair_plan(int rows_r, int rows_c, int K, bool glu, int max_bn, PairPlan* plan);
// R [rows_r, K] is the row operand (256 rows per tile), C the column operand; swap: R holds the weights and out[j * ldo + i] = R_i . C_j.
int mary_gemm_pair_run(const void* R, const void* C, int rows_r, int rows_c, int K, int64_t ldr, int64_t ldc, bool swap, const PairOut& o,
                       const PairPlan& plan, cudaStream_t stream);
