// fp32 products of many rows: the tensor-core form (csrc/gemm_f32_tc.cu) behind b2_gemm_f32 (csrc/gemm_f32.cu).
#pragma once
#include "mixers.cuh"

// rows of both operands on 16-byte boundaries; t_tile a multiple of 16 up to 128; splits as b2_gemm_f32_splits counts them
int gemm_f32_tc_launch(const GemmF32Params* p, int t_tile, int splits, cudaStream_t s);
