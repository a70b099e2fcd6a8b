// The 32-bit product on the tensor cores (gemm_f32_split.cu), for the launcher that chooses (gemm_f32.cu).
#pragma once
#include "common.cuh"

namespace kb {

bool gemm_f32_pieces_take(int m, int k, const void* a, const void* w);
int gemm_f32_segments(int m, int n, int k);
long long gemm_f32_pieces_floats(int m, int k);                    // scratch that m rows take
int launch_f32_pieces(float* c, const float* a, const float* w, int m, int n, int k, int epilogue, float cap, int segments, float* scratch, cudaStream_t s);

}  // namespace kb
