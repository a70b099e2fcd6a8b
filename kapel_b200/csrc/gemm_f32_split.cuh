// The 32-bit product on the tensor cores (gemm_f32_split.cu), for the launcher that chooses (gemm_f32.cu).
#pragma once
#include "common.cuh"

namespace kb {

enum FpWay { FP_BESIDE = 0, FP_WHOLE = 1, FP_APART = 2 };           // how the groups of K are done

bool gemm_f32_pieces_take(int k, const void* a, const void* w);
int gemm_f32_groups(int n, int k, int sms);
int gemm_f32_way(int m, int n, int k, int groups, int sms);
long long gemm_f32_pieces_floats(int m, int k);                    // scratch that the pieces of m rows take
long long gemm_f32_scratch_floats(int m, int n, int k);            // and all that a product takes
int gemm_f32_rows_at_once(int k);                                  // rows a launch takes: their pieces are FP_SCRATCH bytes at most
int launch_f32_pieces(float* c, const float* a, const float* w, int m, int n, int k, int epilogue, float cap, int groups, int way, float* scratch, cudaStream_t s);

}  // namespace kb
