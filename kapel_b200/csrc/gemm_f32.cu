// C[M,N] = A[M,K] . W[N,K]^T in true 32-bit (the 32-bit path of the whole model; Kapel's f32 tiles: crates/kapel-cuda/src/tile.rs:196). The
// kernels of this file use multiply-adds only; `kb_gemm_f32_fast` hands what is large enough to those of gemm_f32_split.cu, which
// cut every input into pieces that hold it exactly. Of the kernels of this file:
//
// Each output element is one accumulator that takes its K products in ascending k, whatever M
// and N are, whichever kernel computes it and wherever the element lies in its tile: the result for
// a row does not depend on which other rows are in the batch. So K is never split, and what is left to choose
// is how the elements are dealt out.
//
// * More than 16 rows: tiles in shared memory, an outer product of TM x TN elements a thread and k. Shared memory hands a
//   multiprocessor's threads 32 words a clock and the FMA pipe takes 128 products, so (TM + TN) / (TM TN) has to be below a
//   quarter for the pipe to be what bounds it: 8 x 16 where there are tiles enough to fill the GPU that way, smaller ones
//   where there are not. Two neighbouring columns share one `fma.rn.f32x2` (each half is rounded as fmaf rounds it), which
//   leaves issue slots to the loads. The tiles come by asynchronous copies of a word each, turned on their way ([k][row]), a ring of
//   stages ahead of their use: nothing waits for memory, and rows need no alignment. 500 rows by 18,432 x 2,304: 828 us (51 of
//   74 Tflop/s; one 64 x 64 tile of 4 x 4 a thread, for all sizes, took 1,899); by 2,304 x 9,216: 549 us (1,213), bound by the few
//   warps that 144 tiles give a multiprocessor.
// * Up to 16 rows: every weight is read once for at most 16 products, so memory bounds it, or the chain of K
//   dependent multiply-adds where N has few columns: 16 columns a block (2,304 columns are then 144 blocks for 148
//   multiprocessors). Warps of their own copy, so that the others do nothing but multiply. One row by 18,432 x 2,304: 39 us (4.3
//   TB/s; the tile kernel took 331), by 2,304 x 9,216: 33 us (780), where the chain alone is 19.
#include "gemm_f32_split.cuh"

namespace kb {

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 twice(float a) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ f32x2 two(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void fma2(f32x2& c, f32x2 a, f32x2 b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b)); }
__device__ __forceinline__ float2 halves(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
// `bytes` (0, or all) of `from` into shared memory, the rest zeros
__device__ __forceinline__ void copy_word(float* to, const float* from, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_words4(float* to, const float* from, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_end() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

constexpr int F32_BK = 16, F32_STAGES = 4;
template <int BM, int BN> constexpr int f32_smem() { return F32_STAGES * F32_BK * (BM + 4 + BN + 4) * (int)sizeof(float); }

// A thread's rows are groups of four, BM / (TM / 4) apart, its columns likewise. A warp copies 8 k of 4 rows at a time: whole
// 32-byte sectors from memory, 32 different banks of the turned tile. epilogue 0: none; 1: cap * tanh(acc / cap)
template <int BM, int BN, int TM, int TN, int EPI>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), TM * TN >= 128 ? 2 : 3)
gemm_f32_kernel(float* __restrict__ c, const float* __restrict__ a, const float* __restrict__ w, int m, int n, int k, float cap) {
    constexpr int THREADS = (BM / TM) * (BN / TN);
    constexpr int LA = BM + 4, LW = BN + 4, STAGE = F32_BK * (LA + LW);
    constexpr int ROWS_AT_ONCE = THREADS / 8;                      // rows all threads copy 8 k of
    static_assert(BM % ROWS_AT_ONCE == 0 && BN % ROWS_AT_ONCE == 0, "whole rounds of copies");
    extern __shared__ __align__(16) float f32_tiles[];             // [stages]: A's tile [k][BM + 4], then W's [k][BN + 4]
    constexpr int TXS = BN / TN;
    const int tid = threadIdx.x, tx = tid % TXS, ty = tid / TXS;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int steps = (k + F32_BK - 1) / F32_BK;
    const int ck = tid & 7, crow = tid >> 3;
    auto fetch = [&](int step) {
        if (step < steps) {
            float* sa = f32_tiles + (step % F32_STAGES) * STAGE;
            float* sw = sa + F32_BK * LA;
#pragma unroll
            for (int half = 0; half < F32_BK / 8; ++half) {
                const int kk = half * 8 + ck, gk = step * F32_BK + kk;
#pragma unroll
                for (int i = 0; i < BM / ROWS_AT_ONCE; ++i) {
                    const int row = crow + i * ROWS_AT_ONCE;
                    const bool there = m0 + row < m && gk < k;
                    copy_word(sa + kk * LA + row, there ? a + (size_t)(m0 + row) * k + gk : a, there ? 4 : 0);
                }
#pragma unroll
                for (int i = 0; i < BN / ROWS_AT_ONCE; ++i) {
                    const int row = crow + i * ROWS_AT_ONCE;
                    const bool there = n0 + row < n && gk < k;
                    copy_word(sw + kk * LW + row, there ? w + (size_t)(n0 + row) * k + gk : w, there ? 4 : 0);
                }
            }
        }
        copies_end();                                              // one group a step, also where nothing is left to copy
    };
#pragma unroll
    for (int st = 0; st < F32_STAGES - 1; ++st) fetch(st);
    f32x2 acc[TM][TN / 2] = {};
    for (int step = 0; step < steps; ++step) {
        copies_wait<F32_STAGES - 2>();
        __syncthreads();                                           // this step's tile is there; the stage read last step is free
        fetch(step + F32_STAGES - 1);
        const float* sa = f32_tiles + (step % F32_STAGES) * STAGE + ty * 4;
        const float* sw = f32_tiles + (step % F32_STAGES) * STAGE + F32_BK * LA + tx * 4;
        // the next k's elements are read while this one's are multiplied
        float4 wf[2][TN / 4], af[2][TM / 4];
        auto fragments = [&](int kk, int which) {
#pragma unroll
            for (int g = 0; g < TN / 4; ++g) wf[which][g] = *reinterpret_cast<const float4*>(sw + kk * LW + g * (BN / (TN / 4)));
#pragma unroll
            for (int g = 0; g < TM / 4; ++g) af[which][g] = *reinterpret_cast<const float4*>(sa + kk * LA + g * (BM / (TM / 4)));
        };
        fragments(0, 0);
#pragma unroll
        for (int kk = 0; kk < F32_BK; ++kk) {
            const int now = kk & 1;
            if (kk + 1 < F32_BK) fragments(kk + 1, now ^ 1);
            f32x2 wv[TN / 2];
#pragma unroll
            for (int g = 0; g < TN / 4; ++g) wv[2 * g] = two(wf[now][g].x, wf[now][g].y), wv[2 * g + 1] = two(wf[now][g].z, wf[now][g].w);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const float4 a4 = af[now][i / 4];
                const f32x2 aa = twice(i % 4 == 0 ? a4.x : i % 4 == 1 ? a4.y : i % 4 == 2 ? a4.z : a4.w);
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], aa, wv[j]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + (i / 4) * (BM / (TM / 4)) + ty * 4 + i % 4;
        if (gm >= m) continue;
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) {
            const int gn = n0 + (j / 2) * (BN / (TN / 4)) + tx * 4 + (j % 2) * 2;
            float2 v = halves(acc[i][j]);
            if (EPI == 1) v.x = cap * tanhf(v.x / cap), v.y = cap * tanhf(v.y / cap);
            if (gn < n) c[(size_t)gm * n + gn] = v.x;
            if (gn + 1 < n) c[(size_t)gm * n + gn + 1] = v.y;
        }
    }
}

// ---------------------------------------------------------------------------------------- up to 16 rows
constexpr int FEW_ROWS = 16, FEW_N = 16, FEW_BK = 128, FEW_LD = FEW_BK + 4, FEW_STAGES = 4, FEW_COPIERS = 128;
template <int ROWS> struct Few {
    static constexpr int R = ROWS >= 8 ? 4 : (ROWS >= 4 ? 2 : 1);                     // rows a working thread has
    static constexpr int WORKERS = (FEW_N * ROWS / R + 31) / 32 * 32;
};

// ROWS rows (a power of two up to 16) x 16 columns a block: a working thread has one column and R rows; the last four warps copy.
// VEC: rows begin at 16-byte boundaries and k is a multiple of 4.
template <int ROWS, int EPI, bool VEC>
__global__ void __launch_bounds__(Few<ROWS>::WORKERS + FEW_COPIERS)
gemm_f32_few_kernel(float* __restrict__ c, const float* __restrict__ a, const float* __restrict__ w, int m, int n, int k, float cap) {
    constexpr int R = Few<ROWS>::R, WORKERS = Few<ROWS>::WORKERS;
    extern __shared__ __align__(16) float few_smem[];
    float* sw = few_smem;                                          // [stages][16][FEW_LD]
    float* sa = few_smem + FEW_STAGES * FEW_N * FEW_LD;            // [stages][ROWS][FEW_LD]
    const int tid = threadIdx.x, n0 = blockIdx.x * FEW_N;
    const int steps = (k + FEW_BK - 1) / FEW_BK;
    const bool copies = tid >= WORKERS;
    auto put = [&](float* to, const float* x, int row, int rows, int k0) {
        if (VEC) {
            const bool there = row < rows && k0 < k;
            copy_words4(to, there ? x + (size_t)row * k + k0 : x, there ? 16 : 0);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const bool there = row < rows && k0 + j < k;
                copy_word(to + j, there ? x + (size_t)row * k + k0 + j : x, there ? 4 : 0);
            }
        }
    };
    auto fetch = [&](int step) {
        if (step < steps) {
            const int buf = step % FEW_STAGES, k0 = step * FEW_BK;
#pragma unroll
            for (int i = 0; i < FEW_N * FEW_BK / 4 / FEW_COPIERS; ++i) {
                const int e = tid - WORKERS + i * FEW_COPIERS, row = e / (FEW_BK / 4), kk = (e % (FEW_BK / 4)) * 4;
                put(sw + (buf * FEW_N + row) * FEW_LD + kk, w, n0 + row, n, k0 + kk);
            }
            for (int e = tid - WORKERS; e < ROWS * FEW_BK / 4; e += FEW_COPIERS) {
                const int row = e / (FEW_BK / 4), kk = (e % (FEW_BK / 4)) * 4;
                put(sa + (buf * ROWS + row) * FEW_LD + kk, a, row, m, k0 + kk);
            }
        }
        copies_end();
    };
    if (copies)
#pragma unroll
        for (int st = 0; st < FEW_STAGES - 1; ++st) fetch(st);
    const int col = tid % FEW_N, r0 = (tid / FEW_N) * R;
    const bool works = !copies && r0 < ROWS;
    float acc[R] = {};
    for (int step = 0; step < steps; ++step) {
        if (copies) copies_wait<FEW_STAGES - 2>();
        __syncthreads();                                           // this step's tile is there; the stage read last step is free
        if (copies) fetch(step + FEW_STAGES - 1);
        if (works) {
            const float* wr = sw + (step % FEW_STAGES * FEW_N + col) * FEW_LD;
            const float* ar = sa + (step % FEW_STAGES * ROWS + r0) * FEW_LD;
            // sixteen k at a time, the next sixteen read while these are multiplied
            float4 wv[2][4], av[2][R][4];
            auto read = [&](int k0, int which) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    wv[which][q] = *reinterpret_cast<const float4*>(wr + k0 + 4 * q);
#pragma unroll
                    for (int i = 0; i < R; ++i) av[which][i][q] = *reinterpret_cast<const float4*>(ar + i * FEW_LD + k0 + 4 * q);
                }
            };
            read(0, 0);
#pragma unroll
            for (int g = 0; g < FEW_BK / 16; ++g) {
                const int now = g & 1;
                if (g + 1 < FEW_BK / 16) read((g + 1) * 16, now ^ 1);
#pragma unroll
                for (int q = 0; q < 4; ++q)
#pragma unroll
                    for (int i = 0; i < R; ++i) {
                        const float4 x = av[now][i][q], v = wv[now][q];
                        acc[i] = fmaf(x.x, v.x, acc[i]);
                        acc[i] = fmaf(x.y, v.y, acc[i]);
                        acc[i] = fmaf(x.z, v.z, acc[i]);
                        acc[i] = fmaf(x.w, v.w, acc[i]);
                    }
            }
        }
    }
    if (!works || n0 + col >= n) return;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        if (r0 + i >= m) continue;
        float v = acc[i];
        if (EPI == 1) v = cap * tanhf(v / cap);
        c[(size_t)(r0 + i) * n + n0 + col] = v;
    }
}

template <int ROWS, int EPI, bool VEC>
static int launch_few(float* c, const float* a, const float* w, int m, int n, int k, float cap, cudaStream_t s) {
    constexpr int smem = FEW_STAGES * (FEW_N + ROWS) * FEW_LD * (int)sizeof(float);
    if (smem > 48 * 1024 && cudaFuncSetAttribute(gemm_f32_few_kernel<ROWS, EPI, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
        return fail("gemm_f32: cannot have %d bytes of shared memory", smem);
    gemm_f32_few_kernel<ROWS, EPI, VEC><<<(n + FEW_N - 1) / FEW_N, Few<ROWS>::WORKERS + FEW_COPIERS, smem, s>>>(c, a, w, m, n, k, cap);
    return 0;
}

template <int BM, int BN, int TM, int TN, int EPI>
static int launch_tiles(float* c, const float* a, const float* w, int m, int n, int k, float cap, cudaStream_t s) {
    dim3 grid((n + BN - 1) / BN, (m + BM - 1) / BM);
    KB_REQUIRE(grid.y <= 65535, "gemm_f32: %d rows is too many for one launch", m);
    constexpr int smem = f32_smem<BM, BN>();
    if (smem > 48 * 1024 && cudaFuncSetAttribute(gemm_f32_kernel<BM, BN, TM, TN, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
        return fail("gemm_f32: cannot have %d bytes of shared memory", smem);
    gemm_f32_kernel<BM, BN, TM, TN, EPI><<<grid, (BM / TM) * (BN / TN), smem, s>>>(c, a, w, m, n, k, cap);
    return 0;
}

template <int EPI>
static int launch_f32(float* c, const float* a, const float* w, int m, int n, int k, float cap, int variant, cudaStream_t s) {
    if (variant < 0) {
        variant = 0;
        if (m > FEW_ROWS) {
            // The tile whose last wave wastes least: elements a multiprocessor computes, over what a tile of that size reaches of the
            // largest's rate (500 rows by 18,432 x 2,304: 828, 925, 942, 1,083 and 1,519 us in this order).
            const int bm[5] = {128, 128, 64, 64, 32}, bn[5] = {128, 64, 128, 64, 64};
            const double reach[5] = {1.0, 0.9, 0.88, 0.76, 0.55};
            const int sms = multiprocessors();
            double best = 0;
            for (int v = 0; v < 5; ++v) {
                const long long tiles = (long long)((m + bm[v] - 1) / bm[v]) * ((n + bn[v] - 1) / bn[v]);
                const double cost = (double)((tiles + sms - 1) / sms) * bm[v] * bn[v] / reach[v];
                if (v == 0 || cost < best) best = cost, variant = v + 1;
            }
        }
    }
    if (variant == 0) {
        const bool vec = k % 4 == 0 && (((uintptr_t)a | (uintptr_t)w) & 15) == 0;
#define KB_FEW(R) return vec ? launch_few<R, EPI, true>(c, a, w, m, n, k, cap, s) : launch_few<R, EPI, false>(c, a, w, m, n, k, cap, s)
        if (m <= 1) KB_FEW(1);
        if (m <= 2) KB_FEW(2);
        if (m <= 4) KB_FEW(4);
        if (m <= 8) KB_FEW(8);
        KB_FEW(16);
#undef KB_FEW
    }
    if (variant == 1) return launch_tiles<128, 128, 8, 16, EPI>(c, a, w, m, n, k, cap, s);
    if (variant == 2) return launch_tiles<128, 64, 8, 8, EPI>(c, a, w, m, n, k, cap, s);
    if (variant == 3) return launch_tiles<64, 128, 8, 8, EPI>(c, a, w, m, n, k, cap, s);
    if (variant == 4) return launch_tiles<64, 64, 8, 4, EPI>(c, a, w, m, n, k, cap, s);
    return launch_tiles<32, 64, 4, 4, EPI>(c, a, w, m, n, k, cap, s);
}

}  // namespace kb

using namespace kb;

// `variant`: -1 the launcher chooses; 0 the kernel for few rows (at most 16), 1 to 5 the tiles 128 x 128, 128 x 64, 64 x 128, 64 x 64, 32 x 64.
extern "C" int kb_gemm_f32_variant(float* c, const float* a, const float* w, int m, int n, int k, int epilogue, float cap, int variant, void* stream) {
    KB_REQUIRE(m >= 0 && n > 0 && k > 0, "gemm_f32: m %d, n %d, k %d", m, n, k);
    KB_REQUIRE(epilogue == 0 || (epilogue == 1 && cap > 0.f), "gemm_f32: epilogue %d with cap %g", epilogue, cap);
    KB_REQUIRE(variant >= -1 && variant <= 5 && (variant != 0 || m <= FEW_ROWS), "gemm_f32: variant %d for %d rows", variant, m);
    if (m == 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    const int e = epilogue == 0 ? launch_f32<0>(c, a, w, m, n, k, cap, variant, s) : launch_f32<1>(c, a, w, m, n, k, cap, variant, s);
    return e ? e : check_launch("gemm_f32");
}
extern "C" int kb_gemm_f32(float* c, const float* a, const float* w, int m, int n, int k, int epilogue, float cap, void* stream) {
    return kb_gemm_f32_variant(c, a, w, m, n, k, epilogue, cap, -1, stream);
}

// The same by whatever is fastest, the tensor cores included. `scratch`: `kb_gemm_f32_scratch_floats` floats (0: none).
extern "C" long long kb_gemm_f32_scratch_floats(const float* a, const float* w, int m, int n, int k) {
    return m > 0 && n > 0 && k > 0 && gemm_f32_pieces_take(k, a, w) ? gemm_f32_scratch_floats(m, n, k) : 0;
}
extern "C" int kb_gemm_f32_fast(float* c, const float* a, const float* w, int m, int n, int k, int epilogue, float cap, float* scratch, void* stream) {
    if (m > 0 && n > 0 && k > 0 && gemm_f32_pieces_take(k, a, w)) {
        KB_REQUIRE(epilogue == 0 || (epilogue == 1 && cap > 0.f), "gemm_f32: epilogue %d with cap %g", epilogue, cap);
        const int sms = multiprocessors(), groups = gemm_f32_groups(n, k, sms), at_once = gemm_f32_rows_at_once(k);
        for (long long r = 0; r < m; r += at_once) {
            const int rows = m - r < at_once ? (int)(m - r) : at_once;
            if (int e = launch_f32_pieces(c + r * n, a + r * k, w, rows, n, k, epilogue, cap, groups, gemm_f32_way(rows, n, k, groups, sms), scratch, (cudaStream_t)stream)) return e;
        }
        return 0;
    }
    return kb_gemm_f32_variant(c, a, w, m, n, k, epilogue, cap, -1, stream);
}
