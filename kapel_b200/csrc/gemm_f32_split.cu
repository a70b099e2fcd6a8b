// C[M,N] = A[M,K] . W[N,K]^T of 32-bit values on the fifth-generation tensor cores, with no less precision than a chain of 32-bit
// multiply-adds: every input is cut into three bfloat16 pieces (pieces.cuh) and of the nine products of pieces the six that matter are added up,
//     w3 a1 + w1 a3 + w2 a2 + w2 a1 + w1 a2 + w1 a1        (in this order, the small ones first).
// The tensor cores add in 32 bits but round towards zero, so a long sum must not be theirs: an accumulator in tensor memory takes one
// chunk of 64 k, of which only the last four additions are to a sum of full size, and the chunks are added up in registers, rounded to
// nearest.
//
// The operands are swapped, 128 weight rows are the MMA's M and 16, 32, 64 or 128 rows of A its N, for a handful of rows and for thousands
// alike. A row's result does not depend on how many others there are: the weight alone says into how many groups of chunks K is cut
// (`gemm_f32_groups`), a group's chunks are added up in their order, then the groups in theirs, whichever way it is done:
//   beside   a block a group, in a cluster of up to eight, which add up their sums through shared memory (few rows, narrow weights)
//   whole    a block has all of a tile's groups one after the other, the sums so far in tensor memory and, of 128 rows, half in shared memory (in the
//            result's place they took 3.3 us a group), and walks over several tiles where they are more than the multiprocessors: beginning and ending
//            (some 6 us) are there once
//   apart    blocks walk over tiles and groups, a group's sums go to scratch, and a second kernel adds them up (tiles that do not fill the GPU)
//
// Twenty warps:
//   warp 0        asks TMA for 32 k of the 128 weight rows, eight stages deep (three with 128 rows, as fast as five), as 32-bit values (and of up to 32 rows of A)
//   warps 3-10    cut the weights, each half of them every second stage: a thread has a row, its pieces go to tensor memory, from where the
//                 MMA takes its A operand
//   warps 1, 2    issue the 24 MMAs of a chunk, one the even chunks, the other the odd ones (issuing takes a thread longer than the tensor
//                 cores need for a small product; each chunk has pieces and an accumulator of its own)
//   warp 19       asks TMA for the pieces of A, the MMA's B operand, which a kernel ahead of this one has cut: every block of a row of
//                 tiles needs them. They come three chunks ahead (four with 64 rows), which takes the place of stages: two ahead, a chunk of
//                 500 rows by 2,304 x 9,216 waited for them (118 us, now 99; four times as many rows 416 and 363). Up to 32
//                 rows are cut here instead, by warps 11-14, which saves that launch
//   warps 11-18   (15-18) add a finished chunk to the sums they hold in registers, and store them at the end
//
// An element that comes out as no finite number is computed again by multiply-adds, as the other kernels do: values that are none (and those that
// round to infinity in bfloat16) have no pieces, infinity less infinity is NaN, and of a finite product near the largest float or beyond it
// the small products may be infinities of either sign before the large one is added.
// Every wait gives up after about a second, raises a flag that `kb_gemm_f32_split_error` reports, and the block still meets at its
// barriers, frees its TMEM and returns.
#include <initializer_list>
#include "attention_tc.cuh"
#include "gemm_f32_split.cuh"
#include "pieces.cuh"
#include "tensor_map.cuh"

namespace kb {

__device__ int g_gemm_f32_split_error = 0;

constexpr int FP_M = 128, FP_K = 64, FP_STAGE_K = 32, FP_THREADS = 20 * 32;
constexpr int FP_WARP_W = 3, FP_WARP_A = 11, FP_WARP_PIECES = 19;
constexpr long long FP_SCRATCH = 256ll << 20;
constexpr int FP_CUT_ROWS = 32;                                    // up to so many rows of A are cut by the block that needs them

template <int NP> struct Pieces {
    static constexpr bool CUTS = NP <= FP_CUT_ROWS;
    static constexpr int W_BYTES = FP_M * 128, STAGE = W_BYTES + (CUTS ? NP * 128 : 0);            // 32 values of a row are 128 bytes
    static constexpr int PIECE = NP * 128, PIECES = 3 * PIECE;                                     // 64 bfloat16 of a row
    static constexpr int STAGES = NP == 128 ? 3 : 8, PLACES = CUTS ? 2 : (NP == 128 ? 3 : 4);      // of the pieces of A
    static constexpr bool ALL_STAGES = STAGES % 2 != 0;                                            // see the cutting of the weights
    static constexpr int WARP_SUM = CUTS ? 15 : 11, COLS = CUTS ? NP : NP / 2;                     // rows of A whose sums a thread holds
    static constexpr int ACC = NP < 32 ? 32 : NP, COL_W = 2 * ACC, COL_HELD = COL_W + 192, HELD = CUTS ? 0 : 32;      // sums of earlier groups a thread has in tensor memory
    static constexpr int MORE = CUTS ? 0 : (COLS - HELD) * 2 * FP_M * 4;                           // and what does not fit there
    static constexpr int SMEM = STAGES * STAGE + PLACES * PIECES + MORE + 1024 /* alignment */ + 288 /* barriers */;
    static constexpr int TMEM_COLS = COL_HELD + 2 * HELD <= 256 ? 256 : 512;
    static_assert(SMEM <= 232448 && COL_HELD + 2 * HELD <= 512, "more shared or tensor memory than a block can have");
    static_assert(STAGES * STAGE + PLACES * PIECES >= NP * FP_M * 4, "the sums take the place of what was multiplied");
};

__device__ __forceinline__ void fp_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}

__device__ __forceinline__ void fp_cut(float x, float y, uint32_t& one, uint32_t& two, uint32_t& three) {
    x *= PIECE_SCALE, y *= PIECE_SCALE;
    cut_pair(x, y, one, two, three);
}
constexpr float FP_UNSCALE = 1.f / PIECE_SCALE / PIECE_SCALE;       // every sum is too large by the square

__device__ __forceinline__ bool fp_finite(float x) { return fabsf(x) < INFINITY; }
// The product by multiply-adds in ascending k; rows of whole 16-byte pieces.
__device__ __noinline__ float fp_chain(const float* x, const float* y, int k) {
    float v = 0.f;
#pragma unroll 1
    for (int i = 0; i < k; i += 4) {
        const float4 a = *reinterpret_cast<const float4*>(x + i), b = *reinterpret_cast<const float4*>(y + i);
        v = fmaf(a.x, b.x, v), v = fmaf(a.y, b.y, v), v = fmaf(a.z, b.z, v), v = fmaf(a.w, b.w, v);
    }
    return v;
}
__device__ __forceinline__ void fp_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Row tiles of a grouped product, an expert's rows each (moe.cu's lists): A's rows lie in the lists' order, the weights are [experts, n, k].
struct F32Tiles {
    const int* expert;
    const int* first;
    const int* rows;
    const int* count;
    const int* order;          // the pair at each place, where the result's rows are placed by pair; else null
};

// epilogue 0: none; 1: cap * tanh(acc / cap). GROUPED: blockIdx.x is a tile of `tiles`, NP rows at most, m the places there are.
// WALK: a block takes item after item, its warps go on to the next one's chunks while the last one's sums are stored. An item is a group of a tile:
// with `leave_apart` (c is [groups, m, n] then) any of all tiles' groups, gridDim.x apart; else all groups of a tile in turn, the tiles gridDim.x apart.
// Without WALK a block has the one that its place in the grid says.
template <int NP, int EPI, bool GROUPED, bool WALK>
__global__ void __launch_bounds__(FP_THREADS, 1)
gemm_f32_pieces_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, float* __restrict__ c,
                       const float* __restrict__ a, const float* __restrict__ w, int m, int n, int k, int groups, int chunks_a_group, float cap, int leave_apart,
                       const F32Tiles tiles) {
    // map_a: of A's 32-bit values where the block cuts them, else of their pieces [3, m, k up to a multiple of 8]
    using C = Pieces<NP>;
    static_assert(!GROUPED || C::CUTS, "a tile's rows are cut by the blocks that need them");
    static_assert(!WALK || !C::CUTS, "the walk is for many rows");
    extern __shared__ unsigned char fp_raw[];
    if (GROUPED && (int)blockIdx.x >= tiles.count[0]) return;
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)fp_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* pieces = smem + C::STAGES * C::STAGE;           // [PLACES][3][NP rows][128 bytes]
    uint64_t* full = reinterpret_cast<uint64_t*>(pieces + C::PLACES * C::PIECES + C::MORE);
    uint64_t* empty = full + C::STAGES;                            // the warps that cut it have read the stage
    uint64_t* cut = empty + C::STAGES;                             // [2] a chunk's pieces are there that are cut here
    uint64_t* a_full = cut + 2;                                    // [PLACES] its pieces of A that are not
    uint64_t* a_empty = a_full + C::PLACES;                        // [PLACES] and their place is free
    uint64_t* done = a_empty + C::PLACES;                                 // [2] a chunk's products are complete: its pieces' place is free, its sum there
    uint64_t* added = done + 2;                                    // [2] the sum has been read
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(added + 2);
    static_assert((2 * C::STAGES + 2 * C::PLACES + 6) * 8 + 4 <= 288, "the barriers outgrew their room");

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = GROUPED ? tiles.first[blockIdx.x] : blockIdx.x * NP, rows = GROUPED ? min(tiles.rows[blockIdx.x], m - m0) : m - m0;      // what lies behind is not stored
    const int n0 = blockIdx.y * FP_M, w0 = GROUPED ? tiles.expert[blockIdx.x] * n + n0 : n0, segment = WALK ? 0 : blockIdx.z;
    const int m_tiles = (m + NP - 1) / NP, all_tiles = m_tiles * ((n + FP_M - 1) / FP_M), chunks_all = (k + FP_K - 1) / FP_K;
    const bool apart = WALK && leave_apart != 0;
    const int units = apart ? all_tiles * groups : all_tiles, mine = WALK ? (units - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 1;
    const int items = WALK && !apart ? mine * groups : mine;       // this block's
    struct Item { int m0, w0, group, chunk0, chunks; };
    auto item = [&](int i) {
        Item r;
        int tile = 0;
        if (!WALK) r.group = segment;
        else if (apart) r.group = ((int)blockIdx.x + i * (int)gridDim.x) / all_tiles, tile = ((int)blockIdx.x + i * (int)gridDim.x) % all_tiles;
        else r.group = i % groups, tile = (int)blockIdx.x + i / groups * (int)gridDim.x;
        r.m0 = WALK ? tile % m_tiles * NP : m0, r.w0 = WALK ? tile / m_tiles * FP_M : w0;
        r.chunk0 = r.group * chunks_a_group, r.chunks = max(0, min(chunks_a_group, chunks_all - r.chunk0));
        return r;
    };
    int chunks = 0;                                                // of all items
    if (WALK && !apart) chunks = mine * chunks_all;
    else
        for (int i = 0; i < items; ++i) chunks += item(i).chunks;

    if (tid == 0) {
        for (int s = 0; s < C::STAGES; ++s) { at_mbar_init(full + s, 1); at_mbar_init(empty + s, C::CUTS ? 6 : C::ALL_STAGES ? 8 : 4); }      // the warps that cut the stage
        for (int b = 0; b < 2; ++b) {
            at_mbar_init(cut + b, C::CUTS ? 12 : 8);
            at_mbar_init(done + b, 1);
            at_mbar_init(added + b, C::CUTS ? 4 : 8);
        }
        for (int b = 0; b < C::PLACES; ++b) { at_mbar_init(a_full + b, 1); at_mbar_init(a_empty + b, 1); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(at_saddr(tmem_slot)), "r"(C::TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    at_fence_before();
    __syncthreads();
    at_fence_after();
    const uint32_t tmem = *tmem_slot;
    bool failed = false;
    constexpr int COLS = C::COLS;
    float sum[COLS];

    if (warp == 0) {
        if (lane == 0) {
            int it = 0;
            for (int i = 0; i < items && !failed; ++i) {
                const Item at = item(i);
                for (int step = 0; step < 2 * at.chunks; ++step, ++it) {
                    const int s = it % C::STAGES;
                    if (!at_mbar_wait(empty + s, ((uint32_t)(it / C::STAGES) & 1u) ^ 1u)) { failed = true; break; }
                    const uint32_t dst = at_saddr(smem + s * C::STAGE);
                    at_mbar_expect_tx(full + s, C::STAGE);
                    at_tma_box(dst, &map_w, at.chunk0 * FP_K + step * FP_STAGE_K, at.w0, full + s);
                    if (C::CUTS) at_tma_box(dst + C::W_BYTES, &map_a, at.chunk0 * FP_K + step * FP_STAGE_K, at.m0, full + s);
                }
            }
            if (failed)                                            // the copies in flight land before the block goes on
                for (int i = max(0, it - C::STAGES); i < it; ++i) at_mbar_wait(full + i % C::STAGES, (uint32_t)(i / C::STAGES) & 1u);
        }
    } else if (warp < FP_WARP_W) {
        // ---------------------------------------------------------------- the products of every second chunk
        // The whole warp walks the loop and one lane's products go: inside a branch of one lane the operands have to be brought into the
        // uniform registers that the instruction takes them from one by one, and a product of 128 rows took 118 clocks, not 64.
        constexpr uint32_t IDESC = at_idesc(FP_M, NP, false);
        const int b = __shfl_sync(0xffffffffu, warp, 0) - 1;
        const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
        const uint32_t d = tm + (uint32_t)(b * C::ACC), aw = tm + (uint32_t)(C::COL_W + b * 96);
        const uint64_t first = at_desc(at_saddr(pieces), 16, 1024);
        int place = b;
        for (int ch = b; ch < chunks; ch += 2) {
            bool there = at_mbar_wait(cut + b, (uint32_t)(ch >> 1) & 1u);
            // With three places this warp meets one every second round; the round between is over: the weights' chunk ch is cut behind the products of ch - 3.
            if (!C::CUTS) there = there && at_mbar_wait(a_full + place, (uint32_t)(ch / C::PLACES) & 1u);
            there = there && at_mbar_wait(added + b, ((uint32_t)(ch >> 1) & 1u) ^ 1u);
            if (!__all_sync(0xffffffffu, there)) { failed = true; break; }
            at_fence_after();
            const uint32_t one = at_elect();
            const uint64_t ba = first + (uint64_t)(place * (C::PIECES >> 4));
#pragma unroll
            for (int p = 0; p < PIECE_PRODUCTS; ++p)
#pragma unroll
                for (int kk = 0; kk < FP_K / 16; ++kk)
                    at_mma_ts_if(one, d, aw + (uint32_t)(piece_a(p) * 32 + kk * 8), ba + (uint64_t)(piece_b(p) * (C::PIECE >> 4) + kk * 2), IDESC, (p | kk) != 0 ? 1u : 0u);
            if (one) at_commit(done + b);
            if (!C::CUTS && one) at_commit(a_empty + place);
            __syncwarp();
            if (!C::CUTS) place = place + 2 >= C::PLACES ? place + 2 - C::PLACES : place + 2;
        }
    } else if (warp < FP_WARP_A) {
        // ---------------------------------------------------------------- cutting the weights: a stage is half a chunk
        // A wait by parity tells a round of a stage from the one before only. With an even number of stages a half has stages of its own. With an odd one a stage is
        // the other half's every second time: then both halves' warps wait for each round of each stage, and it is empty when all of them have.
        const int quarter = warp & 3, half = (warp - FP_WARP_W) >> 2;      // of the TMEM lanes, which are the weight rows; of the chunk
        const int row = quarter * 32 + lane;
        for (int ch = 0; ch < chunks; ++ch) {
            const int it = 2 * ch + half, s = it % C::STAGES, b = ch & 1;
            auto pass_on = [&](int other) {                        // the other half's stage
                if (!__all_sync(0xffffffffu, at_mbar_wait(full + other % C::STAGES, (uint32_t)(other / C::STAGES) & 1u))) return false;
                if (lane == 0) at_mbar_arrive(empty + other % C::STAGES);
                return true;
            };
            if (C::ALL_STAGES && half == 1 && !pass_on(it - 1)) { failed = true; break; }
            if (!__all_sync(0xffffffffu, at_mbar_wait(full + s, (uint32_t)(it / C::STAGES) & 1u))) { failed = true; break; }
            const unsigned char* from = smem + s * C::STAGE + row * 128;
            uint32_t one[16], two[16], three[16];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float4 x = *reinterpret_cast<const float4*>(from + ((j ^ (row & 7)) << 4));
                fp_cut(x.x, x.y, one[2 * j], two[2 * j], three[2 * j]);
                fp_cut(x.z, x.w, one[2 * j + 1], two[2 * j + 1], three[2 * j + 1]);
            }
            __syncwarp();
            if (lane == 0) at_mbar_arrive(empty + s);
            if (C::ALL_STAGES && half == 0 && !pass_on(it + 1)) { failed = true; break; }
            // the chunk two before this one was the last to lie here
            if (!__all_sync(0xffffffffu, at_mbar_wait(done + b, ((uint32_t)(ch >> 1) & 1u) ^ 1u))) { failed = true; break; }
            at_fence_after();
            const uint32_t to = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(C::COL_W + b * 96 + half * 16);
            at_st16(to, one);
            at_st16(to + 32, two);
            at_st16(to + 64, three);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            at_fence_before();
            __syncwarp();
            if (lane == 0) at_mbar_arrive(cut + b);
        }
    } else if (C::CUTS && warp < C::WARP_SUM) {
        // ---------------------------------------------------------------- cutting a few rows of A, two warps a half of the chunk
        const int half = (warp - FP_WARP_A) >> 1, t = ((warp - FP_WARP_A) & 1) * 32 + lane, row = t % NP;
        for (int ch = 0; ch < chunks; ++ch) {
            const int it = 2 * ch + half, s = it % C::STAGES, b = ch & 1;
            if (!__all_sync(0xffffffffu, at_mbar_wait(full + s, (uint32_t)(it / C::STAGES) & 1u))) { failed = true; break; }
            if (!__all_sync(0xffffffffu, at_mbar_wait(done + b, ((uint32_t)(ch >> 1) & 1u) ^ 1u))) { failed = true; break; }
            const unsigned char* from = smem + s * C::STAGE + C::W_BYTES + row * 128;
            unsigned char* to = pieces + b * C::PIECES + row * 128;
#pragma unroll
            for (int i = t; i < NP * 4; i += 64) {                 // eight values at a time
                const int g = i / NP;
                const float4 x = *reinterpret_cast<const float4*>(from + (((2 * g) ^ (row & 7)) << 4));
                const float4 y = *reinterpret_cast<const float4*>(from + (((2 * g + 1) ^ (row & 7)) << 4));
                uint4 one, two, three;
                fp_cut(x.x, x.y, one.x, two.x, three.x);
                fp_cut(x.z, x.w, one.y, two.y, three.y);
                fp_cut(y.x, y.y, one.z, two.z, three.z);
                fp_cut(y.z, y.w, one.w, two.w, three.w);
                const int at = ((half * 4 + g) ^ (row & 7)) << 4;
                *reinterpret_cast<uint4*>(to + at) = one;
                *reinterpret_cast<uint4*>(to + C::PIECE + at) = two;
                *reinterpret_cast<uint4*>(to + 2 * C::PIECE + at) = three;
            }
            at_fence_async_smem();                                 // the MMAs read what was written here
            __syncwarp();
            if (lane == 0) {
                at_mbar_arrive(empty + s);
                at_mbar_arrive(cut + b);
            }
        }
    } else if (warp == FP_WARP_PIECES) {
        if (!C::CUTS) {
            // ------------------------------------------------------------ A's pieces
            if (lane == 0) {
                int ch = 0;
                for (int i = 0; i < items && !failed; ++i) {
                    const Item at = item(i);
                    for (int j = 0; j < at.chunks; ++j, ++ch) {
                        const int b = ch % C::PLACES;
                        if (!at_mbar_wait(a_empty + b, ((uint32_t)(ch / C::PLACES) & 1u) ^ 1u)) { failed = true; break; }
                        at_mbar_expect_tx(a_full + b, C::PIECES);
                        for (int p = 0; p < 3; ++p)
                            at_tma_box(at_saddr(pieces + b * C::PIECES + p * C::PIECE), &map_a, (at.chunk0 + j) * FP_K, p * m + at.m0, a_full + b);
                    }
                }
                if (failed)                                        // as above
                    for (int i = max(0, ch - C::PLACES); i < ch; ++i) at_mbar_wait(a_full + i % C::PLACES, (uint32_t)(i / C::PLACES) & 1u);
            }
        }
    } else {
        // ---------------------------------------------------------------- adding up: a weight row and COLS of A's rows a thread
        const int quarter = warp & 3, half = (warp - C::WARP_SUM) >> 2;
        const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * COLS);
        int ch = 0;
        for (int i = 0; i < items && !failed; ++i) {
            const Item at = item(i);
#pragma unroll
            for (int j = 0; j < COLS; ++j) sum[j] = 0.f;
            for (const int end = ch + at.chunks; ch < end; ++ch) {
                const int b = ch & 1;
                if (!__all_sync(0xffffffffu, at_mbar_wait(done + b, (uint32_t)(ch >> 1) & 1u))) { failed = true; break; }
                at_fence_after();
#pragma unroll
                for (int c0 = 0; c0 < COLS; c0 += 16) {
                    uint32_t r[16];
                    fp_ld16(lanes + (uint32_t)(b * C::ACC + c0), r);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (c0 + 16 == COLS) {
                        at_fence_before();
                        __syncwarp();
                        if (lane == 0) at_mbar_arrive(added + b);
                    }
#pragma unroll
                    for (int j = 0; j < 16; ++j) sum[c0 + j] += __uint_as_float(r[j]);
                }
            }
            if constexpr (WALK) {
                if (failed) break;
                if (!apart && groups > 1) {                        // the groups so far, half of 128 rows' sums (all of 64) in tensor memory
                    const uint32_t held = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(C::COL_HELD + half * C::HELD);
                    float* more = reinterpret_cast<float*>(pieces + C::PLACES * C::PIECES) + half * (COLS - C::HELD) * FP_M + quarter * 32 + lane;
                    if (at.group > 0) {
#pragma unroll
                        for (int c0 = 0; c0 < C::HELD; c0 += 16) {
                            uint32_t r[16];
                            fp_ld16(held + (uint32_t)c0, r);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                            for (int j = 0; j < 16; ++j) sum[c0 + j] = __uint_as_float(r[j]) + sum[c0 + j];
                        }
#pragma unroll
                        for (int j = C::HELD; j < COLS; ++j) sum[j] = more[(j - C::HELD) * FP_M] + sum[j];
                    }
                    if (at.group < groups - 1) {
#pragma unroll
                        for (int c0 = 0; c0 < C::HELD; c0 += 16) {
                            uint32_t r[16];
#pragma unroll
                            for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(sum[c0 + j]);
                            at_st16(held + (uint32_t)c0, r);
                        }
                        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int j = C::HELD; j < COLS; ++j) more[(j - C::HELD) * FP_M] = sum[j];
                        continue;
                    }
                }
                const int w_row = at.w0 + quarter * 32 + lane, j0 = half * COLS, many = min(COLS, m - at.m0 - j0);
                if (w_row < n) {
                    float* to = c + (size_t)((apart ? at.group * m : 0) + at.m0 + j0) * n + w_row;
                    float check = 0.f;                             // NaN once a sum is no finite number
#pragma unroll
                    for (int j = 0; j < COLS; ++j) {
                        float v = sum[j];
                        check = fmaf(v, 0.f, check);
                        if (!apart) v *= FP_UNSCALE;
                        if (EPI == 1 && !apart) v = cap * tanhf(v / cap);
                        if (j < many) to[(size_t)j * n] = v;
                    }
                    if (!apart && check != check) {                // as they are, then one after the other
                        if (EPI == 1) {
#pragma unroll
                            for (int j = 0; j < COLS; ++j)
                                if (j < many) to[(size_t)j * n] = sum[j] * FP_UNSCALE;
                        }
#pragma unroll 1
                        for (int j = 0; j < many; ++j) {
                            float v = to[(size_t)j * n];
                            if (!fp_finite(v)) v = fp_chain(a + (size_t)(at.m0 + j0 + j) * k, w + (size_t)w_row * k, k);
                            to[(size_t)j * n] = EPI == 1 ? cap * tanhf(v / cap) : v;
                        }
                    }
                }
            }
        }
    }
    __syncthreads();                                               // the stages have been read
    float* sums = reinterpret_cast<float*>(smem);                  // [NP][128], where K is cut
    constexpr bool ONE = C::CUTS;                                  // K may be in one group (many rows walk then)
    auto to = [&](int j) { return (size_t)(GROUPED && tiles.order != nullptr ? tiles.order[m0 + j] : m0 + j) * n + n0; };
    if (!WALK && warp >= C::WARP_SUM && warp != FP_WARP_PIECES) {
        const int r = (warp & 3) * 32 + lane, j0 = ((warp - C::WARP_SUM) >> 2) * COLS;
        if (!ONE || groups > 1) {
#pragma unroll
            for (int j = 0; j < COLS; ++j) sums[(j0 + j) * FP_M + r] = sum[j];
        } else if (n0 + r < n) {
            float check = 0.f;                                     // as above
#pragma unroll
            for (int j = 0; j < COLS; ++j) {
                float v = sum[j] * FP_UNSCALE;
                check = fmaf(v, 0.f, check);
                if (EPI == 1) v = cap * tanhf(v / cap);
                if (j0 + j < rows) c[to(j0 + j) + r] = v;
            }
            if (check != check) {
                if (EPI == 1) {
#pragma unroll
                    for (int j = 0; j < COLS; ++j)
                        if (j0 + j < rows) c[to(j0 + j) + r] = sum[j] * FP_UNSCALE;
                }
#pragma unroll 1
                for (int j = 0; j < min(COLS, rows - j0); ++j) {
                    float v = c[to(j0 + j) + r];
                    if (!fp_finite(v)) v = fp_chain(a + (size_t)(m0 + j0 + j) * k, w + (size_t)(w0 + r) * k, k);
                    c[to(j0 + j) + r] = EPI == 1 ? cap * tanhf(v / cap) : v;
                }
            }
        }
    }
    if (!WALK && (!ONE || groups > 1)) {
        fp_cluster_sync();
        const int per = NP / groups;                               // rows of A this block adds up
        for (int i = tid; i < per * FP_M; i += FP_THREADS) {
            const int j = segment * per + i / FP_M, r = i % FP_M;
            const uint32_t at = at_saddr(sums + j * FP_M + r);
            float v = 0.f;
            for (int s = 0; s < groups; ++s) {
                float x;
                asm volatile("{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %1, %2;\n\tld.shared::cluster.f32 %0, [ra];\n\t}"
                             : "=f"(x) : "r"(at), "r"(s) : "memory");
                v = s == 0 ? x : v + x;
            }
            if (j < rows && n0 + r < n) {
                v *= FP_UNSCALE;
                if (!fp_finite(v)) v = fp_chain(a + (size_t)(m0 + j) * k, w + (size_t)(w0 + r) * k, k);
                c[to(j) + r] = EPI == 1 ? cap * tanhf(v / cap) : v;
            }
        }
        fp_cluster_sync();                                         // nobody leaves while its sums are read
    }
    if (failed) atomicExch(&g_gemm_f32_split_error, 1);
    at_fence_before();
    __syncthreads();
    if (warp == 1) {
        at_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::TMEM_COLS) : "memory");
    }
}

// A's rows cut for a product of more than FP_CUT_ROWS: pieces [3, m, kp], kp the next multiple of 8 (the columns beyond k are zeros).
// A block a row.
__global__ void __launch_bounds__(256)
f32_cut_rows_kernel(const float* __restrict__ a, uint32_t* __restrict__ pieces, int m, int k, int kp) {
    const int row = blockIdx.x;
    const float* from = a + (size_t)row * k;
    uint32_t* to = pieces + (size_t)row * (kp / 2);
    const size_t piece = (size_t)m * (kp / 2);
    for (int x = threadIdx.x * 4; x < kp; x += 1024) {             // k is a multiple of four
        const float4 v = x < k ? *reinterpret_cast<const float4*>(from + x) : make_float4(0.f, 0.f, 0.f, 0.f);
        uint2 one, two, three;
        fp_cut(v.x, v.y, one.x, two.x, three.x);
        fp_cut(v.z, v.w, one.y, two.y, three.y);
        *reinterpret_cast<uint2*>(to + x / 2) = one;
        *reinterpret_cast<uint2*>(to + piece + x / 2) = two;
        *reinterpret_cast<uint2*>(to + 2 * piece + x / 2) = three;
    }
}

// c = the groups' sums added up in their order: four elements a thread.
template <int EPI>
__global__ void __launch_bounds__(256)
f32_add_groups_kernel(float* __restrict__ c, const float* __restrict__ partial, const float* __restrict__ a, const float* __restrict__ w, long long all, int n, int k, int groups, float cap) {
    const long long first = (long long)blockIdx.x * 1024 + threadIdx.x;
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = first + 256 * j < all ? partial[first + 256 * j] : 0.f;
#pragma unroll 3
    for (int g = 1; g < groups; ++g)
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (first + 256 * j < all) v[j] += partial[(size_t)g * all + first + 256 * j];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const long long i = first + 256 * j;
        if (i >= all) break;
        v[j] *= FP_UNSCALE;
        if (!fp_finite(v[j])) v[j] = fp_chain(a + (size_t)(i / n) * k, w + (size_t)(i % n) * k, k);
        c[i] = EPI == 1 ? cap * tanhf(v[j] / cap) : v[j];
    }
}

template <int NP, int EPI>
static int launch_pieces(float* c, const float* a, const float* w, int m, int n, int k, int groups, int way, float cap, float* scratch, cudaStream_t s) {
    using C = Pieces<NP>;
    CUtensorMap map_a, map_w;
    const int kp = (k + 7) & ~7, chunks = (k + FP_K - 1) / FP_K, chunks_a_group = (chunks + groups - 1) / groups, sms = multiprocessors();
    KB_REQUIRE((n + FP_M - 1) / FP_M <= 65535, "gemm_f32: a weight of %d rows is too much for one launch", n);
    const bool walk = !C::CUTS && (way != FP_BESIDE || groups == 1);
    if (walk) groups = (chunks + chunks_a_group - 1) / chunks_a_group;       // those that are empty add nothing
    const long long tiles = (long long)((m + NP - 1) / NP) * ((n + FP_M - 1) / FP_M), units = way == FP_APART ? tiles * groups : tiles;
    KB_REQUIRE(units <= 0x7fffffff - sms && (units / sms + 1) * chunks < 0x3fffffff, "gemm_f32: %d rows by %d x %d are too much for one launch", m, n, k);
    float* partial = walk && way == FP_APART ? scratch + gemm_f32_pieces_floats(m, k) : nullptr;
    auto kernel = gemm_f32_pieces_kernel<NP, EPI, false, false>;
    if constexpr (!C::CUTS)
        if (walk) kernel = gemm_f32_pieces_kernel<NP, EPI, false, true>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) != cudaSuccess)
        return fail("gemm_f32: cannot have %d bytes of shared memory", C::SMEM);
    if (int e = encode_map_f32(&map_w, w, n, k, k, FP_M)) return e;
    if (C::CUTS) {
        if (int e = encode_map_f32(&map_a, a, m, k, k, NP)) return e;
    } else {
        KB_REQUIRE(scratch != nullptr && ((uintptr_t)scratch & 15) == 0, "gemm_f32: %d rows by pieces without scratch", m);
        if (int e = encode_map_bf16(&map_a, scratch, 3ull * m, kp, kp, NP)) return e;
        f32_cut_rows_kernel<<<m, 256, 0, s>>>(a, reinterpret_cast<uint32_t*>(scratch), m, k, kp);
        if (int e = check_launch("gemm_f32 cut")) return e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = walk ? dim3((unsigned)(units < sms ? units : sms)) : dim3((m + NP - 1) / NP, (n + FP_M - 1) / FP_M, groups);
    cfg.blockDim = FP_THREADS;
    cfg.dynamicSmemBytes = C::SMEM;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = walk ? 1 : groups;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, map_a, map_w, partial != nullptr ? partial : c, a, w, m, n, k, groups, chunks_a_group, cap, (int)(partial != nullptr), F32Tiles{});
    if (int e = check_launch("gemm_f32 pieces")) return e;
    if (partial == nullptr) return 0;
    const long long all = (long long)m * n;
    KB_REQUIRE((all + 1023) / 1024 <= 0x7fffffffll, "gemm_f32: %d rows by %d are too much for one launch", m, n);
    f32_add_groups_kernel<EPI><<<(unsigned)((all + 1023) / 1024), 256, 0, s>>>(c, partial, a, w, all, n, k, groups, cap);
    return check_launch("gemm_f32 groups");
}

// Clusters of four and eight do not fit every group of multiprocessors, so that seven eighths and three quarters run at once (144 blocks in
// clusters of eight: two waves).
static int fp_clusters(int groups, int sms) {
    const int at_once = groups <= 2 ? sms : (groups == 4 ? sms * 7 / 8 : sms * 3 / 4) / groups * groups;
    return at_once > 0 ? at_once : 1;
}
// Groups of K: what is fastest for up to 32 rows, whatever the rows there are. The waves of blocks times what a block takes, 0.65 us a chunk, and 5 or (in a
// cluster) 6.5 us to begin and end.
int gemm_f32_groups(int n, int k, int sms) {
    const int tiles = (n + FP_M - 1) / FP_M, chunks = (k + FP_K - 1) / FP_K;
    int best = 1;
    double least = 0;
    for (int g = 1; g <= 8 && g <= chunks; g *= 2) {
        const int at_once = fp_clusters(g, sms), waves = (int)(((long long)tiles * g + at_once - 1) / at_once);
        const double us = waves * ((chunks + g - 1) / g * 0.65 + (g == 1 ? 5.0 : 6.5));
        if (g == 1 || us < least) least = us, best = g;
    }
    return best;
}
// How the groups are done: what the three ways take, 0.68 us a chunk with 64 rows a tile and 1.2 with 128, 0.7 us to leave a group's sums and take
// them up again, 1 us and 4 TB/s to add up what lies apart. In us, beside, whole and apart, by 2,304 x 9,216 in four groups: 128 rows 50, 137, 52; 256 rows
// 90, 140, 56; 500 rows 140, 155, 101; 2,048 rows 543, 413, 447. By 4,096 x 2,304 in four: 128 rows 25, 44, 27; 256 rows 41, 46, 37; 500 rows 73, 48, 60; 2,048 rows 266, 176, 200
// (in one group 165).
int gemm_f32_way(int m, int n, int k, int groups, int sms) {
    if (m <= FP_CUT_ROWS) return FP_BESIDE;
    if (groups == 1) return FP_WHOLE;
    const int np = m <= 64 ? 64 : 128, chunks = (k + FP_K - 1) / FP_K, each = (chunks + groups - 1) / groups;
    const long long tiles = (long long)((m + np - 1) / np) * ((n + FP_M - 1) / FP_M);
    const auto waves = [](long long blocks, int at_once) { return (double)((blocks + at_once - 1) / at_once); };
    const double chunk_us = np == 64 ? 0.68 : 1.2;
    const double beside = waves(tiles * groups, fp_clusters(groups, sms)) * (each * chunk_us + 6.5);
    const double whole = waves(tiles, sms) * (chunks * chunk_us + 0.7 * (groups - 1)) + 5.0;
    const double apart = waves(tiles * groups, sms) * (each * chunk_us + 0.7) + 5.0 + 1.0 + (groups + 1.0) * m * n * 1e-6;
    const bool room = (long long)groups * m * n * 4 <= FP_SCRATCH;
    return beside <= whole && (beside <= apart || !room) ? FP_BESIDE : whole <= apart || !room ? FP_WHOLE : FP_APART;
}
// From 256 inputs on, whatever the rows: one accumulator an element in ascending k, a kernel for each, is limited by
// its chain or by the FMA pipe; here a chunk's 24 products take the same time whatever the rows, up to 64. 500 rows by 18,432 x 2,304: 824 us by
// chains, 178 by pieces; by 2,304 x 9,216 545 and 101, by 2,304 x 2,048 131 and 36, by 64 x 2,048 62 and 18, by 512 x 512 17 and 18, by 1,024 x 256 13 and
// 15 (64 rows 9.3 and 12). Eight rows: 56 and 33, 107 and 45, 27 and 17, 19 and 9, 8.2 and 8.4, 8.3 and 8.3. One and two rows are no
// faster in all: by 18,432 x 2,304 39 and 33, by 2,304 x 9,216 48 and 45, by 2,304 x 2,048 15 and 17, by 2,048 x 1,024 8.3 and 10.6, by 256,000 x 2,304 369
// and 416; they go this way so that a row has the same bits alone and beside others. The error against 64 bits is 0.07 to 0.3 of the
// chains' (500 rows by 2,304 x 9,216: 1.4e-7 and 1.7e-6; by 1,024 x 256: 8.8e-8 and 2.9e-7).
bool gemm_f32_pieces_take(int k, const void* a, const void* w) { return k >= 256 && k % 4 == 0 && (((uintptr_t)a | (uintptr_t)w) & 15) == 0; }
long long gemm_f32_pieces_floats(int m, int k) { return m <= FP_CUT_ROWS ? 0 : (long long)m * 3 * ((k + 7) / 8 * 4); }
// Scratch does not grow with the rows beyond FP_SCRATCH for pieces and as much for groups that lie apart: more rows go by several launches, of at least 1,024.
int gemm_f32_rows_at_once(int k) {
    const long long rows = FP_SCRATCH / (6ll * ((k + 7) / 8 * 8)) / 128 * 128;
    return rows < 1024 ? 1024 : rows > 0x3fffff80 ? 0x3fffff80 : (int)rows;
}
long long gemm_f32_scratch_floats(int m, int n, int k) {
    const int sms = multiprocessors(), groups = gemm_f32_groups(n, k, sms), at_once = gemm_f32_rows_at_once(k);
    long long most = 0;
    for (int rows : {m < at_once ? m : at_once, m % at_once}) {
        const long long floats = gemm_f32_pieces_floats(rows, k) + (gemm_f32_way(rows, n, k, groups, sms) == FP_APART ? (long long)groups * rows * n : 0);
        most = floats > most ? floats : most;
    }
    return most;
}

int launch_f32_pieces(float* c, const float* a, const float* w, int m, int n, int k, int epilogue, float cap, int groups, int way, float* scratch, cudaStream_t s) {
    KB_REQUIRE(k % 4 == 0 && (((uintptr_t)a | (uintptr_t)w) & 15) == 0, "gemm_f32: rows of %d values must begin at 16-byte boundaries", k);
    KB_REQUIRE((groups == 1 || groups == 2 || groups == 4 || groups == 8) && way >= FP_BESIDE && way <= FP_APART, "gemm_f32: %d groups by way %d", groups, way);
#define KB_PIECES(NP) \
    return epilogue == 0 ? launch_pieces<NP, 0>(c, a, w, m, n, k, groups, way, cap, scratch, s) : launch_pieces<NP, 1>(c, a, w, m, n, k, groups, way, cap, scratch, s)
    if (m <= 16) KB_PIECES(16);
    if (m <= 32) KB_PIECES(32);
    if (m <= 64) KB_PIECES(64);
    KB_PIECES(128);
#undef KB_PIECES
}

// Whether the experts' 32-bit products of this inner size go by pieces.
bool moe_f32_pieces_take(int k, const void* a, const void* w) { return k >= 256 && k % 4 == 0 && (((uintptr_t)a | (uintptr_t)w) & 15) == 0; }

}  // namespace kb

using namespace kb;

// c [places, n]: a [places, k] (in the lists' order) by the expert's weights w [experts, n, k], tiles of at most FP_CUT_ROWS rows; `order` not null: rows
// placed by pair number. A block a tile and 128 columns, K in one: the tiles alone fill the GPU. 1,200 pairs of 16 experts of 2,048 x 1,024, both
// products: 555 us by multiply-adds, 146 so; 16 pairs 316 and 28.
extern "C" int kb_moe_f32_pieces_takes(const float* a, const float* w, int k) { return moe_f32_pieces_take(k, a, w) ? 1 : 0; }
extern "C" int kb_moe_f32_pieces(float* c, const float* a, const float* w, int experts, const int* tile_expert, const int* tile_first, const int* tile_rows,
                                 const int* n_tiles, int tile_cap, const int* order, int places, int n, int k, void* stream) {
    using C = Pieces<FP_CUT_ROWS>;
    KB_REQUIRE(experts > 0 && places >= 0 && n > 0 && k > 0 && tile_cap >= 0, "moe_f32: %d experts, %d places, n %d, k %d, %d tiles", experts, places, n, k, tile_cap);
    KB_REQUIRE(k % 4 == 0 && (((uintptr_t)a | (uintptr_t)w) & 15) == 0, "moe_f32: rows of %d values must begin at 16-byte boundaries", k);
    KB_REQUIRE((n + FP_M - 1) / FP_M <= 65535 && (long long)experts * n <= 0x7fffffffll, "moe_f32: %d experts of %d rows are too much for one launch", experts, n);
    if (tile_cap == 0 || places == 0) return 0;
    auto kernel = gemm_f32_pieces_kernel<FP_CUT_ROWS, 0, true, false>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) != cudaSuccess) return fail("moe_f32: cannot have %d bytes of shared memory", C::SMEM);
    CUtensorMap map_a, map_w;
    if (int e = encode_map_f32(&map_a, a, places, k, k, FP_CUT_ROWS)) return e;
    if (int e = encode_map_f32(&map_w, w, (unsigned long long)experts * n, k, k, FP_M)) return e;
    kernel<<<dim3(tile_cap, (n + FP_M - 1) / FP_M), FP_THREADS, C::SMEM, (cudaStream_t)stream>>>(map_a, map_w, c, a, w, places, n, k, 1, (k + FP_K - 1) / FP_K, 0.f, 0,
                                                                                                  F32Tiles{tile_expert, tile_first, tile_rows, n_tiles, order});
    return check_launch("moe_f32 pieces");
}

extern "C" int kb_gemm_f32_split_error() {
    int flag = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&flag, g_gemm_f32_split_error, sizeof(int)) != cudaSuccess) return -1;
    if (flag) cudaMemcpyToSymbol(g_gemm_f32_split_error, &zero, sizeof(int));
    return flag;
}
// The kernels over pieces whatever the sizes, K in `groups` (0: as the rule has it), by `way` (FpWay; -1: as the rule has it).
extern "C" int kb_gemm_f32_pieces_by(float* c, const float* a, const float* w, int m, int n, int k, int epilogue, float cap, int groups, int way, float* scratch, void* stream) {
    KB_REQUIRE(m >= 0 && n > 0 && k > 0, "gemm_f32: m %d, n %d, k %d", m, n, k);
    KB_REQUIRE(epilogue == 0 || (epilogue == 1 && cap > 0.f), "gemm_f32: epilogue %d with cap %g", epilogue, cap);
    if (m == 0) return 0;
    const int sms = multiprocessors();
    if (groups <= 0) groups = gemm_f32_groups(n, k, sms);
    return launch_f32_pieces(c, a, w, m, n, k, epilogue, cap, groups, way < 0 ? gemm_f32_way(m, n, k, groups, sms) : way, scratch, (cudaStream_t)stream);
}
extern "C" int kb_gemm_f32_groups(int n, int k) { return gemm_f32_groups(n, k, multiprocessors()); }
// The same by clusters, or in one group.
extern "C" int kb_gemm_f32_pieces(float* c, const float* a, const float* w, int m, int n, int k, int epilogue, float cap, int segments, float* scratch, void* stream) {
    return kb_gemm_f32_pieces_by(c, a, w, m, n, k, epilogue, cap, segments, FP_BESIDE, scratch, stream);
}
