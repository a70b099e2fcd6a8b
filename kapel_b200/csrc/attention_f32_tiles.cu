// Attention of prompt portions over the paged cache in true 32-bit: tiles of rows instead of one row a block.
//
// The row-wise kernel reads every key again for every token and finishes a chunk of 256 keys a block (399 us for 500 tokens, 8 heads
// over 4 of 256). Here a block takes 32 rows -- (token, query head) pairs of one kv head -- and walks their keys 64 at a time: scores by 32-bit
// multiply-adds from shared memory, the running maximum and the weights eight threads a row, then the weighted sum into registers. Keys and values come
// by asynchronous copies, the next keys while the values are multiplied, the values while the scores are made. No tensor-core instruction: nothing
// rounds an input; exponentials and soft caps are the library's. Sums go by pieces (chains of 8 components; of 64 keys, then of 256), so that their
// rounding is no larger than the row-wise kernel's, whose lanes and chunks cut them as short: 0.7 to 0.99 of its error against 64 bits at 500
// to 4,608 keys, where one chain a sum had 1.8 to 4.7 times as much and took 139 us instead of 147. Shared memory's 32 words a clock bound it (0.75
// and 0.38 words a multiply-add), and how few blocks a short prompt gives: 146 us for those 500 tokens by a block a tile, which is what the 8 steps of
// the last rows' block take. With heads of 128 two blocks share a multiprocessor. Where the tiles are few, a cluster of two blocks takes one, every second
// step each, and the first merges what the second leaves in its shared memory: 99 us.
#include <type_traits>
#include "common.cuh"

namespace kb {

constexpr int AFT_ROWS = 32, AFT_KEYS = 64, AFT_THREADS = 256;

struct F32TileParams {
    const float* q;            // [rows, hq, D]
    const float* k_table;      // [pages, hkv, page_size, D]
    const float* v_table;
    const int* block_table;    // [entries, table_width]
    const int* row_count;      // [rows]
    const int* tile_entry;
    const int* tile_row0;
    const int* tile_nq;
    const float* sinks;        // [hq] or null
    float* out;                // [rows, hq, D]
    int hq, hkv, page_size, table_width, n_pages, window;
    float scale, cap;
};

__device__ __forceinline__ void aft_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// A float at the same place in the cluster's block `rank`.
__device__ __forceinline__ float aft_remote(const float* at, int rank) {
    float v;
    asm volatile("{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %1, %2;\n\tld.shared::cluster.f32 %0, [ra];\n\t}"
                 : "=f"(v) : "r"((uint32_t)__cvta_generic_to_shared(at)), "r"(rank) : "memory");
    return v;
}
__device__ __forceinline__ float4 aft_remote_four(const float* at, int rank) {
    float4 v;
    asm volatile("{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %4, %5;\n\tld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [ra];\n\t}"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"((uint32_t)__cvta_generic_to_shared(at)), "r"(rank) : "memory");
    return v;
}

// PARTS: blocks (of a cluster, along z) a tile, 1 or 2
template <int D, int PARTS>
__global__ void __launch_bounds__(AFT_THREADS, D == 128 ? 2 : 1)
attention_f32_tiles_kernel(const F32TileParams p) {
    constexpr int LD = D + 4, D4 = D / 4, CG = D / 128;          // column groups of four a lane holds: 4 (lane + 32 g)
    extern __shared__ __align__(16) float aft_smem[];
    float* sq = aft_smem;                                        // [32][LD]
    float* sk = sq + AFT_ROWS * LD;                              // [64][LD]
    float* sv = sk + AFT_KEYS * LD;                              // [64][LD]
    float* sp = sv + AFT_KEYS * LD;                              // [32][68] scores, then weights
    float* fade = sp + AFT_ROWS * (AFT_KEYS + 4);                // [32] what a row's sums are scaled by this step; at the end its reciprocal
    int* paged = reinterpret_cast<int*>(fade + AFT_ROWS);        // [2][64] whether a key of this step, of the next, has a page: one without is seen by nobody
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kvh = blockIdx.x, tile = gridDim.y - 1 - blockIdx.y;       // later tiles of a prompt see more keys: they start first
    const int group = p.hq / p.hkv;
    const int row0 = p.tile_row0[tile], nq = p.tile_nq[tile], entry = p.tile_entry[tile];
    const int rows_valid = nq * group;
    const int c_first = p.row_count[row0];
    const int klo = (p.window > 0 && c_first > p.window) ? c_first - p.window : 0;
    const int khi = c_first > 0 ? c_first + nq - 1 : 0;          // a padding row sees nothing
    constexpr int stride = AFT_KEYS * PARTS;
    const int part = PARTS == 1 ? 0 : blockIdx.z, from_key = klo + part * AFT_KEYS;      // this block's steps
    auto fetch = [&](float* to, const float* table, int k0) {
        for (int key = warp; key < AFT_KEYS; key += AFT_THREADS / 32) {      // a warp a line; keys nobody sees are zeros
            const int pos = k0 + key, lp = pos / p.page_size;
            int page = -1;
            if (pos < khi && lp < p.table_width) page = p.block_table[(size_t)entry * p.table_width + lp];
            const bool there = page >= 0 && page < p.n_pages;
            if (table == p.k_table && lane == 0) paged[((k0 - klo) / stride & 1) * AFT_KEYS + key] = there;
            const float* from = there ? table + kv_row((long long)page * p.page_size + pos % p.page_size, kvh, p.hkv, p.page_size) * D : table;
            for (int x = lane; x < D4; x += 32)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(to + key * LD + x * 4)), "l"(from + x * 4), "r"(there ? 16 : 0) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int i = tid; i < AFT_ROWS * D4; i += AFT_THREADS) {
        const int r = i / D4, x = (i - r * D4) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < rows_valid) v = *reinterpret_cast<const float4*>(p.q + ((size_t)(row0 + r / group) * p.hq + kvh * group + r % group) * D + x);
        *reinterpret_cast<float4*>(sq + r * LD + x) = v;
    }
    // This warp's four rows of the weighted sum see the keys [lo4, hi4). A weight of zero times a value that is no finite number is no
    // zero, so where not every row sees every key of a step the others are left out of the sum.
    int lo4[4], hi4[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = 4 * warp + i;
        hi4[i] = r < rows_valid ? c_first + r / group : 0;
        lo4[i] = p.window > 0 ? max(0, hi4[i] - p.window) : 0;
    }
    const int all_from = p.window > 0 ? max(0, khi - p.window) : 0;      // every row sees the keys [all_from, c_first)
    // the row whose softmax this thread shares with its seven neighbours
    const int sr = tid >> 3, sc = tid & 7;
    const bool own = sr < rows_valid;
    const int cnt = own ? c_first + sr / group : 0;
    const int fst = (own && p.window > 0 && cnt > p.window) ? cnt - p.window : 0;
    float m = -INFINITY, l = 0.f, l_near = 0.f, l_fade = 1.f;
    const int qy = tid >> 4, qx = tid & 15;                      // scores: rows 2 qy and 2 qy + 1, keys qx + 16 j
    // Sums over the keys of rows 4 warp .. + 3: a step's 64 keys, those of up to four steps, and all before; o is still to be scaled by o_fade.
    float o[4][4 * CG] = {}, near[4][4 * CG] = {}, o_fade[4] = {1.f, 1.f, 1.f, 1.f};
    auto gather = [&]() {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int c = 0; c < 4 * CG; ++c) o[i][c] = fmaf(o[i][c], o_fade[i], near[i][c]), near[i][c] = 0.f;
            o_fade[i] = 1.f;
        }
        l = fmaf(l, l_fade, l_near), l_near = 0.f, l_fade = 1.f;
    };
    if (from_key < khi) {
        fetch(sk, p.k_table, from_key);
        fetch(sv, p.v_table, from_key);
    }
    for (int k0 = from_key; k0 < khi; k0 += stride) {
        const bool more = k0 + stride < khi;
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                                         // the keys are there
        {
            float s[2][4] = {}, half[2][4] = {};
#pragma unroll 1
            for (int x0 = 0; x0 < D; x0 += 32) {                 // 32 components in four chains of eight; pieces meet in pairs
                float4 c[2][4] = {};
#pragma unroll 4
                for (int x = x0; x < x0 + 32; x += 4) {
                    const float4 a = *reinterpret_cast<const float4*>(sq + (2 * qy) * LD + x), b = *reinterpret_cast<const float4*>(sq + (2 * qy + 1) * LD + x);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float4 k = *reinterpret_cast<const float4*>(sk + (qx + 16 * j) * LD + x);
                        c[0][j].x = fmaf(a.x, k.x, c[0][j].x), c[0][j].y = fmaf(a.y, k.y, c[0][j].y), c[0][j].z = fmaf(a.z, k.z, c[0][j].z), c[0][j].w = fmaf(a.w, k.w, c[0][j].w);
                        c[1][j].x = fmaf(b.x, k.x, c[1][j].x), c[1][j].y = fmaf(b.y, k.y, c[1][j].y), c[1][j].z = fmaf(b.z, k.z, c[1][j].z), c[1][j].w = fmaf(b.w, k.w, c[1][j].w);
                    }
                }
                const bool second = x0 & 32;
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float piece = (c[i][j].x + c[i][j].y) + (c[i][j].z + c[i][j].w);
                        s[i][j] += second ? half[i][j] + piece : 0.f;
                        half[i][j] = piece;
                    }
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) sp[(2 * qy + i) * (AFT_KEYS + 4) + qx + 16 * j] = s[i][j];
        }
        __syncthreads();                                         // the scores are there, the keys are done with
        if (more) fetch(sk, p.k_table, k0 + stride);
        else asm volatile("cp.async.commit_group;" ::: "memory");
        {
            float w[8], top = -INFINITY;
            const int* there = paged + ((k0 - klo) / stride & 1) * AFT_KEYS;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int key = k0 + sc + 8 * j;
                float x = sp[sr * (AFT_KEYS + 4) + sc + 8 * j] * p.scale;
                if (p.cap > 0.f) x = p.cap * tanhf(x / p.cap);
                w[j] = key >= fst && key < cnt && there[sc + 8 * j] ? x : -INFINITY;
                top = fmaxf(top, w[j]);
            }
#pragma unroll
            for (int d = 1; d < 8; d <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, d));
            const float now = fmaxf(m, top);
            const float f = m == -INFINITY ? 0.f : expf(m - now);
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                w[j] = w[j] == -INFINITY ? 0.f : expf(w[j] - now);
                sum += w[j];
                sp[sr * (AFT_KEYS + 4) + sc + 8 * j] = w[j];
            }
#pragma unroll
            for (int d = 1; d < 8; d <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
            l_near = l_near * f + sum;
            l_fade *= f;
            m = now;
            if (sc == 0) fade[sr] = f;
        }
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                                         // the weights and the values are there
        float now[4][4 * CG] = {};
        auto sum = [&](auto all) {
#pragma unroll 4
            for (int k = 0; k < AFT_KEYS; k += 4) {
                float4 w[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) w[i] = *reinterpret_cast<const float4*>(sp + (4 * warp + i) * (AFT_KEYS + 4) + k);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                    for (int g = 0; g < CG; ++g) {
                        const float4 v = *reinterpret_cast<const float4*>(sv + (k + kk) * LD + 4 * (lane + 32 * g));
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            if (!decltype(all)::value && (k0 + k + kk < lo4[i] || k0 + k + kk >= hi4[i])) continue;      // the same for the whole warp
                            const float x = kk == 0 ? w[i].x : kk == 1 ? w[i].y : kk == 2 ? w[i].z : w[i].w;
                            now[i][4 * g] = fmaf(x, v.x, now[i][4 * g]);
                            now[i][4 * g + 1] = fmaf(x, v.y, now[i][4 * g + 1]);
                            now[i][4 * g + 2] = fmaf(x, v.z, now[i][4 * g + 2]);
                            now[i][4 * g + 3] = fmaf(x, v.w, now[i][4 * g + 3]);
                        }
                    }
            }
        };
        if (k0 >= all_from && k0 + AFT_KEYS <= c_first) sum(std::true_type{});
        else sum(std::false_type{});
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float f = fade[4 * warp + i];
#pragma unroll
            for (int c = 0; c < 4 * CG; ++c) near[i][c] = fmaf(near[i][c], f, now[i][c]);
            o_fade[i] *= f;
        }
        if (((k0 - klo) / stride & 3) == 3) gather();
        __syncthreads();                                         // the values and the weights are done with
        if (more) fetch(sv, p.v_table, k0 + stride);
        else asm volatile("cp.async.commit_group;" ::: "memory");
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    gather();
    if constexpr (PARTS == 2) {
        float* ml = sp;                                          // [2][32] a row's maximum and sum, where scores were
        __syncthreads();                                         // the last step's weights and values have been read
        if (part == 1) {
            if (sc == 0) ml[sr] = m, ml[AFT_ROWS + sr] = l;
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int g = 0; g < CG; ++g)
                    *reinterpret_cast<float4*>(sk + (4 * warp + i) * LD + 4 * (lane + 32 * g)) = make_float4(o[i][4 * g], o[i][4 * g + 1], o[i][4 * g + 2], o[i][4 * g + 3]);
        }
        aft_cluster_sync();
        if (part == 0) {
            if (sc == 0) {                                       // both parts' sums against the larger maximum
                const float m1 = aft_remote(ml + sr, 1), l1 = aft_remote(ml + AFT_ROWS + sr, 1), top = fmaxf(m, m1);
                const float f0 = m == -INFINITY ? 0.f : expf(m - top), f1 = m1 == -INFINITY ? 0.f : expf(m1 - top);
                m = top, l = fmaf(l, f0, l1 * f1);
                ml[sr] = f0, ml[AFT_ROWS + sr] = f1;
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float f0 = ml[4 * warp + i], f1 = ml[AFT_ROWS + 4 * warp + i];
#pragma unroll
                for (int g = 0; g < CG; ++g) {
                    const float4 v = aft_remote_four(sk + (4 * warp + i) * LD + 4 * (lane + 32 * g), 1);
                    o[i][4 * g] = fmaf(o[i][4 * g], f0, v.x * f1), o[i][4 * g + 1] = fmaf(o[i][4 * g + 1], f0, v.y * f1);
                    o[i][4 * g + 2] = fmaf(o[i][4 * g + 2], f0, v.z * f1), o[i][4 * g + 3] = fmaf(o[i][4 * g + 3], f0, v.w * f1);
                }
            }
        }
        aft_cluster_sync();                                      // nobody leaves while its sums are read
        if (part == 1) return;
    }
    if (sc == 0) {
        float inv = 0.f;
        if (l > 0.f) {
            if (p.sinks != nullptr) {                            // the weights were taken against the keys' maximum m
                const float sink = p.sinks[kvh * group + sr % group], top = fmaxf(m, sink), wk = expf(m - top);
                inv = wk / (l * wk + expf(sink - top));
            } else {
                inv = 1.f / l;
            }
        }
        fade[sr] = inv;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = 4 * warp + i;
        if (r >= rows_valid) continue;
        const float inv = fade[r];
        float* dst = p.out + ((size_t)(row0 + r / group) * p.hq + kvh * group + r % group) * D;
#pragma unroll
        for (int g = 0; g < CG; ++g)
            *reinterpret_cast<float4*>(dst + 4 * (lane + 32 * g)) = make_float4(o[i][4 * g] * inv, o[i][4 * g + 1] * inv, o[i][4 * g + 2] * inv, o[i][4 * g + 3] * inv);
    }
}

template <int D, int PARTS>
static int launch_f32_tiles_parts(const F32TileParams& p, int tiles, cudaStream_t s) {
    constexpr int smem = ((AFT_ROWS + 2 * AFT_KEYS) * (D + 4) + AFT_ROWS * (AFT_KEYS + 4) + AFT_ROWS + 2 * AFT_KEYS) * (int)sizeof(float);
    static bool attr_set = false;
    if (!attr_set) {
        if (cudaFuncSetAttribute(attention_f32_tiles_kernel<D, PARTS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
            return fail("attention_f32_tiles: cannot have %d bytes of shared memory", smem);
        attr_set = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.hkv, tiles, PARTS);
    cfg.blockDim = AFT_THREADS;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = PARTS;
    cfg.attrs = attr;
    cfg.numAttrs = PARTS > 1 ? 1 : 0;
    cudaLaunchKernelEx(&cfg, attention_f32_tiles_kernel<D, PARTS>, p);
    return check_launch("attention_f32_tiles");
}

}  // namespace kb

using namespace kb;

extern "C" int kb_attention_f32_tiles_takes(int hq, int hkv, int d) { return (d == 128 || d == 256) && hkv > 0 && hq % hkv == 0 && hq / hkv <= AFT_ROWS; }

// q and out [rows, hq, d] float32, tables [pages, hkv, page_size, d] float32; tiles of at most 32 / (hq / hkv) tokens of one request at
// consecutive positions; `window` 0: every key; `cap` 0: no soft cap; `sinks` [hq] or null; `blocks` a tile, 1 or 2.
extern "C" int kb_attention_f32_tiles(float* out, const float* q, const float* k_table, const float* v_table, const int* block_table, const int* row_count,
                                      const int* tile_entry, const int* tile_row0, const int* tile_nq, int tiles, int rows, int hq, int hkv, int d,
                                      int page_size, int table_width, int n_pages, int window, float scale, float cap, const float* sinks, int blocks, void* stream) {
    KB_REQUIRE(rows >= 0 && tiles >= 0 && tiles <= 65535, "attention_f32_tiles: rows %d, tiles %d", rows, tiles);
    KB_REQUIRE(blocks == 1 || blocks == 2, "attention_f32_tiles: %d blocks a tile", blocks);
    KB_REQUIRE(kb_attention_f32_tiles_takes(hq, hkv, d), "attention_f32_tiles: %d heads over %d of %d are not taken", hq, hkv, d);
    KB_REQUIRE(page_size > 0 && table_width > 0 && n_pages > 0 && window >= 0, "attention_f32_tiles: pages of %d, table width %d, pages %d, window %d", page_size, table_width, n_pages, window);
    KB_REQUIRE((((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_table | (uintptr_t)v_table) & 15) == 0, "attention_f32_tiles: operands must be 16-byte aligned");
    if (rows == 0 || tiles == 0) return 0;
    F32TileParams p = {q, k_table, v_table, block_table, row_count, tile_entry, tile_row0, tile_nq, sinks, out, hq, hkv, page_size, table_width, n_pages, window, scale, cap};
    cudaStream_t s = (cudaStream_t)stream;
    if (d == 128) return blocks == 2 ? launch_f32_tiles_parts<128, 2>(p, tiles, s) : launch_f32_tiles_parts<128, 1>(p, tiles, s);
    return blocks == 2 ? launch_f32_tiles_parts<256, 2>(p, tiles, s) : launch_f32_tiles_parts<256, 1>(p, tiles, s);
}
