// What the prompt path of latent attention needs around its products: the cached lines of whole requests laid out densely (the
// input of the product that makes every head's keys and values of them), and the queries in the attention kernel's type.
// Both only move values: memory bounds them.
#include <algorithm>
#include "common.cuh"

namespace kb {

typedef __nv_bfloat16 bf16;

// Lines [kv_rank + rot] of the positions 0 .. length - 1 of each request, the latent into c [positions, kv_rank], the rotated part into
// rot_keys [positions, rot], rows entry_base[e] + position; zeros behind them up to a multiple of `align` rows. A position without a page
// gives zeros. 16 bytes a thread.
__global__ void latent_gather_kernel(const uint4* __restrict__ table, const int* __restrict__ block_table, int table_width, int n_pages,
                                     int page_size, const int* __restrict__ entry_base, const int* __restrict__ entry_length, int align,
                                     uint4* __restrict__ c, uint4* __restrict__ rot_keys, int c_pieces, int rot_pieces) {
    const int entry = blockIdx.y;
    const int pieces = c_pieces + rot_pieces;
    const int length = entry_length[entry];
    const long long total = (long long)((length + align - 1) / align * align) * pieces;
    const size_t base = (size_t)entry_base[entry];
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const int pos = (int)(i / pieces), at = (int)(i - (long long)pos * pieces);
        const int lp = pos / page_size;
        const int page = pos < length && lp < table_width ? block_table[(size_t)entry * table_width + lp] : -1;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (page >= 0 && page < n_pages) v = table[((size_t)page * page_size + pos % page_size) * pieces + at];
        if (at < c_pieces) c[(base + pos) * c_pieces + at] = v;
        else rot_keys[(base + pos) * rot_pieces + (at - c_pieces)] = v;
    }
}

// q [rows, heads, d + rot] in the attention's type from the product's 32-bit values: the last `rot` components of every head turned in
// pairs (i, i + rot/2) by cos_sin [rows, rot/2]. A thread: two neighbouring components, or two neighbouring pairs.
template <typename TS>
__global__ void latent_query_kernel(const Src<TS> src, const float2* __restrict__ cos_sin, bf16* __restrict__ q, int rows, int heads, int d, int rot) {
    const int half = rot >> 1, width = d + rot;
    const int units = (d + half) >> 1;                          // a head's work: d / 2 plain couples, rot / 4 couples of pairs
    const long long total = (long long)rows * heads * units;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const long long rh = i / units;
        const int u = (int)(i - rh * units), r = (int)(rh / heads);
        const size_t base = (size_t)rh * width;
        const int x = 2 * u;
        if (x < d) {
            *reinterpret_cast<__nv_bfloat162*>(q + base + x) = __floats2bfloat162_rn(src.at(base + x), src.at(base + x + 1));
        } else {
            const int j = x - d;                                 // pairs j and j + 1
            float a0 = src.at(base + d + j), a1 = src.at(base + d + j + 1);
            float b0 = src.at(base + d + half + j), b1 = src.at(base + d + half + j + 1);
            rope_rotate(a0, b0, cos_sin[(size_t)r * half + j]);
            rope_rotate(a1, b1, cos_sin[(size_t)r * half + j + 1]);
            *reinterpret_cast<__nv_bfloat162*>(q + base + d + j) = __floats2bfloat162_rn(a0, a1);
            *reinterpret_cast<__nv_bfloat162*>(q + base + d + half + j) = __floats2bfloat162_rn(b0, b1);
        }
    }
}

}  // namespace kb

using namespace kb;

// table [pages, 1, page_size, kv_rank + rot] bfloat16; `longest`: the most positions of any request; c [positions, kv_rank], rot_keys [positions, rot],
// a request's rows followed by zeros up to a multiple of `align`.
extern "C" int kb_latent_gather(void* c, void* rot_keys, const void* table, const int* block_table, int table_width, int n_pages, int page_size,
                                const int* entry_base, const int* entry_length, int entries, int longest, int align, int kv_rank, int rot, void* stream) {
    KB_REQUIRE(align >= 1, "latent_gather: rows up to a multiple of %d", align);
    KB_REQUIRE(entries >= 0 && longest >= 0 && kv_rank > 0 && rot > 0 && kv_rank % 8 == 0 && rot % 8 == 0, "latent_gather: lines of %d + %d (multiples of 8)", kv_rank, rot);
    KB_REQUIRE(table_width > 0 && n_pages > 0 && page_size > 0 && entries <= 65535, "latent_gather: table width %d, pages %d of %d, %d requests", table_width, n_pages, page_size, entries);
    KB_REQUIRE(c && rot_keys && table && block_table && entry_base && entry_length, "latent_gather: a null input");
    KB_REQUIRE((((uintptr_t)c | (uintptr_t)rot_keys | (uintptr_t)table) & 15) == 0, "latent_gather: tensors must be 16-byte aligned");
    if (entries == 0 || longest == 0) return 0;
    const long long work = (long long)longest * ((kv_rank + rot) / 8);
    const unsigned blocks = (unsigned)std::min<long long>((work + 255) / 256, 4096);
    latent_gather_kernel<<<dim3(blocks, entries), 256, 0, (cudaStream_t)stream>>>((const uint4*)table, block_table, table_width, n_pages, page_size,
                                                                                   entry_base, entry_length, align, (uint4*)c, (uint4*)rot_keys, kv_rank / 8, rot / 8);
    return check_launch("latent_gather");
}

// src: float32 or bfloat16, maybe split-K partial sums, [rows, heads (d + rot)]; q bfloat16.
extern "C" int kb_latent_query(void* q, const void* src, int in_dt, int splits, long long split_stride, const float* cos_sin, int rows, int heads,
                               int d, int rot, void* stream) {
    KB_REQUIRE(rows >= 0 && heads > 0 && d > 0 && d % 2 == 0 && rot > 0 && rot % 4 == 0, "latent_query: rows %d, heads %d of %d + %d", rows, heads, d, rot);
    KB_REQUIRE(splits >= 1 && (splits == 1 || split_stride >= (long long)rows * heads * (d + rot)), "latent_query: %d slices %lld apart", splits, split_stride);
    KB_REQUIRE(((uintptr_t)q & 3) == 0 && cos_sin != nullptr, "latent_query: an aligned output and a table are needed");
    if (rows == 0) return 0;
    const long long work = (long long)rows * heads * ((d + rot / 2) / 2);
    const unsigned blocks = (unsigned)std::min<long long>((work + 255) / 256, multiprocessors() * 16);
    if (in_dt == KB_DT_F32) latent_query_kernel<float><<<blocks, 256, 0, (cudaStream_t)stream>>>(Src<float>{(const float*)src, splits, (size_t)split_stride}, (const float2*)cos_sin, (bf16*)q, rows, heads, d, rot);
    else if (in_dt == KB_DT_BF16) latent_query_kernel<bf16><<<blocks, 256, 0, (cudaStream_t)stream>>>(Src<bf16>{(const bf16*)src, splits, (size_t)split_stride}, (const float2*)cos_sin, (bf16*)q, rows, heads, d, rot);
    else return fail("latent_query: dtype code %d is not known", in_dt);
    return check_launch("latent_query");
}
