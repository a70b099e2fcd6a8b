// Attention of prompt portions on the fifth-generation tensor cores (bfloat16) where nothing bounds the scores: layers without
// a soft cap, with or without a window and a sink, and the expanded heads of latent attention, whose keys and values differ in size.
//
// One block takes 128 rows -- (token, query head) pairs of one kv head -- and walks its keys 128 at a time:
//   S = Q K^T      tcgen05.mma, Q [128 x DQK] and the key tile [128 x DQK] K-major in shared memory (128-byte swizzle), S
//                  [128 x 128] float32 in one of three TMEM buffers;
//   P = exp(S scale - m), masked, by eight warps, two to each quarter of the rows, half of the tile's keys each; written back
//                  over S as bfloat16;
//   O += P V       tcgen05.mma with P as the A operand straight from TMEM, the value tile [128 x DV] an MN-major B operand; O
//                  [128 x DV] float32 stays in TMEM.
// m is a row's reference, its largest score so far. When a tile raises it, the warps of the row's quarter wait until
// the product of the tile before has gone through, scale their rows of O in TMEM and go on: the product of this tile cannot
// start before their P is there, so nobody else touches O meanwhile. Letting m lag by up to 2^8 would save most of these waits and less than
// 0.5 % of a prompt's pass, but then the largest weight of a row is no power of two and is rounded: an error up to 1.24 times as large where one
// key has nearly all the weight. The row's sum adds up the rounded P, as the product does.
//
// What bounds it: a tile takes 64 clocks a 16-element step, (DQK + DV) / 16 of them, on the tensor cores and 1,024 clocks of
// exponentials (16 a clock a multiprocessor). 2,048 tokens, 16 heads of 192 / 128: 49 us (440 Tflop/s; the kernel over shared lines
// took 867 us and the two products a head around it 248); 16 heads over 4 of 128: 44 us (the mma.sync kernel: 111). A launch of 256
// blocks is 1.7 waves, and a block of few tiles spends most of its time on what precedes its first product and follows its last.
//
// Keys and values come from the paged cache (boxes of 16 keys x 64 elements, four warps asking, a half of the keys or values each) or,
// DENSE, from matrices with a row a position and a head's components side by side (boxes of 128 keys x 64 elements): the heads'
// keys and values that latent attention makes of its lines, with one rotated part [position, 64] for all heads as the last chunk of a key.
// Warps: 0 and 12 ask for keys, 11 and 13 for values; 1 allocates TMEM and issues the score products; 2-9 softmax and epilogue; 10
// issues the P V products. Every wait gives up after about a second, raises a flag that `kb_attention_flash_error` reports, and the
// block still meets at its final barrier, frees its TMEM and returns.
#include "attention_tc.cuh"
#include "common.cuh"
#include "tensor_map.cuh"

namespace kb {

typedef __nv_bfloat16 bf16;

constexpr int AF_ROWS = 128, AF_KEYS = 128, AF_THREADS = 448, AF_S_BUFS = 3;
constexpr int AF_WARP_PV = 10, AF_WARP_V = 11, AF_WARP_K2 = 12, AF_WARP_V2 = 13;

__device__ int g_attention_flash_error = 0;

struct FlashParams {
    const bf16* q;             // [rows, hq, DQK]
    const int* block_table;    // [entries, table_width] (paged)
    const int* entry_base;     // [entries] row of an entry's position 0 in the dense matrices
    const int* row_count;      // [rows]
    const int* tile_entry;     // [tiles]
    const int* tile_row0;      // [tiles]
    const int* tile_nq;        // [tiles]
    const float* sinks;        // [hq] or null
    void* out;                 // [rows, hq, DV]
    float* partial;            // [rows, hq, slots, DV + 2] when slots > 1: (sum p v, m, sum p)
    int rows, hq, hkv, page_size, table_width, n_pages;
    int window, split, slots;
    float scale;
    int v_col;                 // dense: the column of head 0's values in the matrix that `map_v` sees
};

template <int DQK, int DV> struct FlashCfg {
    static constexpr int QB = DQK / 64, VB = DV / 64;            // chunks of 64 elements
    static constexpr int K_BYTES = AF_KEYS * DQK * 2, V_BYTES = AF_KEYS * DV * 2, Q_BYTES = AF_ROWS * DQK * 2;
    static constexpr int K_SLOTS = DQK <= 64 ? 4 : 2, V_SLOTS = DQK <= 64 ? 4 : (DQK <= 128 ? 3 : 2);
    static constexpr int COL_O = 0, COL_S = DV, TMEM_COLS = 512;
    static constexpr int RING = K_SLOTS * K_BYTES + V_SLOTS * V_BYTES;
    static constexpr int SMEM = Q_BYTES + RING + 1024 /* alignment */ + 256 /* barriers */ + 2 * 2 * AF_ROWS * 4 /* maxima, sums */;
    static_assert(DV + AF_S_BUFS * AF_KEYS <= TMEM_COLS, "O and the S buffers outgrew TMEM");
    static_assert((2 * (K_SLOTS + V_SLOTS) + 3 * AF_S_BUFS + 1) * 8 + 8 <= 256, "the barriers outgrew their room");
    static_assert(SMEM <= 232448, "more shared memory than a block can have");
};

template <int DQK, int DV, bool DENSE, typename TOUT>
__global__ void __launch_bounds__(AF_THREADS, 1)
attention_flash_kernel(const FlashParams p, const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_rot,
                       const __grid_constant__ CUtensorMap map_v) {
    using C = FlashCfg<DQK, DV>;
    constexpr int QB = C::QB, VB = C::VB, KS = C::K_SLOTS, VS = C::V_SLOTS, SB = AF_S_BUFS;
    constexpr int WARPS_A_SLOT = DENSE ? 1 : 2;                  // warps that bring a tile of keys (or of values)
    extern __shared__ unsigned char af_smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)af_smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* q_smem = smem;                                // [chunk][128 rows][128 bytes]
    unsigned char* k_ring = smem + C::Q_BYTES;                   // slots of [chunk][128 keys][128 bytes]
    unsigned char* v_ring = k_ring + KS * C::K_BYTES;            // the same of values
    uint64_t* k_full = reinterpret_cast<uint64_t*>(smem + C::Q_BYTES + C::RING);
    uint64_t* k_empty = k_full + KS;
    uint64_t* v_full = k_empty + KS;
    uint64_t* v_empty = v_full + VS;
    uint64_t* s_full = v_empty + VS;                             // [SB] S complete
    uint64_t* p_full = s_full + SB;                              // [SB] P written, eight warps arrive
    uint64_t* s_free = p_full + SB;                              // [SB] the product that read P is complete
    uint64_t* o_full = s_free + SB;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 1);
    float* exchange = reinterpret_cast<float*>(smem + C::Q_BYTES + C::RING + 256);      // [2][2][128]: a tile's maxima by (turn, half, row)

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kvh = blockIdx.x, slot = blockIdx.y;
    const int tile = gridDim.z - 1 - blockIdx.z;                 // later tiles of a prompt see more keys: they start first
    const int group = p.hq / p.hkv;
    const int row0 = p.tile_row0[tile], nq = p.tile_nq[tile];
    const int entry = p.tile_entry[tile];
    const int rows_valid = nq * group;
    const int c_first = p.row_count[row0];
    int klo = (p.window > 0 && c_first > p.window) ? c_first - p.window : 0;
    int khi = c_first > 0 ? c_first + nq - 1 : 0;                // a padding row sees nothing
    if (p.split > 0) {
        klo = max(klo, slot * p.split);
        khi = min(khi, (slot + 1) * p.split);
    }
    TOUT* out = static_cast<TOUT*>(p.out);
    if (klo >= khi) {                                            // nothing for this block: before anything is allocated
        if (p.slots == 1 && c_first <= 0)
            for (int i = tid; i < rows_valid * DV; i += AF_THREADS) {
                const int r = i / DV, c = i % DV;
                Elem<TOUT>::store(out + ((size_t)(row0 + r / group) * p.hq + kvh * group + r % group) * DV + c, 0.f);
            }
        return;
    }
    const int k_begin = klo / AF_KEYS * AF_KEYS;
    const int n_tiles = (khi - k_begin + AF_KEYS - 1) / AF_KEYS;

    if (tid == 0) {
        for (int s = 0; s < KS; ++s) { at_mbar_init(k_full + s, WARPS_A_SLOT); at_mbar_init(k_empty + s, 1); }
        for (int s = 0; s < VS; ++s) { at_mbar_init(v_full + s, WARPS_A_SLOT); at_mbar_init(v_empty + s, 1); }
        for (int b = 0; b < SB; ++b) { at_mbar_init(s_full + b, 1); at_mbar_init(p_full + b, 8); at_mbar_init(s_free + b, 1); }
        at_mbar_init(o_full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(at_saddr(tmem_slot)), "r"(C::TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // Q, K-major under the 128-byte swizzle: chunk c (64 elements) of row r at c * 16 KB + r * 128, its 16-byte pieces
    // exchanged by r mod 8. Eight neighbouring threads bring a row's 128 bytes.
    for (int i = tid; i < AF_ROWS * QB * 8; i += AF_THREADS) {
        const int j = i & 7, r = (i >> 3) % AF_ROWS, c = (i >> 3) / AF_ROWS;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (r < rows_valid) v = *reinterpret_cast<const uint4*>(p.q + ((size_t)(row0 + r / group) * p.hq + kvh * group + r % group) * DQK + c * 64 + j * 8);
        *reinterpret_cast<uint4*>(q_smem + (size_t)c * (AF_ROWS * 128) + (size_t)r * 128 + ((j ^ (r & 7)) << 4)) = v;
    }
    at_fence_async_smem();
    at_fence_before();
    __syncthreads();
    at_fence_after();
    const uint32_t tmem = *tmem_slot;
    bool failed = false;

    const bool brings_keys = warp == 0 || (!DENSE && warp == AF_WARP_K2), brings_values = warp == AF_WARP_V || (!DENSE && warp == AF_WARP_V2);
    if (DENSE && (brings_keys || brings_values)) {
        // ---------------------------------------------------------------- dense keys or values: a box a chunk, from one lane
        if (lane == 0) {
            const int base = p.entry_base[entry];
            for (int kt = 0; kt < n_tiles; ++kt) {
                const int s = brings_keys ? kt % KS : kt % VS, round = brings_keys ? kt / KS : kt / VS;
                uint64_t* full = (brings_keys ? k_full : v_full) + s;
                if (!at_mbar_wait((brings_keys ? k_empty : v_empty) + s, ((uint32_t)round & 1u) ^ 1u)) { failed = true; break; }
                const int row = base + k_begin + kt * AF_KEYS;   // the last tile's keys behind the request's end: zeros (`latent_gather`)
                at_mbar_expect_tx(full, brings_keys ? C::K_BYTES : C::V_BYTES);
                if (brings_keys) {
                    const uint32_t dst = at_saddr(k_ring) + (uint32_t)s * C::K_BYTES;
                    for (int c = 0; c < QB - 1; ++c) at_tma_box(dst + (uint32_t)c * (AF_KEYS * 128), &map_k, kvh * (DQK - 64) + c * 64, row, full);
                    at_tma_box(dst + (uint32_t)(QB - 1) * (AF_KEYS * 128), &map_rot, 0, row, full);
                } else {
                    const uint32_t dst = at_saddr(v_ring) + (uint32_t)s * C::V_BYTES;
                    for (int c = 0; c < VB; ++c) at_tma_box(dst + (uint32_t)c * (AF_KEYS * 128), &map_v, p.v_col + kvh * DV + c * 64, row, full);
                }
            }
        }
    } else if (brings_keys || brings_values) {
        // ---------------------------------------------------------------- paged: eight pages of 16 keys a tile, four of them this warp's
        const bool second = warp == AF_WARP_K2 || warp == AF_WARP_V2;
        const int NB = brings_keys ? QB : VB;
        // The pages of four tiles are looked up at once, lane 8 t + sub for keys 16 sub .. of tile t, one batch ahead of their use. Values
        // of a group without a page (before the window, past the end) are cleared: 0 * garbage could be NaN.
        auto lookup = [&](int kt_first) -> int {
            const int kt = kt_first + (lane >> 3);
            const int j = k_begin + kt * AF_KEYS + (lane & 7) * 16;
            int page = -1;
            if (kt < n_tiles && j < khi && j + 16 > klo) {
                const int lp = max(j, klo) / p.page_size;
                if (lp < p.table_width) page = p.block_table[(size_t)entry * p.table_width + lp];
                if (page >= p.n_pages) page = -1;
            }
            return page;
        };
        int pages_now = 0, pages_next = lookup(0);
        for (int kt = 0; kt < n_tiles; ++kt) {
            if ((kt & 3) == 0) { pages_now = pages_next; pages_next = lookup(kt + 4); }
            const int j0 = k_begin + kt * AF_KEYS;
            const int page = __shfl_sync(0xffffffffu, pages_now, (kt & 3) * 8 + (lane & 7));
            const uint32_t have = (__ballot_sync(0xffffffffu, page >= 0) >> (second ? 4 : 0)) & 0xFu;      // this warp's four groups
            const int s = brings_keys ? kt % KS : kt % VS, round = brings_keys ? kt / KS : kt / VS;
            uint64_t* full = (brings_keys ? k_full : v_full) + s;
            bool ok = true;
            if (lane == 0) ok = at_mbar_wait((brings_keys ? k_empty : v_empty) + s, ((uint32_t)round & 1u) ^ 1u);
            if (!__shfl_sync(0xffffffffu, ok ? 1 : 0, 0)) { failed = true; break; }
            unsigned char* dst = (brings_keys ? k_ring + s * C::K_BYTES : v_ring + s * C::V_BYTES) + (second ? 4 * 2048 : 0);
            if (brings_values && have != 0xFu) {
                for (int sub = 0; sub < 4; ++sub) {
                    if (have & (1u << sub)) continue;
                    for (int e = lane; e < NB * 128; e += 32)    // 128 pieces of 16 bytes a chunk
                        *reinterpret_cast<uint4*>(dst + (size_t)(e >> 7) * (AF_KEYS * 128) + sub * 2048 + (e & 127) * 16) = make_uint4(0u, 0u, 0u, 0u);
                }
                at_fence_async_smem();
                __syncwarp();
            }
            if (lane == 0) at_mbar_expect_tx(full, (uint32_t)(__popc(have) * NB) * 2048u);
            __syncwarp();
            const int sub = lane & 3, bx = lane >> 2;            // a box a lane: 4 groups x NB chunks
            const int pg = __shfl_sync(0xffffffffu, page, sub + (second ? 4 : 0));
            if (bx < NB && pg >= 0) {
                const int j = j0 + (sub + (second ? 4 : 0)) * 16;
                const int row = (pg * p.hkv + kvh) * p.page_size + j % p.page_size;
                at_tma_box(at_saddr(dst) + (uint32_t)bx * (AF_KEYS * 128) + (uint32_t)sub * 2048u, brings_keys ? &map_k : &map_v, bx * 64, row, full);
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- the score products: the whole warp walks, see at_elect()
        const uint32_t one = at_elect(), tm = __shfl_sync(0xffffffffu, tmem, 0);
        constexpr uint32_t IDESC_S = at_idesc(AF_ROWS, AF_KEYS, false);
        const uint32_t q_addr = at_saddr(q_smem), ring_addr = at_saddr(k_ring);
        for (int kt = 0; kt < n_tiles; ++kt) {
            const int s = kt % KS, b = kt % SB;
            if (!__all_sync(0xffffffffu, at_mbar_wait(k_full + s, (uint32_t)(kt / KS) & 1u))) { failed = true; break; }
            // the buffer still holds tile kt - SB's P until the product that reads it is complete
            if (kt >= SB && !__all_sync(0xffffffffu, at_mbar_wait(s_free + b, (uint32_t)(kt / SB - 1) & 1u))) { failed = true; break; }
            at_fence_after();
            const uint32_t d_tmem = tm + (uint32_t)(C::COL_S + b * AF_KEYS);
#pragma unroll
            for (int bx = 0; bx < QB; ++bx) {
                const uint64_t adesc = at_desc(q_addr + bx * (AF_ROWS * 128), 16, 1024);
                const uint64_t bdesc = at_desc(ring_addr + (uint32_t)s * C::K_BYTES + bx * (AF_KEYS * 128), 16, 1024);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) at_mma_ss_if(one, d_tmem, adesc + (uint64_t)(kk * 2), bdesc + (uint64_t)(kk * 2), IDESC_S, (bx | kk) != 0 ? 1u : 0u);
            }
            if (one) at_commit(k_empty + s);
            if (one) at_commit(s_full + b);
        }
    } else if (warp == AF_WARP_PV) {
        // ---------------------------------------------------------------- the P V products, likewise
        const uint32_t one = at_elect(), tm = __shfl_sync(0xffffffffu, tmem, 0);
        constexpr uint32_t IDESC_O = at_idesc(AF_ROWS, DV, true);
        const uint32_t ring_addr = at_saddr(v_ring);
        for (int kt = 0; kt < n_tiles; ++kt) {
            const int b = kt % SB, s = kt % VS;
            if (!__all_sync(0xffffffffu, at_mbar_wait(v_full + s, (uint32_t)(kt / VS) & 1u))) { failed = true; break; }
            if (!__all_sync(0xffffffffu, at_mbar_wait(p_full + b, (uint32_t)(kt / SB) & 1u))) { failed = true; break; }
            at_fence_after();
            const uint32_t a_tmem = tm + (uint32_t)(C::COL_S + b * AF_KEYS);          // P lies over its S
#pragma unroll
            for (int kk = 0; kk < AF_KEYS / 16; ++kk) {
                // keys 16 kk ..: their two eight-key groups 1 KB apart, chunks of 64 elements 16 KB apart
                const uint64_t bdesc = at_desc(ring_addr + (uint32_t)s * C::V_BYTES + (uint32_t)kk * 2048u, AF_KEYS * 128, 1024);
                at_mma_ts_if(one, tm + C::COL_O, a_tmem + (uint32_t)(kk * 8), bdesc, IDESC_O, (kt | kk) != 0 ? 1u : 0u);
            }
            if (one) at_commit(v_empty + s);
            if (one) at_commit(s_free + b);
        }
        if (!failed && one) at_commit(o_full);
    } else if (warp >= 2 && warp < 10) {
        // ---------------------------------------------------------------- softmax and epilogue, half a row a thread
        const int quarter = warp & 3;
        const int half = (warp - 2) >> 2;                        // 0: keys 0-63 of a tile (and O's first half), 1: the rest
        const int r = quarter * 32 + lane;                       // the row of the tile, and the TMEM lane
        const bool own = r < rows_valid;
        const int cnt = own ? c_first + r / group : 0;
        const int fst = (own && p.window > 0 && cnt > p.window) ? cnt - p.window : 0;
        const int lo = max(fst, klo), hi = min(cnt, khi);        // this row sees keys [lo, hi) of this block's
        const int lo_max = __reduce_max_sync(0xffffffffu, lo), hi_min = __reduce_min_sync(0xffffffffu, hi);
        const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16);
        const float c = p.scale * 1.4426950408889634f;           // scores in powers of two
        float ref = -INFINITY, l = 0.f;
        for (int kt = 0; kt < n_tiles; ++kt) {
            const int b = kt % SB;
            const int j0 = k_begin + kt * AF_KEYS + half * 64;   // this warp's 64 keys of the tile
            // a wait that ran out is not repeated, but the walk goes on: the quarter's warps meet at every tile's barrier
            if (!failed && !__all_sync(0xffffffffu, at_mbar_wait(s_full + b, (uint32_t)(kt / SB) & 1u))) failed = true;
            at_fence_after();
            uint32_t sa[32], sb[32];                             // keys j0 .. j0 + 31 and j0 + 32 .. j0 + 63
            at_ld32(lanes + (uint32_t)(C::COL_S + b * AF_KEYS + half * 64), sa);
            at_ld32(lanes + (uint32_t)(C::COL_S + b * AF_KEYS + half * 64 + 32), sb);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (j0 < lo_max || j0 + 64 > hi_min) {               // the same for the whole warp
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    if (j0 + j < lo || j0 + j >= hi) sa[j] = 0xff800000u;
                    if (j0 + 32 + j < lo || j0 + 32 + j >= hi) sb[j] = 0xff800000u;
                }
            }
            float top = __uint_as_float(sa[0]), top2 = __uint_as_float(sb[0]);
#pragma unroll
            for (int j = 1; j < 32; ++j) {
                top = fmaxf(top, __uint_as_float(sa[j]));
                top2 = fmaxf(top2, __uint_as_float(sb[j]));
            }
            top = fmaxf(top, top2);
            // The quarter's two warps tell each other their halves' maxima; behind this barrier both have their scores in registers, so P
            // may be written over them. Two sets of places in turn: a warp writes the next tile's only when the other has read this one's.
            float* turn = exchange + (kt & 1) * 2 * AF_ROWS;
            turn[half * AF_ROWS + r] = top;
            asm volatile("bar.sync %0, 64;" ::"r"(2 + quarter) : "memory");
            top = fmaxf(top, turn[(half ^ 1) * AF_ROWS + r]) * c;
            const bool moves = top > ref;
            const float was = ref;
            if (moves) ref = top;
            const float fade = moves ? (was == -INFINITY ? 0.f : at_exp2(was - ref)) : 1.f;      // a row that has seen nothing holds zeros
            l *= fade;
            if (kt > 0 && __any_sync(0xffffffffu, moves && was != -INFINITY)) {
                const int before = kt - 1;
                if (!failed && !__all_sync(0xffffffffu, at_mbar_wait(s_free + before % SB, (uint32_t)(before / SB) & 1u))) failed = true;
                at_fence_after();
                for (int c0 = half * (DV / 2); c0 < (half + 1) * (DV / 2); c0 += 32) {
                    uint32_t o[32];
                    __syncwarp();
                    at_ld32(lanes + (uint32_t)(C::COL_O + c0), o);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * fade);
                    at_st32(lanes + (uint32_t)(C::COL_O + c0), o);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            }
            const float m = ref == -INFINITY ? 0.f : ref;
            float la = 0.f, lb = 0.f;
            uint32_t pr[32];
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
                const float p0 = at_exp2(fmaf(__uint_as_float(sa[j]), c, -m)), p1 = at_exp2(fmaf(__uint_as_float(sa[j + 1]), c, -m));
                const uint32_t w = at_pack(p0, p1);
                la += __uint_as_float(w << 16);
                lb += __uint_as_float(w & 0xffff0000u);
                pr[j >> 1] = w;
            }
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
                const float p0 = at_exp2(fmaf(__uint_as_float(sb[j]), c, -m)), p1 = at_exp2(fmaf(__uint_as_float(sb[j + 1]), c, -m));
                const uint32_t w = at_pack(p0, p1);
                la += __uint_as_float(w << 16);
                lb += __uint_as_float(w & 0xffff0000u);
                pr[16 + (j >> 1)] = w;
            }
            l += la + lb;
            at_st32(lanes + (uint32_t)(C::COL_S + b * AF_KEYS + half * 32), pr);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            at_fence_before();
            __syncwarp();
            if (lane == 0) at_mbar_arrive(p_full + b);
        }
        // The row's sum over both halves: through shared memory, each half's share where its maxima were. Both warps of a quarter meet
        // here whatever happened above.
        asm volatile("bar.sync %0, 64;" ::"r"(2 + quarter) : "memory");
        exchange[half * AF_ROWS + r] = l;
        asm volatile("bar.sync %0, 64;" ::"r"(2 + quarter) : "memory");
        l += exchange[(half ^ 1) * AF_ROWS + r];
        if (!failed && !__all_sync(0xffffffffu, at_mbar_wait(o_full, 0u))) failed = true;
        if (!failed) {
            at_fence_after();
            // With several slots, a row whose keys all lie in one slot is finished by that slot's block.
            const int z0 = p.slots > 1 ? fst / p.split : 0;
            const int z1 = p.slots > 1 ? min(p.slots - 1, (max(cnt, 1) - 1) / p.split) : 0;
            const bool direct = z0 == z1;
            const bool writes = own && (!direct || slot == z0);
            const int row = row0 + r / group, head = kvh * group + r % group;
            float total = l;
            if (p.sinks != nullptr) total += exp2f(own ? p.sinks[head] * 1.4426950408889634f - (ref == -INFINITY ? 0.f : ref) : 0.f);
            const float inv = l > 0.f ? 1.f / total : 0.f;
            TOUT* dst = out + ((size_t)row * p.hq + head) * DV;
            float* pdst = p.partial ? p.partial + (((size_t)row * p.hq + head) * p.slots + slot) * (DV + 2) : nullptr;
            for (int c0 = half * (DV / 2); c0 < (half + 1) * (DV / 2); c0 += 32) {
                uint32_t o[32];
                __syncwarp();
                at_ld32(lanes + (uint32_t)(C::COL_O + c0), o);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (!writes) continue;
                if (!direct) {
#pragma unroll
                    for (int j = 0; j < 32; j += 2)
                        *reinterpret_cast<float2*>(pdst + c0 + j) = make_float2(__uint_as_float(o[j]), __uint_as_float(o[j + 1]));
                } else if constexpr (sizeof(TOUT) == 4) {
#pragma unroll
                    for (int j = 0; j < 32; j += 4)
                        *reinterpret_cast<float4*>(reinterpret_cast<float*>(dst) + c0 + j) =
                            make_float4(__uint_as_float(o[j]) * inv, __uint_as_float(o[j + 1]) * inv, __uint_as_float(o[j + 2]) * inv, __uint_as_float(o[j + 3]) * inv);
                } else {
#pragma unroll
                    for (int j = 0; j < 32; j += 8) {
                        uint4 v;
                        v.x = at_pack(__uint_as_float(o[j]) * inv, __uint_as_float(o[j + 1]) * inv);
                        v.y = at_pack(__uint_as_float(o[j + 2]) * inv, __uint_as_float(o[j + 3]) * inv);
                        v.z = at_pack(__uint_as_float(o[j + 4]) * inv, __uint_as_float(o[j + 5]) * inv);
                        v.w = at_pack(__uint_as_float(o[j + 6]) * inv, __uint_as_float(o[j + 7]) * inv);
                        *reinterpret_cast<uint4*>(dst + c0 + j) = v;
                    }
                }
            }
            if (writes && !direct && half == 0) {
                pdst[DV] = ref == -INFINITY ? -INFINITY : ref * 0.6931471805599453f;
                pdst[DV + 1] = l;
            }
        }
    }
    if (failed) atomicExch(&g_attention_flash_error, 1);
    at_fence_before();
    __syncthreads();
    if (warp == 1) {
        at_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::TMEM_COLS) : "memory");
    }
}

template <int DQK, int DV, bool DENSE, typename TOUT>
static int launch_flash(const FlashParams& p, const CUtensorMap& mk, const CUtensorMap& mr, const CUtensorMap& mv, int tiles, cudaStream_t s) {
    using C = FlashCfg<DQK, DV>;
    static bool attr_set = false;
    if (!attr_set) {
        const cudaError_t e = cudaFuncSetAttribute(attention_flash_kernel<DQK, DV, DENSE, TOUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
        if (e != cudaSuccess) return fail("attention_flash: cannot have %d bytes of shared memory: %s", C::SMEM, cudaGetErrorString(e));
        attr_set = true;
    }
    attention_flash_kernel<DQK, DV, DENSE, TOUT><<<dim3(p.hkv, p.slots, tiles), AF_THREADS, C::SMEM, s>>>(p, mk, mr, mv);
    return check_launch("attention_flash");
}

}  // namespace kb

using namespace kb;

// 1 if a wait inside the kernel ever ran out (and clears the flag); synchronises the device.
extern "C" int kb_attention_flash_error() {
    int flag = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&flag, g_attention_flash_error, sizeof(int)) != cudaSuccess) return -1;
    if (flag) cudaMemcpyToSymbol(g_attention_flash_error, &zero, sizeof(int));
    return flag;
}

// 1 where the kernel takes a paged layer: keys and values of one size, 64 or 128, pages of a multiple of 16 positions, at most 128
// query heads a kv head, a scale above zero (a row's largest score is the largest product).
extern "C" int kb_attention_flash_takes(int hq, int hkv, int d, int page_size, float scale) {
    return (d == 64 || d == 128) && page_size > 0 && page_size % 16 == 0 && hkv > 0 && hq % hkv == 0 && hq / hkv <= AF_ROWS && scale > 0.f;
}

// Prompt portions over the paged cache; arguments as kb_attention_tc's, tiles of 128 rows, `sinks` [hq] or null. With slots > 1 the caller merges
// `scratch` [rows, hq, slots, d + 2] (and the sinks).
extern "C" int kb_attention_flash(void* out, const void* q, const void* k_table, const void* v_table, const int* block_table,
                                  const int* row_count, const int* tile_entry, const int* tile_row0, const int* tile_nq, int tiles,
                                  int rows, int hq, int hkv, int d, int page_size, int table_width, int n_pages, int window,
                                  int split, int slots, float scale, float* scratch, const float* sinks, void* stream) {
    KB_REQUIRE(rows >= 0 && tiles >= 0 && hq > 0 && hkv > 0, "attention_flash: rows %d, tiles %d, heads %d over %d", rows, tiles, hq, hkv);
    KB_REQUIRE(kb_attention_flash_takes(hq, hkv, d, page_size, scale), "attention_flash: head size %d, %d heads over %d, pages of %d, scale %g are not taken",
               d, hq, hkv, page_size, scale);
    KB_REQUIRE(table_width > 0 && n_pages > 0 && window >= 0, "attention_flash: table width %d, pages %d, window %d", table_width, n_pages, window);
    KB_REQUIRE((split == 0 && slots == 1) || (split > 0 && split % 64 == 0 && slots >= 1 && slots <= 65535),
               "attention_flash: split %d (a multiple of 64) with %d slots", split, slots);
    KB_REQUIRE(slots == 1 || scratch != nullptr, "attention_flash: %d slots need scratch memory", slots);
    KB_REQUIRE(tiles <= 65535, "attention_flash: %d tiles is too many for one launch", tiles);
    KB_REQUIRE((((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_table | (uintptr_t)v_table) & 15) == 0, "attention_flash: operands must be 16-byte aligned");
    if (rows == 0 || tiles == 0) return 0;
    FlashParams p = {};
    p.q = (const bf16*)q; p.block_table = block_table; p.row_count = row_count; p.tile_entry = tile_entry; p.tile_row0 = tile_row0;
    p.tile_nq = tile_nq; p.sinks = sinks; p.out = out; p.partial = slots > 1 ? scratch : nullptr; p.rows = rows; p.hq = hq; p.hkv = hkv;
    p.page_size = page_size; p.table_width = table_width; p.n_pages = n_pages; p.window = window; p.split = split; p.slots = slots; p.scale = scale;
    const unsigned long long lines = (unsigned long long)n_pages * hkv * page_size;
    CUtensorMap mk, mv;
    if (int e = encode_map_bf16(&mk, k_table, lines, d, d, 16)) return e;
    if (int e = encode_map_bf16(&mv, v_table, lines, d, d, 16)) return e;
    cudaStream_t s = (cudaStream_t)stream;
    return d == 64 ? launch_flash<64, 64, false, bf16>(p, mk, mk, mv, tiles, s) : launch_flash<128, 128, false, bf16>(p, mk, mk, mv, tiles, s);
}

// 1 where the kernel takes a latent layer's expanded heads: plain keys and values of 128 components, a rotated part of 64.
extern "C" int kb_attention_flash_latent_takes(int hq, int d, int rot, int dv, float scale) {
    return hq > 0 && d == 128 && rot == 64 && dv == 128 && scale > 0.f;
}

// Prompt portions over dense keys and values. q [rows, hq, d + rot] bfloat16; kv [positions, hq d + hq dv]: a position's plain keys of all
// heads, then its values; rot_keys [positions, rot]; `entry_base` [entries]: the row of an entry's position 0; tiles of 128 rows.
// out [rows, hq, dv] float32.
extern "C" int kb_attention_flash_latent(float* out, const void* q, const void* kv, const void* rot_keys, const int* entry_base, int positions,
                                         const int* row_count, const int* tile_entry, const int* tile_row0, const int* tile_nq, int tiles, int rows,
                                         int hq, int d, int rot, int dv, float scale, const float* sinks, void* stream) {
    KB_REQUIRE(rows >= 0 && tiles >= 0 && positions > 0, "attention_flash_latent: rows %d, tiles %d, positions %d", rows, tiles, positions);
    KB_REQUIRE(kb_attention_flash_latent_takes(hq, d, rot, dv, scale), "attention_flash_latent: %d heads of %d + %d and %d, scale %g are not taken", hq, d, rot, dv, scale);
    KB_REQUIRE(tiles <= 65535, "attention_flash_latent: %d tiles is too many for one launch", tiles);
    KB_REQUIRE((((uintptr_t)q | (uintptr_t)out | (uintptr_t)kv | (uintptr_t)rot_keys) & 15) == 0, "attention_flash_latent: operands must be 16-byte aligned");
    if (rows == 0 || tiles == 0) return 0;
    FlashParams p = {};
    p.q = (const bf16*)q; p.entry_base = entry_base; p.row_count = row_count; p.tile_entry = tile_entry; p.tile_row0 = tile_row0; p.tile_nq = tile_nq;
    p.sinks = sinks; p.out = out; p.rows = rows; p.hq = hq; p.hkv = hq; p.slots = 1; p.scale = scale; p.v_col = hq * d;
    const unsigned long long width = (unsigned long long)hq * (d + dv);
    CUtensorMap mk, mr;
    if (int e = encode_map_bf16(&mk, kv, positions, width, width, AF_KEYS)) return e;
    if (int e = encode_map_bf16(&mr, rot_keys, positions, rot, rot, AF_KEYS)) return e;
    return launch_flash<192, 128, true, float>(p, mk, mr, mk, tiles, (cudaStream_t)stream);
}
