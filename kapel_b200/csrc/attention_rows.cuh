// (shared by attention_f32.cu and attention_bf16.cu)
// Attention over the paged cache, one query row at a time ("rows" kernels), for any element
// type. A query row that has seen c positions (its own included) reads keys
// [max(0, c - window), c) of its sequence through the block table, and with `keep` > 0 also the
// keys [0, keep) that lie below its window; with `block` > 0 only the keys of its own block of that
// many positions (blocks are counted from position 0); score = scale * q.k, then
// cap * tanh(score / cap) if a cap is given, softmax over what it sees, weighted sum of values;
// a row that sees nothing gives zeros. Scores, soft cap, softmax and sums are 32-bit.
//
// Kapel's counterparts: kernels/src/lib.rs paged_attention :1850, paged_combine :2135; rules in
// crates/kapel-ops/src/paged.rs:16-25,65-70.
//
// One block = one row x one kv head (a slice of up to GMAX of its query heads) x one chunk of
// CHUNK key positions. Chunks are cut at absolute multiples of CHUNK, so what a row computes
// does not depend on the rest of the batch. With more than one chunk slot the blocks write
// (sum p.v, max, sum p) to scratch memory and `combine_kernel` merges them in slot order. The
// first `keep_slots` slots are the kept first keys' chunks, the others the window's. Values may
// have another size than keys (`dv`), and may lie `v_stride` apart: a value table that is the key
// table itself, whose first `dv` components of a line are the value (attention through a latent).
// With `sinks`, e^(sinks[head]) joins a row's denominator: a key without a value, not scaled.
//
// A chunk's keys and values are waited for, not the arithmetic: a key's place in the tables is divided out once into shared memory (by every thread that
// read it the 64-bit divisions were most of the time), and eight keys and values are asked for before the first is used. 32-bit, 8 heads over 4 of
// 256: 4 tokens behind 500 positions 231 -> 46 us, 128 behind 1,024 372 -> 205.
#pragma once
#include "common.cuh"

namespace kb {

constexpr int ATT_CHUNK = 256;
constexpr int ATT_THREADS = 128;
constexpr int ATT_WARPS = ATT_THREADS / 32;

// exp for the softmax: the library's in the 32-bit path, the fast one otherwise.
template <typename T> __device__ __forceinline__ float soft_exp(float x) { return __expf(x); }
template <> __device__ __forceinline__ float soft_exp<float>(float x) { return expf(x); }

template <typename T> struct Vec;      // 16 bytes of T
template <> struct Vec<float> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void load(const float* p, float (&out)[4]) {
        const float4 v = *reinterpret_cast<const float4*>(p);
        out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
    }
};
template <> struct Vec<__nv_bfloat16> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void load(const __nv_bfloat16* p, float (&out)[8]) {
        const uint4 v = *reinterpret_cast<const uint4*>(p);
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            out[2 * i] = __uint_as_float(u[i] << 16);
            out[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
        }
    }
};

struct AttParams {
    const void* q;            // [rows, hq, d]
    const void* k_table;      // [pages, hkv, page_size, d]
    const void* v_table;
    const int* block_table;   // [entries, table_width]
    const int* row_entry;     // [rows]
    const int* row_count;     // [rows]
    void* out;                // [rows, hq, dv]
    float* partial;           // [rows, hq, slots, dv + 2] or null when slots == 1
    int rows, hq, hkv, d, page_size, table_width, n_pages;
    int dv;                   // the values' size (the v table is [pages, hkv, page_size, v_stride])
    int v_stride;             // elements between two lines' values (dv, or more when values lie inside wider lines)
    const float* sinks;       // [hq] or null: a term e^sink in the denominator of every row of the head
    int vec;                  // 1: a key is a whole number of 16-byte pieces and is loaded as such
    int window;               // 0: none
    int block;                // > 0: a row at position i sees only the keys from floor(i / block) * block on (blocks counted from position 0)
    int keep;                 // with a window: the keys [0, keep) stay visible below it
    int keep_slots;           // ceil(keep / CHUNK) with a window and keep > 0, else 0: the slots of those keys
    int slots;                // chunk slots a row may touch, the kept keys' included
    int chunk;                // keys a slot holds: ATT_CHUNK for the row-wise kernel (its shared memory is made for that); another kernel may cut longer
    float scale, cap;         // cap 0: none
};

// The keys [lo, hi) that slot z of a row with `count` positions holds (empty when hi <= lo): the
// first `keep_slots` slots are chunks of the kept first keys below the window's start, the others
// the window's chunks, counted from the chunk that holds its first key.
__device__ __forceinline__ void slot_range(const AttParams& p, int count, int z, int& lo, int& hi) {
    int first = (p.window > 0 && count > p.window) ? count - p.window : 0;
    if (p.block > 0 && count > 0) first = max(first, (count - 1) / p.block * p.block);
    if (z < p.keep_slots) {
        lo = z * p.chunk;
        hi = min(min(p.keep, first), (z + 1) * p.chunk);
    } else {
        const int chunk = first / p.chunk + (z - p.keep_slots);       // absolute chunk index
        lo = max(first, chunk * p.chunk);
        hi = min(count, (chunk + 1) * p.chunk);
    }
}

// LPK: lanes that share one key (a power of two); VPL: 16-byte vectors of a key each lane holds.
template <typename T, int GMAX, int LPK, int VPL>
__global__ void __launch_bounds__(ATT_THREADS)
rows_kernel(const AttParams p) {
    constexpr int VN = Vec<T>::N;
    extern __shared__ __align__(16) float smem[];
    const int group = p.hq / p.hkv;
    const int gslices = (group + GMAX - 1) / GMAX;
    const int r = blockIdx.x;
    const int kvh = blockIdx.y / gslices;
    const int g0 = (blockIdx.y % gslices) * GMAX;
    const int gn = min(GMAX, group - g0);                 // query heads of this block
    const int d = p.d;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    const int count = p.row_count[r];
    int lo, hi;
    slot_range(p, count, blockIdx.z, lo, hi);
    const int nkeys = hi - lo;
    const int dv = p.dv;
    T* out = static_cast<T*>(p.out);

    if (nkeys <= 0) {
        // Nothing in this slot. The first slot of a row that sees nothing at all writes zeros.
        if (blockIdx.z == 0 && count <= 0)
            for (int g = 0; g < gn; ++g)
                for (int i = tid; i < dv; i += ATT_THREADS)
                    Elem<T>::store(out + ((size_t)r * p.hq + kvh * group + g0 + g) * dv + i, 0.f);
        return;
    }

    // shared: q [GMAX][dq] | scores [GMAX][CHUNK] | rows [CHUNK] | stats [2*GMAX] | acc [groups][GMAX][dv]
    // (dq: d rounded up to whole 16-byte pieces, the rest zeros)
    const int nvec = (d + VN - 1) / VN;
    const int dq = nvec * VN;
    float* sq = smem;
    float* ss = sq + GMAX * dq;
    long long* srow = reinterpret_cast<long long*>(ss + GMAX * ATT_CHUNK);      // a key's row of the tables: divided out once, not by every thread that reads it
    float* sstat = reinterpret_cast<float*>(srow + ATT_CHUNK);
    float* sacc = sstat + 2 * GMAX;

    const int entry = p.row_entry[r];
    const T* q = static_cast<const T*>(p.q) + ((size_t)r * p.hq + kvh * group + g0) * d;
    for (int i = tid; i < gn * dq; i += ATT_THREADS) {
        const int g = i / dq, c = i - g * dq;
        sq[i] = c < d ? Elem<T>::load(q + (size_t)g * d + c) : 0.f;
    }
    for (int j = tid; j < nkeys; j += ATT_THREADS) {
        const int pos = lo + j;
        const int lp = pos / p.page_size;
        const int page = lp < p.table_width ? p.block_table[(size_t)entry * p.table_width + lp] : -1;
        // A page outside the table would be a fault of the cache manager; such a key is skipped
        // by giving it row -1, and its score becomes -inf below.
        srow[j] = (page >= 0 && page < p.n_pages) ? ((long long)page * p.hkv + kvh) * p.page_size + pos % p.page_size : -1;
    }
    __syncthreads();

    // ---- scores
    const T* kt = static_cast<const T*>(p.k_table);
    constexpr int KPW = 32 / LPK;                          // keys a warp handles at a time
    const int sub = lane / LPK, li = lane % LPK;
    constexpr int AT_ONCE = VPL * VN <= 8 ? 8 : (VPL * VN <= 16 ? 4 : 2);      // keys of a warp asked for before the first is used
    for (int j0 = warp * KPW; j0 < nkeys; j0 += AT_ONCE * ATT_WARPS * KPW) {
        float kv[AT_ONCE][VPL][VN];
        bool has[AT_ONCE];
#pragma unroll
        for (int u = 0; u < AT_ONCE; ++u) {
            const int j = j0 + u * ATT_WARPS * KPW + sub;
            const long long at = j < nkeys ? srow[j] : -1;
            has[u] = at >= 0;
#pragma unroll
            for (int v = 0; v < VPL; ++v) {
                const int vi = li + v * LPK;
#pragma unroll
                for (int e = 0; e < VN; ++e) kv[u][v][e] = 0.f;
                if (has[u] && vi < nvec) {
                    const T* kp = kt + (size_t)at * d + vi * VN;
                    if (p.vec) {
                        Vec<T>::load(kp, kv[u][v]);
                    } else {
#pragma unroll
                        for (int e = 0; e < VN; ++e)
                            if (vi * VN + e < d) kv[u][v][e] = Elem<T>::load(kp + e);
                    }
                }
            }
        }
        for (int g = 0; g < gn; ++g) {
            float dot[AT_ONCE];
#pragma unroll
            for (int u = 0; u < AT_ONCE; ++u) dot[u] = 0.f;
#pragma unroll
            for (int v = 0; v < VPL; ++v) {
                const int vi = li + v * LPK;
                if (vi < nvec) {
#pragma unroll
                    for (int e = 0; e < VN; ++e) {
                        const float x = sq[g * dq + vi * VN + e];
#pragma unroll
                        for (int u = 0; u < AT_ONCE; ++u) dot[u] = fmaf(kv[u][v][e], x, dot[u]);
                    }
                }
            }
#pragma unroll
            for (int o = LPK / 2; o > 0; o >>= 1)           // the keys' sums of lanes side by side
#pragma unroll
                for (int u = 0; u < AT_ONCE; ++u) dot[u] += __shfl_xor_sync(0xffffffffu, dot[u], o);
#pragma unroll
            for (int u = 0; u < AT_ONCE; ++u) {
                const int j = j0 + u * ATT_WARPS * KPW + sub;
                if (j < nkeys && li == 0) ss[g * ATT_CHUNK + j] = has[u] ? dot[u] * p.scale : -INFINITY;
            }
        }
    }
    if (p.cap > 0.f) {                                      // a thread a key, not one of the lanes that share it
        __syncthreads();
        for (int i = tid; i < gn * nkeys; i += ATT_THREADS) {
            float& s = ss[i / nkeys * ATT_CHUNK + i % nkeys];
            if (srow[i % nkeys] >= 0) s = p.cap * tanhf(s / p.cap);
        }
    }
    __syncthreads();

    // ---- softmax within the chunk: one warp a head
    for (int g = warp; g < gn; g += ATT_WARPS) {
        float m = -INFINITY;
        for (int j = lane; j < nkeys; j += 32) m = fmaxf(m, ss[g * ATT_CHUNK + j]);
        m = warp_max(m);
        float l = 0.f;
        for (int j = lane; j < nkeys; j += 32) {
            const float s = ss[g * ATT_CHUNK + j];
            const float e = (m == -INFINITY) ? 0.f : soft_exp<T>(s - m);
            ss[g * ATT_CHUNK + j] = e;
            l += e;
        }
        l = warp_sum(l);
        if (lane == 0) { sstat[2 * g] = m; sstat[2 * g + 1] = l; }
    }
    __syncthreads();

    // ---- weighted sum of values: a thread owns two neighbouring components; thread groups of
    // d/2 share the keys when d/2 < ATT_THREADS, and add up in group order afterwards.
    const T* vt = static_cast<const T*>(p.v_table);
    const int pairs = (dv + 1) / 2;
    const int dvs = 2 * pairs;                              // a row of the groups' partial sums
    const int tgroups = pairs >= ATT_THREADS ? 1 : ATT_THREADS / pairs;
    const int tg = tid / pairs;                            // this thread's group (may be >= tgroups)
    float acc[GMAX][2];
    for (int pi = (tgroups == 1 ? tid : tid % pairs); pi < pairs; pi += ATT_THREADS) {
#pragma unroll
        for (int g = 0; g < GMAX; ++g) acc[g][0] = acc[g][1] = 0.f;
        if (tgroups == 1 || tg < tgroups) {
            const int jstart = tgroups == 1 ? 0 : tg;
            constexpr int AT_ONCE_V = 8;                    // likewise of the values; added up in the keys' order all the same
            for (int j0 = jstart; j0 < nkeys; j0 += AT_ONCE_V * tgroups) {
                float v0[AT_ONCE_V], v1[AT_ONCE_V];
                bool has[AT_ONCE_V];
#pragma unroll
                for (int u = 0; u < AT_ONCE_V; ++u) {
                    const int j = j0 + u * tgroups;
                    const long long at = j < nkeys ? srow[j] : -1;
                    has[u] = at >= 0;
                    v0[u] = v1[u] = 0.f;
                    if (has[u]) {
                        const T* vp = vt + (size_t)at * p.v_stride + 2 * pi;
                        v0[u] = Elem<T>::load(vp);
                        if (2 * pi + 1 < dv) v1[u] = Elem<T>::load(vp + 1);
                    }
                }
#pragma unroll
                for (int u = 0; u < AT_ONCE_V; ++u) {
                    if (!has[u]) continue;
#pragma unroll
                    for (int g = 0; g < GMAX; ++g) {
                        if (g < gn) {
                            const float w = ss[g * ATT_CHUNK + j0 + u * tgroups];
                            acc[g][0] = fmaf(w, v0[u], acc[g][0]);
                            acc[g][1] = fmaf(w, v1[u], acc[g][1]);
                        }
                    }
                }
            }
        }
        if (tgroups > 1) {
            if (tg < tgroups) {
#pragma unroll
                for (int g = 0; g < GMAX; ++g)
                    if (g < gn) {
                        sacc[((size_t)tg * GMAX + g) * dvs + 2 * pi] = acc[g][0];
                        sacc[((size_t)tg * GMAX + g) * dvs + 2 * pi + 1] = acc[g][1];
                    }
            }
            __syncthreads();
            if (tg == 0) {
#pragma unroll
                for (int g = 0; g < GMAX; ++g)
                    if (g < gn)
                        for (int x = 1; x < tgroups; ++x) {
                            acc[g][0] += sacc[((size_t)x * GMAX + g) * dvs + 2 * pi];
                            acc[g][1] += sacc[((size_t)x * GMAX + g) * dvs + 2 * pi + 1];
                        }
            }
        }
        if (tgroups == 1 || tg == 0) {
#pragma unroll
            for (int g = 0; g < GMAX; ++g) {
                if (g >= gn) continue;
                const int h = kvh * group + g0 + g;
                if (p.slots == 1) {
                    float l = sstat[2 * g + 1];
                    float inv = l > 0.f ? 1.f / l : 0.f;
                    if (p.sinks != nullptr) {                   // the weights were taken against the keys' maximum m
                        const float m = sstat[2 * g], sink = p.sinks[h];
                        const float top = fmaxf(m, sink);
                        const float wk = m == -INFINITY ? 0.f : soft_exp<T>(m - top);
                        l = l * wk + soft_exp<T>(sink - top);
                        inv = wk / l;
                    }
                    T* o = out + ((size_t)r * p.hq + h) * dv + 2 * pi;
                    Elem<T>::store(o, acc[g][0] * inv);
                    if (2 * pi + 1 < dv) Elem<T>::store(o + 1, acc[g][1] * inv);
                } else {
                    float* o = p.partial + (((size_t)r * p.hq + h) * p.slots + blockIdx.z) * (dv + 2);
                    o[2 * pi] = acc[g][0];
                    if (2 * pi + 1 < dv) o[2 * pi + 1] = acc[g][1];
                    if (pi == 0) { o[dv] = sstat[2 * g]; o[dv + 1] = sstat[2 * g + 1]; }
                }
            }
        }
    }
}

// out[r, h, :] = sum_z e^(m_z - M) acc_z / sum_z e^(m_z - M) l_z over the slots that held keys of the row.
// The slots' maxima and sums are read by the block's threads side by side (a slot a thread), the weights
// e^(m_z - M) left in shared memory; then a thread a component walks the slots with independent loads.
constexpr int COMBINE_SUMS = 128;      // threads that add up the slots' sums: a block has that many at least
constexpr int COMBINE_SLOTS = 1024;    // slots whose weights fit shared memory; beyond that they are computed again a component
template <typename T>
__global__ void combine_kernel(const AttParams p) {
    dependent_wait();                                       // returns at once after a plain launch
    dependent_trigger();
    __shared__ float scratch[32];
    __shared__ float weight[COMBINE_SLOTS];
    const int r = blockIdx.x, h = blockIdx.y;
    const int count = p.row_count[r];
    const int dv = p.dv;
    T* o = static_cast<T*>(p.out) + ((size_t)r * p.hq + h) * dv;
    if (count <= 0) return;                                // the rows kernel wrote zeros
    const float* base = p.partial + ((size_t)r * p.hq + h) * p.slots * (dv + 2);
    float mx = -INFINITY;
    for (int z = threadIdx.x; z < p.slots; z += blockDim.x) {
        int lo, hi;
        slot_range(p, count, z, lo, hi);
        if (hi > lo) mx = fmaxf(mx, base[(size_t)z * (dv + 2) + dv]);
    }
    mx = block_max(mx, scratch);
    if (p.sinks != nullptr) mx = fmaxf(mx, p.sinks[h]);
    float denom = 0.f;
    for (int z = threadIdx.x; z < p.slots && threadIdx.x < COMBINE_SUMS; z += COMBINE_SUMS) {      // the same sums whatever the block's size
        int lo, hi;
        slot_range(p, count, z, lo, hi);
        float w = 0.f;
        if (hi > lo) {
            const float m = base[(size_t)z * (dv + 2) + dv];
            w = m == -INFINITY ? 0.f : soft_exp<T>(m - mx);
            denom += w * base[(size_t)z * (dv + 2) + dv + 1];
        }
        if (z < COMBINE_SLOTS) weight[z] = w;
    }
    denom = block_sum(denom, scratch);                     // (its barriers also publish the weights)
    if (p.sinks != nullptr) denom += soft_exp<T>(p.sinks[h] - mx);
    const float inv = denom > 0.f ? 1.f / denom : 0.f;
    for (int i = threadIdx.x; i < dv; i += blockDim.x) {
        float acc = 0.f;
        const int known = min(p.slots, COMBINE_SLOTS);
        for (int z0 = 0; z0 < known; z0 += 8) {             // eight slots asked for before the first is added
            float v[8], w[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                w[u] = z0 + u < known ? weight[z0 + u] : 0.f;
                v[u] = w[u] != 0.f ? base[(size_t)(z0 + u) * (dv + 2) + i] : 0.f;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (w[u] != 0.f) acc = fmaf(w[u], v[u], acc);
        }
        for (int z = known; z < p.slots; ++z) {
            int lo, hi;
            slot_range(p, count, z, lo, hi);
            if (hi <= lo) continue;
            const float m = base[(size_t)z * (dv + 2) + dv];
            const float w = m == -INFINITY ? 0.f : soft_exp<T>(m - mx);
            acc = fmaf(w, base[(size_t)z * (dv + 2) + i], acc);
        }
        Elem<T>::store(o + i, acc * inv);
    }
}

// A thread a component, up to 512, where blocks are few (a decoding step): with 128 threads a component after the other waits for its slots' values (8 rows, 16 heads of
// 512, 24 slots: 13 us). Many blocks (300 rows of 16 heads: 16 us) lose more to the larger blocks' sums (53).
static int combine_threads(int dv, long long blocks) { return dv <= 128 || blocks > 4 * multiprocessors() ? 128 : dv <= 256 ? 256 : 512; }

static size_t rows_smem_bytes(int gmax, int d, int dv) {
    const int pairs = (dv + 1) / 2;
    const int tgroups = pairs >= ATT_THREADS ? 1 : ATT_THREADS / pairs;
    const int dq = (d + 7) / 8 * 8;                          // room for d rounded up to either element type's pieces
    size_t floats = (size_t)gmax * dq + (size_t)gmax * ATT_CHUNK + 2 * ATT_CHUNK + 2 * gmax;
    if (tgroups > 1) floats += (size_t)tgroups * gmax * (dv + 1);
    return floats * sizeof(float);
}

template <typename T, int GMAX, int LPK, int VPL>
static int launch_rows(const AttParams& p, cudaStream_t s) {
    const size_t smem = rows_smem_bytes(GMAX, p.d, p.dv);
    if (smem > 48 * 1024) {
        if (smem > 200 * 1024) return fail("paged_attention: head_dim %d needs %zu bytes of shared memory", p.d, smem);
        cudaFuncSetAttribute(rows_kernel<T, GMAX, LPK, VPL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    }
    const int group = p.hq / p.hkv;
    dim3 grid(p.rows, p.hkv * ((group + GMAX - 1) / GMAX), p.slots);
    rows_kernel<T, GMAX, LPK, VPL><<<grid, ATT_THREADS, smem, s>>>(p);
    return check_launch("paged_attention rows");
}

template <typename T, int GMAX>
static int dispatch_lanes(const AttParams& p, cudaStream_t s) {
    const int nvec = (p.d + Vec<T>::N - 1) / Vec<T>::N;   // 16-byte pieces of a key, the last maybe in part
    int lpk = 1;
    while (lpk * 2 <= nvec && lpk < 32) lpk *= 2;
    const int vpl = (nvec + lpk - 1) / lpk;
#define KB_ATT(L, V) return launch_rows<T, GMAX, L, V>(p, s)
    if (vpl == 1) {
        switch (lpk) {
            case 1: KB_ATT(1, 1);
            case 2: KB_ATT(2, 1);
            case 4: KB_ATT(4, 1);
            case 8: KB_ATT(8, 1);
            case 16: KB_ATT(16, 1);
            case 32: KB_ATT(32, 1);
        }
    } else if (vpl == 2) {
        switch (lpk) {
            case 2: KB_ATT(2, 2);
            case 4: KB_ATT(4, 2);
            case 8: KB_ATT(8, 2);
            case 16: KB_ATT(16, 2);
            case 32: KB_ATT(32, 2);
        }
    } else if (vpl <= 4 && lpk == 32) {
        KB_ATT(32, 4);
    } else if (vpl <= 8 && lpk == 32) {
        KB_ATT(32, 8);
    }
#undef KB_ATT
    return fail("paged_attention: head_dim %d is not handled (at most %d)", p.d, 32 * 8 * Vec<T>::N);
}

template <typename T>
static int dispatch_group(const AttParams& p, cudaStream_t s) {
    const int group = p.hq / p.hkv;
    if (group <= 1) return dispatch_lanes<T, 1>(p, s);
    if (group <= 2) return dispatch_lanes<T, 2>(p, s);
    if (group <= 4) return dispatch_lanes<T, 4>(p, s);
    return dispatch_lanes<T, 8>(p, s);                    // larger groups run as slices of 8 heads
}


template <typename T>
static int run_rows(const AttParams& p, cudaStream_t s, bool combine) {
    if (int e = dispatch_group<T>(p, s)) return e;
    if (combine) {
        combine_kernel<T><<<dim3(p.rows, p.hq), combine_threads(p.dv, (long long)p.rows * p.hq), 0, s>>>(p);
        return check_launch("paged_attention combine");
    }
    return 0;
}

int rows_f32(const AttParams& p, cudaStream_t s, bool combine);
int rows_bf16(const AttParams& p, cudaStream_t s, bool combine);

}  // namespace kb
