// A matrix memory with a fixed decay a head, by chunks of rows: the same steps as the decay scan's SCAN_FIXED
// (S <- w S + k v^T, o = S^T q) summed in another order, for the long portions of prompts.
//
// With the memory S_0 before a chunk of n <= 64 rows, its row t reads
//     o_t = w^t (w q_t)^T S_0 + sum_{s < t} w^(t-s-1) (w q_t . k_s) v_s + (q_t . k_t) v_t
// and the memory behind it is w^n S_0 + sum_s w^(n-1-s) k_s v_s^T. Three kernels: `retention_sums` makes every
// chunk's own sum (all chunks side by side), `retention_states` walks a request's chunks and puts in each sum's
// place the memory before that chunk (the one part that is a chain: one multiply-add a chunk), and
// `retention_rows` makes the rows' read-outs (all chunks side by side again). Chunks are counted from a
// request's first row of the step. Everything is 32-bit multiply-adds; powers of w come from powf (w = 0 is
// allowed: no division by w anywhere). Shared memory's 32 words a clock bound the sums and the rows (0.4 words a multiply-add), memory the
// states. Four requests of 340 rows, 16 heads of 128 x 128: sums 28 us, states 13, rows 51; with loads a word at a time, waited for before
// each multiplication, and the state read across its columns 46, 33 and 61.
#include "common.cuh"

namespace kb {

constexpr int RT_C = 64;               // rows a chunk
constexpr int RT_K = 32;               // inner steps staged at a time
constexpr int RT_THREADS = 256;

struct RetentionChunks {
    const float* vec;           // [rows, heads, 2, d]: w q, then k
    const float* val;           // [rows, heads, e]
    const float* scal;          // [rows, heads, 2]: the second is k.q
    const float* decay;         // [heads]
    float* sums;                // [chunks, heads, d, e]
    float* state;               // [slots, heads, e, d]
    const int* entry_start;
    const int* entry_end;
    const int* slots;
    int n_slots, heads, d, e;
    float* out;                 // [rows, heads, e]
};

// Where a request's first chunk lies: requests' rows follow one another, so ceil(n / 64) chunks fit between two of these.
__device__ __forceinline__ int first_chunk(int entry, int r0) { return r0 / RT_C + entry; }

__device__ __forceinline__ void rt_copy(float* to, const float* from, int words) {       // 16 bytes, or zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from), "r"(words * 4) : "memory");
}
// Columns x .. x + 3 of a row of `width` at `row` into shared memory, zeros where there are none. VEC: the rows are whole
// pieces of 16 bytes.
template <bool VEC>
__device__ __forceinline__ void rt_fetch(float* to, const float* row, bool there, int x, int width) {
    if (VEC) {
        const bool in = there && x < width;
        rt_copy(to, in ? row + x : row, in ? 4 : 0);
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) to[j] = there && x + j < width ? row[x + j] : 0.f;
    }
}
__device__ __forceinline__ void rt_fma(float (&acc)[4], float a, const float4& v) {
    acc[0] = fmaf(a, v.x, acc[0]);
    acc[1] = fmaf(a, v.y, acc[1]);
    acc[2] = fmaf(a, v.z, acc[2]);
    acc[3] = fmaf(a, v.w, acc[3]);
}
template <bool VEC>
__device__ __forceinline__ void rt_store(float* row, int x, int width, const float (&v)[4]) {
    if (VEC) {
        if (x < width) *reinterpret_cast<float4*>(row + x) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (x + j < width) row[x + j] = v[j];
    }
}

// sums[chunk, head, i, c] = sum_s w^(n-1-s) k_s[i] v_s[c]. One block = 64 key channels x 128 value components of a chunk; a
// thread 8 x 4 of them. The chunk's rows are asked for at once; the other blocks of the multiprocessor multiply meanwhile.
template <bool VEC>
__global__ void __launch_bounds__(RT_THREADS, 4)
retention_sums_kernel(const RetentionChunks p, int etiles) {
    extern __shared__ __align__(16) float rt_smem[];
    float* sk = rt_smem;                                        // [64][64]
    float* sv = rt_smem + RT_C * 64;                            // [64][128]
    __shared__ float pw[RT_C];
    const int entry = blockIdx.z, head = blockIdx.y;
    const int dtiles = (p.d + 63) / 64;
    const int chunk = blockIdx.x / (dtiles * etiles), tile = blockIdx.x % (dtiles * etiles);
    const int i0 = tile / etiles * 64, c0 = tile % etiles * 128;
    const int r0 = p.entry_start[entry], r1 = p.entry_end[entry];
    const int first = r0 + chunk * RT_C, n = min(RT_C, r1 - first);
    const int slot = p.slots[entry];
    if (n <= 0 || slot <= 0 || slot >= p.n_slots) return;
    const int tid = threadIdx.x, ti = tid / 32, tc = tid % 32;
    const float w = p.decay[head];
    for (int idx = tid; idx < n * 16; idx += RT_THREADS) {
        const int s = idx / 16, x = idx % 16 * 4;
        rt_fetch<VEC>(sk + s * 64 + x, p.vec + ((size_t)(first + s) * p.heads + head) * 2 * p.d + p.d, true, i0 + x, p.d);
    }
    for (int idx = tid; idx < n * 32; idx += RT_THREADS) {
        const int s = idx / 32, x = idx % 32 * 4;
        rt_fetch<VEC>(sv + s * 128 + x, p.val + ((size_t)(first + s) * p.heads + head) * p.e, true, c0 + x, p.e);
    }
    if (tid < RT_C) pw[tid] = powf(w, (float)tid);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    float acc[8][4] = {};
#pragma unroll 2
    for (int s = 0; s < n; ++s) {
        const float4 ka = *reinterpret_cast<const float4*>(sk + s * 64 + ti * 8), kb4 = *reinterpret_cast<const float4*>(sk + s * 64 + ti * 8 + 4);
        float4 v4 = *reinterpret_cast<const float4*>(sv + s * 128 + tc * 4);
        const float f = pw[n - 1 - s];
        v4.x *= f, v4.y *= f, v4.z *= f, v4.w *= f;
        const float k[8] = {ka.x, ka.y, ka.z, ka.w, kb4.x, kb4.y, kb4.z, kb4.w};
#pragma unroll
        for (int x = 0; x < 8; ++x) rt_fma(acc[x], k[x], v4);
    }
    float* dst = p.sums + ((size_t)(first_chunk(entry, r0) + chunk) * p.heads + head) * p.d * p.e;
#pragma unroll
    for (int x = 0; x < 8; ++x)
        if (i0 + ti * 8 + x < p.d) rt_store<VEC>(dst + (size_t)(i0 + ti * 8 + x) * p.e, c0 + tc * 4, p.e, acc[x]);
}

// Every chunk's sum becomes the memory before that chunk; the last one behind goes to the request's slot. A block 32 x 32 values of
// the memory, a thread four; the slot holds a column of the memory together where the sums hold a row, so the slot's values turn in
// shared memory. The sums of four chunks are asked for before the chain walks them.
__global__ void __launch_bounds__(RT_THREADS)
retention_states_kernel(const RetentionChunks p, int etiles) {
    __shared__ float turn[32][33];                              // [component][channel]
    const int entry = blockIdx.z, head = blockIdx.y;
    const int i0 = blockIdx.x / etiles * 32, c0 = blockIdx.x % etiles * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int r0 = p.entry_start[entry], r1 = p.entry_end[entry];
    const int slot = p.slots[entry];
    if (r1 <= r0 || slot <= 0 || slot >= p.n_slots) return;
    const size_t size = (size_t)p.d * p.e, stride = (size_t)p.heads * size;
    float* st = p.state + ((size_t)slot * p.heads + head) * size;
#pragma unroll
    for (int j = 0; j < 32; j += 8)
        if (c0 + ty + j < p.e && i0 + tx < p.d) turn[ty + j][tx] = st[(size_t)(c0 + ty + j) * p.d + i0 + tx];
    __syncthreads();
    const float w = p.decay[head], whole = powf(w, (float)RT_C);
    const int chunks = (r1 - r0 + RT_C - 1) / RT_C;
    const float tail = powf(w, (float)(r1 - r0 - (chunks - 1) * RT_C));
    float* at = p.sums + (size_t)first_chunk(entry, r0) * stride + (size_t)head * size + (size_t)(i0 + ty) * p.e + c0 + tx;
    float S[4];
    bool in[4];
#pragma unroll
    for (int y = 0; y < 4; ++y) {
        in[y] = i0 + ty + 8 * y < p.d && c0 + tx < p.e;
        S[y] = in[y] ? turn[tx][ty + 8 * y] : 0.f;
    }
    for (int ch = 0; ch < chunks; ch += 4) {
        float x[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int y = 0; y < 4; ++y) x[j][y] = ch + j < chunks && in[y] ? at[(size_t)(ch + j) * stride + (size_t)(8 * y) * p.e] : 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (ch + j < chunks) {
                const float f = ch + j < chunks - 1 ? whole : tail;
#pragma unroll
                for (int y = 0; y < 4; ++y) {
                    if (in[y]) at[(size_t)(ch + j) * stride + (size_t)(8 * y) * p.e] = S[y];
                    S[y] = fmaf(f, S[y], x[j][y]);
                }
            }
    }
    __syncthreads();
#pragma unroll
    for (int y = 0; y < 4; ++y)
        if (in[y]) turn[tx][ty + 8 * y] = S[y];
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 32; j += 8)
        if (c0 + ty + j < p.e && i0 + tx < p.d) st[(size_t)(c0 + ty + j) * p.d + i0 + tx] = turn[ty + j][tx];
}

// The read-outs of a chunk's rows for 128 value components: a thread 8 rows x 4 components, and 8 rows x 2 of the rows' scores
// against one another on the way. Queries, keys and the memory come 32 inner steps at a time by asynchronous copies, the next ones under
// this one's products; the chunk's values follow into the memory's places.
constexpr int RT_LD = RT_K + 4;
constexpr int RT_STAGE = 2 * RT_C * RT_LD + RT_K * 128;         // floats: queries [64][36], keys [64][36], memory (or values) [32][128]
template <bool VEC>
__global__ void __launch_bounds__(RT_THREADS, 3)
retention_rows_kernel(const RetentionChunks p) {
    extern __shared__ __align__(16) float rt_smem[];            // two stages
    static_assert(RT_C == 2 * RT_K && RT_C * (RT_C + 4) <= 2 * RT_C * RT_LD, "two pieces of values; the scores take the place of queries and keys");
    __shared__ float pw[RT_C + 1];
    const int entry = blockIdx.z, head = blockIdx.y;
    const int etiles = (p.e + 127) / 128;
    const int chunk = blockIdx.x / etiles, c0 = blockIdx.x % etiles * 128;
    const int r0 = p.entry_start[entry], r1 = p.entry_end[entry];
    const int first = r0 + chunk * RT_C, n = min(RT_C, r1 - first);
    if (n <= 0) return;
    const int tid = threadIdx.x, tr = tid / 32, tc = tid % 32;
    const int slot = p.slots[entry];
    const int d = p.d, e = p.e;
    if (slot <= 0 || slot >= p.n_slots) {                       // rows of no request: zeros
        for (int idx = tid; idx < n * 128; idx += RT_THREADS) {
            const int t = idx / 128, c = c0 + idx % 128;
            if (c < e) p.out[((size_t)(first + t) * p.heads + head) * e + c] = 0.f;
        }
        return;
    }
    const float w = p.decay[head];
    const float* before = p.sums + ((size_t)(first_chunk(entry, r0) + chunk) * p.heads + head) * d * e;
    auto queries = [&](int stage) { return rt_smem + stage * RT_STAGE; };
    auto keys = [&](int stage) { return rt_smem + stage * RT_STAGE + RT_C * RT_LD; };
    auto wide = [&](int stage) { return rt_smem + stage * RT_STAGE + 2 * RT_C * RT_LD; };
    const int steps = (d + RT_K - 1) / RT_K;
    // piece i: inner steps 32 i .., behind the last of them the values' rows 0 .. 31, then 32 .. 63
    auto fetch = [&](int i) {
        const int stage = i & 1;
        if (i < steps) {
            const int k0 = i * RT_K;
            for (int idx = tid; idx < RT_C * (RT_K / 4); idx += RT_THREADS) {
                const int t = idx / (RT_K / 4), x = idx % (RT_K / 4) * 4;
                const float* row = p.vec + ((size_t)(first + (t < n ? t : 0)) * p.heads + head) * 2 * d;
                rt_fetch<VEC>(queries(stage) + t * RT_LD + x, row, t < n, k0 + x, d);
                rt_fetch<VEC>(keys(stage) + t * RT_LD + x, row + d, t < n, k0 + x, d);
            }
            for (int idx = tid; idx < RT_K * 32; idx += RT_THREADS) {
                const int k = idx / 32, x = idx % 32 * 4;
                rt_fetch<VEC>(wide(stage) + k * 128 + x, before + (size_t)(k0 + k < d ? k0 + k : 0) * e, k0 + k < d, c0 + x, e);
            }
        } else {
            const int s0 = (i - steps) * RT_K;
            for (int idx = tid; idx < RT_K * 32; idx += RT_THREADS) {
                const int s = s0 + idx / 32, x = idx % 32 * 4;
                rt_fetch<VEC>(wide(stage) + idx / 32 * 128 + x, p.val + ((size_t)(first + (s < n ? s : 0)) * p.heads + head) * e, s < n, c0 + x, e);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0);
    if (tid <= RT_C) pw[tid] = powf(w, (float)tid);
    float o[8][4] = {}, sc[8][2] = {};
    for (int i = 0; i < steps; ++i) {
        fetch(i + 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const float *q = queries(i & 1) + tr * 8 * RT_LD, *k = keys(i & 1) + tc * RT_LD, *b = wide(i & 1) + tc * 4;
#pragma unroll 1
        for (int x4 = 0; x4 < RT_K; x4 += 4) {
            const float4 ka = *reinterpret_cast<const float4*>(k + x4), kb4 = *reinterpret_cast<const float4*>(k + 32 * RT_LD + x4);
            float4 m4[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) m4[j] = *reinterpret_cast<const float4*>(b + (x4 + j) * 128);
#pragma unroll
            for (int x = 0; x < 8; ++x) {
                const float4 a = *reinterpret_cast<const float4*>(q + x * RT_LD + x4);
                rt_fma(o[x], a.x, m4[0]);
                rt_fma(o[x], a.y, m4[1]);
                rt_fma(o[x], a.z, m4[2]);
                rt_fma(o[x], a.w, m4[3]);
                sc[x][0] = fmaf(a.w, ka.w, fmaf(a.z, ka.z, fmaf(a.y, ka.y, fmaf(a.x, ka.x, sc[x][0]))));
                sc[x][1] = fmaf(a.w, kb4.w, fmaf(a.z, kb4.z, fmaf(a.y, kb4.y, fmaf(a.x, kb4.x, sc[x][1]))));
            }
        }
        __syncthreads();
    }
    fetch(steps + 1);                                           // the values' second half, where the memory's last piece was
    float* ss = queries(0);                                     // [s][t], rows of 68: what row s gives to row t
#pragma unroll
    for (int y = 0; y < 2; ++y) {
        const int s = tc + 32 * y;
        float g[8];
#pragma unroll
        for (int x = 0; x < 8; ++x) {
            const int t = tr * 8 + x;
            g[x] = 0.f;
            if (s < t && t < n) g[x] = pw[t - s - 1] * sc[x][y];
            else if (s == t && t < n) g[x] = p.scal[((size_t)(first + t) * p.heads + head) * 2 + 1];
        }
        *reinterpret_cast<float4*>(ss + s * (RT_C + 4) + tr * 8) = make_float4(g[0], g[1], g[2], g[3]);
        *reinterpret_cast<float4*>(ss + s * (RT_C + 4) + tr * 8 + 4) = make_float4(g[4], g[5], g[6], g[7]);
    }
#pragma unroll
    for (int x = 0; x < 8; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) o[x][y] *= pw[tr * 8 + x];
    for (int half = 0; half < 2; ++half) {
        const int s0 = half * RT_K;
        if (s0 >= n) break;                                     // the same for the whole block
        if (half == 0) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (tr * 8 + 7 < s0) continue;                          // rows before these sources take nothing from them
        const float* b = wide((steps + half) & 1) + tc * 4;
#pragma unroll 2
        for (int s = 0; s < RT_K; ++s) {
            const float4 ga = *reinterpret_cast<const float4*>(ss + (s0 + s) * (RT_C + 4) + tr * 8), gb = *reinterpret_cast<const float4*>(ss + (s0 + s) * (RT_C + 4) + tr * 8 + 4);
            const float4 v4 = *reinterpret_cast<const float4*>(b + s * 128);
            const float g[8] = {ga.x, ga.y, ga.z, ga.w, gb.x, gb.y, gb.z, gb.w};
#pragma unroll
            for (int x = 0; x < 8; ++x) rt_fma(o[x], g[x], v4);
        }
    }
#pragma unroll
    for (int x = 0; x < 8; ++x)
        if (tr * 8 + x < n) rt_store<VEC>(p.out + ((size_t)(first + tr * 8 + x) * p.heads + head) * e, c0 + tc * 4, e, o[x]);
    asm volatile("cp.async.wait_all;" ::: "memory");
}

long long retention_chunk_floats(int rows, int entries, int heads, int d, int e) {
    return ((long long)rows / RT_C + entries) * heads * d * e;
}

// vec, val, scal: the decay scan's inputs in its SCAN_FIXED order. `longest`: the most rows a request brings.
int run_retention_chunks(float* out, const float* vec, const float* val, const float* scal, const float* decay, float* sums, float* state,
                         int n_slots, const int* entry_start, const int* entry_end, const int* slots, int entries, int longest, int heads,
                         int d, int e, cudaStream_t s) {
    RetentionChunks p;
    p.vec = vec; p.val = val; p.scal = scal; p.decay = decay; p.sums = sums; p.state = state; p.entry_start = entry_start;
    p.entry_end = entry_end; p.slots = slots; p.n_slots = n_slots; p.heads = heads; p.d = d; p.e = e; p.out = out;
    const long long chunks = (longest + RT_C - 1) / RT_C;
    const int dtiles = (d + 63) / 64, etiles = (e + 127) / 128;
    KB_REQUIRE(heads <= 65535 && entries <= 65535 && chunks * dtiles * etiles <= 0x7fffffffll, "retention: too many heads, requests or rows for one launch");
    const bool vec4 = d % 4 == 0 && e % 4 == 0 && (((uintptr_t)vec | (uintptr_t)val | (uintptr_t)sums | (uintptr_t)out) & 15) == 0;
    constexpr int sums_smem = RT_C * (64 + 128) * 4, rows_smem = 2 * RT_STAGE * 4;
    static bool attr_set = false;
    if (!attr_set) {
        if (cudaFuncSetAttribute(retention_sums_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, sums_smem) != cudaSuccess ||
            cudaFuncSetAttribute(retention_sums_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, sums_smem) != cudaSuccess ||
            cudaFuncSetAttribute(retention_rows_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, rows_smem) != cudaSuccess ||
            cudaFuncSetAttribute(retention_rows_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, rows_smem) != cudaSuccess)
            return fail("retention: cannot have %d bytes of shared memory", rows_smem);
        attr_set = true;
    }
    const dim3 sums_grid((unsigned)(chunks * dtiles * etiles), heads, entries), rows_grid((unsigned)(chunks * etiles), heads, entries);
    if (vec4) retention_sums_kernel<true><<<sums_grid, RT_THREADS, sums_smem, s>>>(p, etiles);
    else retention_sums_kernel<false><<<sums_grid, RT_THREADS, sums_smem, s>>>(p, etiles);
    if (int err = check_launch("retention sums")) return err;
    retention_states_kernel<<<dim3((unsigned)(((d + 31) / 32) * ((e + 31) / 32)), heads, entries), RT_THREADS, 0, s>>>(p, (e + 31) / 32);
    if (int err = check_launch("retention states")) return err;
    if (vec4) retention_rows_kernel<true><<<rows_grid, RT_THREADS, rows_smem, s>>>(p);
    else retention_rows_kernel<false><<<rows_grid, RT_THREADS, rows_smem, s>>>(p);
    return check_launch("retention rows");
}

}  // namespace kb
