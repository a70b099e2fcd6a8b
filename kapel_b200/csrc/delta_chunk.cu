// The gated delta rule over long portions of prompts, by chunks of 32 rows: the steps of the scan
//     S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q
// summed in another order. With the memory S_0 before a chunk, G_t the decay from the chunk's start up to and with row t and D_ts the
// decay of the rows s + 1 .. t (products of the rows' decays, never quotients: a decay of 0 is a decay like any other),
//     u_t = beta_t (v_t - G_t S_0^T k_t - sum_{s < t} D_ts (k_s . k_t) u_s)
// so U = U0 - W S_0, where (I + A) [W | U0] = [beta G K | beta V], A_ts = beta_t D_ts (k_t . k_s) below the diagonal: a forward substitution
// that needs no memory, chunk by chunk side by side. Then
//     o_t = G_t S_0^T q_t + sum_{s <= t} D_ts (q_t . k_s) u_s,     S = G_C S_0 + sum_s D_Cs k_s u_s^T.
// `delta_chunk_kernel`, a block a chunk and head: the keys against the keys and the queries, W, U0, the weights within the chunk and the
// decays, by 32-bit multiply-adds. `delta_chain_kernel`, a block a head and 16 of its value components of one request: the chain over the chunks, whose three
// products go by mma.sync over bfloat16 pieces that hold the 32-bit values exactly (pieces.cuh; the first kernel leaves W, queries and keys cut, the memory
// and the writes are cut as they arise), each of 16 or 32 terms at most in the tensor cores, the sums of more in 32-bit registers, and so is the memory.
// What bounds the chain: 144 products of 16 x 8 x 16 a chunk on each quarter of a multiprocessor (1,250 clocks), some 1,900 clocks of shared memory and the
// hand-overs between its warps: 1.65 us a chunk (3.9 by multiply-adds from shared memory; the scan's 32 steps take 9.7). 2,048 rows, 16 heads of 128 over 4
// key heads: 49 us for the chunks and 106 us for the chain (54 and 249; the scan: 619 us); 500 rows 18 and 29, 64 rows 14 and 7 (the scan 24).
// Sums go by short chains, so that the error against 64 bits stays at the scan's: 1.01 of it where memories fade within a row, 1.08 within some twenty
// rows, 0.93 to 0.98 where they hardly do (by multiply-adds 0.99, 1.08 and 1.00). (A block a chunk and key head, four heads one after the other, took 61 us.)
#include <initializer_list>
#include "delta_chunk.cuh"
#include "pieces.cuh"

namespace kb {

constexpr int DCH_THREADS = 128, DCH_E = 16, DCH_MAX_D = 128, DCH_LD = DCH_MAX_D + 4;

// Requests by chunks whose rows lie ahead of row r0; all lanes of a warp call (at the kernels' beginning: the loads go beside their first ones).
__device__ __forceinline__ int delta_chunks_before(const DeltaChunks& p, int r0) {
    if (p.entries == 1) return 0;
    int before = 0;
    for (int i = threadIdx.x & 31; i < p.entries; i += 32) {
        const int start = p.entry_start[i];
        before += start < r0 && p.entry_end[i] - start >= p.from_rows;
    }
    return __reduce_add_sync(0xffffffffu, before);
}

__global__ void __launch_bounds__(DCH_THREADS, 4)
delta_chunk_kernel(const DeltaChunks p) {
    __shared__ __align__(16) float sk[DCH_C][DCH_LD], sq[DCH_C][DCH_LD];
    __shared__ __align__(16) float kk[DCH_C][DCH_C + 4], qk[DCH_C][DCH_C + 4], decay[DCH_C][DCH_C + 4];      // [t][s]
    __shared__ float sg[DCH_C], sbeta[DCH_C];
    const int entry = blockIdx.z, h = blockIdx.y, per = p.heads / p.kv_heads, kvh = h / per;
    const int r0 = p.entry_start[entry], r1 = p.entry_end[entry], before = delta_chunks_before(p, r0);
    const int first = r0 + blockIdx.x * DCH_C, n = min(DCH_C, r1 - first);
    const int slot = p.slots[entry];
    if (r1 - r0 < p.from_rows || n <= 0 || slot <= 0 || slot >= p.n_slots) return;
    const int tid = threadIdx.x, d = p.d, e = p.e, d4 = d >> 2;
    for (int i = tid; i < DCH_C * d4; i += DCH_THREADS) {
        const int t = i / d4, x = (i - t * d4) * 4;
        const size_t from = ((size_t)(first + min(t, n - 1)) * p.kv_heads + kvh) * d + x;
        const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);                     // rows beyond the last: no key, no query
        *reinterpret_cast<float4*>(&sk[t][x]) = t < n ? *reinterpret_cast<const float4*>(p.kn + from) : none;
        *reinterpret_cast<float4*>(&sq[t][x]) = t < n ? *reinterpret_cast<const float4*>(p.qn + from) : none;
    }
    __syncthreads();
    const int place = delta_chunk_place(first, before), ld = delta_piece_row(d);
    for (int i = h == kvh * per ? tid : DCH_C * d; i < DCH_C * (d >> 1); i += DCH_THREADS) {                  // their pieces, by the kv head's first head
        const int t = i / (d >> 1), x = (i - t * (d >> 1)) * 2;
        uint32_t* q = reinterpret_cast<uint32_t*>(p.qk + (((size_t)place * p.kv_heads + kvh) * 2 * DCH_C + t) * ld + x);
        uint32_t* k = q + DCH_C * ld / 2;
        float a = sq[t][x], b = sq[t][x + 1];
        cut_pair(a, b, q[0], q[d / 2], q[d]);
        a = sk[t][x], b = sk[t][x + 1];
        cut_pair(a, b, k[0], k[d / 2], k[d]);
    }
    {   // a thread: row t against rows s0, s0 + 4, .. of the chunk (neighbouring rows begin in different banks)
        const int t = tid >> 2, s0 = tid & 3;
        float a[8] = {}, b[8] = {};
        for (int x0 = 0; x0 < d; x0 += 32) {                    // 32 components in four chains of eight: the rounding of a warp's sum of lanes
            float4 ka[8] = {}, qa[8] = {};
#pragma unroll 1
            for (int x = x0; x < x0 + 32; x += 4) {
                const float4 k = *reinterpret_cast<const float4*>(&sk[t][x]), q = *reinterpret_cast<const float4*>(&sq[t][x]);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float4 o = *reinterpret_cast<const float4*>(&sk[s0 + 4 * j][x]);
                    ka[j].x = fmaf(k.x, o.x, ka[j].x), ka[j].y = fmaf(k.y, o.y, ka[j].y), ka[j].z = fmaf(k.z, o.z, ka[j].z), ka[j].w = fmaf(k.w, o.w, ka[j].w);
                    qa[j].x = fmaf(q.x, o.x, qa[j].x), qa[j].y = fmaf(q.y, o.y, qa[j].y), qa[j].z = fmaf(q.z, o.z, qa[j].z), qa[j].w = fmaf(q.w, o.w, qa[j].w);
                }
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                a[j] += (ka[j].x + ka[j].y) + (ka[j].z + ka[j].w);
                b[j] += (qa[j].x + qa[j].y) + (qa[j].z + qa[j].w);
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)                             // a row against itself: as the scan has it, from before the vectors were rounded
            kk[t][s0 + 4 * j] = a[j], qk[t][s0 + 4 * j] = s0 + 4 * j == t && t < n ? p.kq[(size_t)(first + t) * p.kv_heads + kvh] : b[j];
    }
    auto am = sq;                                               // [t][s] the substitution's matrix, once the queries are done with
    if (tid < DCH_C) {
        const float2 gb = tid < n ? *reinterpret_cast<const float2*>(p.scal + ((size_t)(first + tid) * p.heads + h) * 2) : make_float2(1.f, 0.f);
        sg[tid] = gb.x, sbeta[tid] = gb.y;
        __syncwarp();
        float D = 0.f, G = 1.f;
#pragma unroll 8
        for (int t = 0; t < DCH_C; ++t) {                       // column s = tid of the decays: zero above the diagonal, 1 on it
            D = t == tid ? 1.f : D * sg[t];
            decay[t][tid] = D;
            G = t <= tid ? G * sg[t] : G;
        }
        const float whole = __shfl_sync(0xffffffffu, G, n - 1);
        float* to = p.within + ((size_t)place * p.heads + h) * DCH_WITHIN;
        to[DCH_G + tid] = tid < n ? G : 0.f;
        to[DCH_F + tid] = tid < n ? decay[n - 1][tid] : 0.f;
        if (tid < 4) to[DCH_ALL + tid] = whole;
    }
    __syncthreads();
    for (int i = tid; i < DCH_C * DCH_C; i += DCH_THREADS) {
        const int t = i / DCH_C, s = i % DCH_C;
        p.within[((size_t)place * p.heads + h) * DCH_WITHIN + t * DCH_LD_W + s] = t < n && s <= t ? decay[t][s] * qk[t][s] : 0.f;
        am[t][s] = s < t ? sbeta[t] * decay[t][s] * kk[t][s] : 0.f;
    }
    __syncthreads();
    // the substitution, two neighbouring columns of [beta G K | beta V] a thread: their 64 values are asked for before the first is needed
    for (int c = tid * 2; c < d + e; c += DCH_THREADS * 2) {
        float x[DCH_C], y[DCH_C];
        float G = 1.f;
#pragma unroll
        for (int t = 0; t < DCH_C; ++t) {
            G *= sg[t];
            const float2 v = c < d ? make_float2(G * sk[t][c], G * sk[t][c + 1])
                                   : *reinterpret_cast<const float2*>(p.vn + ((size_t)(first + min(t, n - 1)) * p.heads + h) * e + (c - d));
            x[t] = sbeta[t] * v.x, y[t] = sbeta[t] * v.y;       // beta is 0 beyond the last row
        }
#pragma unroll
        for (int t = 1; t < DCH_C; ++t) {
            float2 sum[2] = {};
#pragma unroll
            for (int s = 0; s < t; s += 4) {                    // zeros on and above the diagonal
                const float4 a = *reinterpret_cast<const float4*>(&am[t][s]);
                sum[0].x = fmaf(a.x, x[s], sum[0].x), sum[0].y = fmaf(a.x, y[s], sum[0].y);
                if (s + 1 < t) sum[1].x = fmaf(a.y, x[s + 1], sum[1].x), sum[1].y = fmaf(a.y, y[s + 1], sum[1].y);
                if (s + 2 < t) sum[0].x = fmaf(a.z, x[s + 2], sum[0].x), sum[0].y = fmaf(a.z, y[s + 2], sum[0].y);
                if (s + 3 < t) sum[1].x = fmaf(a.w, x[s + 3], sum[1].x), sum[1].y = fmaf(a.w, y[s + 3], sum[1].y);
            }
            x[t] -= sum[0].x + sum[1].x, y[t] -= sum[0].y + sum[1].y;
        }
#pragma unroll
        for (int t = 0; t < DCH_C; ++t)
            if (t >= n) x[t] = y[t] = 0.f;
        if (c < d) {
            uint32_t* to = reinterpret_cast<uint32_t*>(p.w + ((size_t)place * p.heads + h) * DCH_C * ld + c);
#pragma unroll
            for (int t = 0; t < DCH_C; ++t, to += ld / 2) cut_pair(x[t], y[t], to[0], to[d / 2], to[d]);
        } else {
            float* to = p.u0 + (((size_t)place * p.heads + h) * e + (c - d)) * DCH_LD_W;
#pragma unroll
            for (int t = 0; t < DCH_C; t += 4) {
                *reinterpret_cast<float4*>(to + t) = make_float4(x[t], x[t + 1], x[t + 2], x[t + 3]);
                *reinterpret_cast<float4*>(to + DCH_LD_W + t) = make_float4(y[t], y[t + 1], y[t + 2], y[t + 3]);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------- the chain
// Sixteen warps. Eight hold the memory, transposed, 16 of the key's components each in registers: S^T is an MMA's result, and as it lies the next
// one's A operand. Four add up the eight shares of (W S)^T and make the chunk's writes, while the eight multiply the queries; four more make
// the read-outs, a chunk behind, and one lane of them asks for the chunks' inputs, bulk copies of what `delta_chunk_kernel` laid out. Barrier 1:
// the shares of W S are there; 2: the chunk's writes, and the shares of Q S; 3: those of the chunk before have been read.
constexpr int DCH_WARPS = 8, DCH_WRITERS = 4, DCH_READERS = 4, DCH_CHAIN = (DCH_WARPS + DCH_WRITERS + DCH_READERS) * 32;
constexpr int DCH_LD_P = DCH_C + 8, DCH_LD_D = DCH_C + 8;
// Shared memory: two sets of the weights within the chunk, the warps' shares of (W S)^T and of (Q S)^T, two of U^T, the pieces of U^T faded to the
// chunk's end, the barriers; then two sets of W and queries, two of keys (pieces, as they lie in memory).
struct DchSmem {
    float within[2][DCH_WITHIN];
    float part[2][DCH_WARPS][DCH_E][DCH_LD_P];
    float u[2][DCH_E][DCH_LD_W];
    __nv_bfloat16 ud[3][DCH_E][DCH_LD_D];
    uint64_t wq_full[2], k_full[2];
};
static_assert(sizeof(DchSmem) % 16 == 0, "the pieces behind it begin at a multiple of 16 bytes");
static int dch_smem(int d) { return (int)sizeof(DchSmem) + 6 * DCH_C * delta_piece_row(d) * 2; }

__device__ int g_delta_chain_error = 0;

__device__ __forceinline__ uint32_t dch_saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool dch_wait(uint64_t* bar, uint32_t parity) {          // false if it did not come within about a second
    const long long start = clock64();
    for (;;) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(dch_saddr(bar)), "r"(parity) : "memory");
        if (ok) return true;
        if (clock64() - start > 2000000000ll) return false;
    }
}
__device__ __forceinline__ void dch_expect(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(dch_saddr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void dch_bulk(void* to, const void* from, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dch_saddr(to)), "l"(from), "r"(bytes), "r"(dch_saddr(bar)) : "memory");
}
__device__ __forceinline__ void dch_ldmatrix(uint32_t (&r)[4], uint32_t at) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void dch_ldmatrix_turned(uint32_t (&r)[4], uint32_t at) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void dch_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__global__ void __launch_bounds__(DCH_CHAIN, 1)
delta_chain_kernel(const DeltaChunks p) {
    extern __shared__ __align__(128) unsigned char dch_raw[];
    DchSmem& m = *reinterpret_cast<DchSmem*>(dch_raw);
    const int entry = blockIdx.z, head = blockIdx.y, c0 = blockIdx.x * DCH_E;
    const int r0 = p.entry_start[entry], r1 = p.entry_end[entry], before = delta_chunks_before(p, r0);
    const int slot = p.slots[entry];
    if (r1 - r0 < p.from_rows) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, d = p.d, e = p.e;
    if (slot <= 0 || slot >= p.n_slots) {                       // rows of no request: zeros, no state
        for (int i = tid; i < (r1 - r0) * DCH_E; i += DCH_CHAIN) p.out[((size_t)(r0 + i / DCH_E) * p.heads + head) * e + c0 + i % DCH_E] = 0.f;
        return;
    }
    const int kvh = head / (p.heads / p.kv_heads);
    float* st = p.state + (size_t)slot * p.state_floats + p.state_off + ((size_t)head * e + c0) * d;      // [16][d]: a column of the memory lies together
    const int chunks = (r1 - r0 + DCH_C - 1) / DCH_C, ld = delta_piece_row(d), image = DCH_C * ld;        // an operand's pieces of a chunk
    __nv_bfloat16* wq = reinterpret_cast<__nv_bfloat16*>(dch_raw + sizeof(DchSmem));                      // [2][W, queries]
    __nv_bfloat16* keys = wq + 4 * image;                                                                 // [2]
    if (tid == 0) {
        for (int b = 0; b < 2; ++b)
            for (uint64_t* bar : {&m.wq_full[b], &m.k_full[b]}) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(dch_saddr(bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    bool failed = false;                                        // a wait that ran out is not repeated, but the walk goes on: the warps meet in every chunk
    auto weights = [&](int ch) { return p.within + ((size_t)delta_chunk_place(r0 + ch * DCH_C, before) * p.heads + head) * DCH_WITHIN; };

    if (warp >= DCH_WARPS + DCH_WRITERS) {
        // ---------------------------------------------------------------- read-outs: a component of four rows a thread; the copies
        const bool copies = tid == (DCH_WARPS + DCH_WRITERS) * 32;
        auto fetch_wq = [&](int ch) {
            if (ch >= chunks || !copies) return;
            const size_t place = delta_chunk_place(r0 + ch * DCH_C, before);
            __nv_bfloat16* to = wq + (ch & 1) * 2 * image;
            dch_expect(&m.wq_full[ch & 1], (uint32_t)image * 4);
            dch_bulk(to, p.w + (place * p.heads + head) * image, (uint32_t)image * 2, &m.wq_full[ch & 1]);
            dch_bulk(to + image, p.qk + (place * p.kv_heads + kvh) * 2 * image, (uint32_t)image * 2, &m.wq_full[ch & 1]);
        };
        auto fetch_k = [&](int ch) {
            if (ch >= chunks || !copies) return;
            const size_t place = delta_chunk_place(r0 + ch * DCH_C, before);
            const int b = ch & 1;
            dch_expect(&m.k_full[b], (uint32_t)image * 2 + sizeof(m.within[0]));
            dch_bulk(keys + b * image, p.qk + ((place * p.kv_heads + kvh) * 2 + 1) * image, (uint32_t)image * 2, &m.k_full[b]);
            dch_bulk(m.within[b], weights(ch), sizeof(m.within[0]), &m.k_full[b]);
        };
        fetch_wq(0);
        fetch_k(0);
        fetch_wq(1);
        __syncwarp();
        asm volatile("bar.arrive 3, %0;" ::"n"((DCH_WARPS + DCH_READERS) * 32) : "memory");
        const int x = lane & 15, t0 = ((tid - (DCH_WARPS + DCH_WRITERS) * 32) >> 4) * 4;
        for (int ch = 0; ch < chunks; ++ch) {
            const int b = ch & 1, first = r0 + ch * DCH_C, n = min(DCH_C, r1 - first);
            asm volatile("bar.sync 2, %0;" ::"n"(DCH_CHAIN) : "memory");        // the next chunk's W and queries have been read, and all of the chunk before
            if (ch == 0) fetch_wq(2);
            fetch_wq(ch + 3);
            fetch_k(ch + 1);
            __syncwarp();
            if (!failed && !dch_wait(&m.k_full[b], (uint32_t)(ch >> 1) & 1u)) failed = true;
            float o[4] = {};
            for (int w2 = 0; w2 < d >> 4; w2 += 2) {
                const float4 v = *reinterpret_cast<const float4*>(&m.part[1][w2][x][t0]), w = *reinterpret_cast<const float4*>(&m.part[1][w2 + 1][x][t0]);
                o[0] += v.x + w.x, o[1] += v.y + w.y, o[2] += v.z + w.z, o[3] += v.w + w.w;
            }
            __syncwarp();
            if (ch + 1 < chunks) asm volatile("bar.arrive 3, %0;" ::"n"((DCH_WARPS + DCH_READERS) * 32) : "memory");
            const float* within = m.within[b];
            const float4 G = *reinterpret_cast<const float4*>(within + DCH_G + t0);
            o[0] *= G.x, o[1] *= G.y, o[2] *= G.z, o[3] *= G.w;
            // Up to the row itself: a later row's write may be no finite number, and then a weight of zero does not keep it out.
            float below[4] = {};
            for (int s = 0; s < t0; s += 4) {
                const float4 u = *reinterpret_cast<const float4*>(&m.u[b][x][s]);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float4 a = *reinterpret_cast<const float4*>(within + (t0 + j) * DCH_LD_W + s);
                    below[j] = fmaf(a.x, u.x, below[j]), below[j] = fmaf(a.y, u.y, below[j]), below[j] = fmaf(a.z, u.z, below[j]), below[j] = fmaf(a.w, u.w, below[j]);
                }
            }
            const float4 u4 = *reinterpret_cast<const float4*>(&m.u[b][x][t0]);
            const float u[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                o[j] += below[j];
#pragma unroll
                for (int i = 0; i <= j; ++i) o[j] = fmaf(within[(t0 + j) * DCH_LD_W + t0 + i], u[i], o[j]);
                if (t0 + j < n) p.out[((size_t)(first + t0 + j) * p.heads + head) * e + c0 + x] = o[j];
            }
        }
        if (copies)                                             // nothing is in flight when the block ends
            for (int ch = max(0, chunks - 2); ch < chunks; ++ch)
                if (!dch_wait(&m.wq_full[ch & 1], (uint32_t)(ch >> 1) & 1u) || !dch_wait(&m.k_full[ch & 1], (uint32_t)(ch >> 1) & 1u)) failed = true;
    } else if (warp >= DCH_WARPS) {
        // ---------------------------------------------------------------- U = U0 - W S: a component of four rows a thread
        const int x = (tid - DCH_WARPS * 32) >> 3, t0 = (tid & 7) * 4;
        auto first_writes = [&](int ch) {
            return *reinterpret_cast<const float4*>(p.u0 + (((size_t)delta_chunk_place(r0 + ch * DCH_C, before) * p.heads + head) * e + c0 + x) * DCH_LD_W + t0);
        };
        auto fade = [&](int ch) { return *reinterpret_cast<const float4*>(weights(ch) + DCH_F + t0); };
        float4 u = first_writes(0), f = fade(0);
        for (int ch = 0; ch < chunks; ++ch) {
            asm volatile("bar.sync 1, %0;" ::"n"((DCH_WARPS + DCH_WRITERS) * 32) : "memory");
            float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int w2 = 0; w2 < d >> 4; w2 += 2) {
                const float4 v = *reinterpret_cast<const float4*>(&m.part[0][w2][x][t0]), w = *reinterpret_cast<const float4*>(&m.part[0][w2 + 1][x][t0]);
                sum.x += v.x + w.x, sum.y += v.y + w.y, sum.z += v.z + w.z, sum.w += v.w + w.w;
            }
            u.x -= sum.x, u.y -= sum.y, u.z -= sum.z, u.w -= sum.w;
            *reinterpret_cast<float4*>(&m.u[ch & 1][x][t0]) = u;
            uint2 one, two, three;
            f.x *= u.x, f.y *= u.y, f.z *= u.z, f.w *= u.w;
            cut_pair(f.x, f.y, one.x, two.x, three.x);
            cut_pair(f.z, f.w, one.y, two.y, three.y);
            *reinterpret_cast<uint2*>(&m.ud[0][x][t0]) = one;
            *reinterpret_cast<uint2*>(&m.ud[1][x][t0]) = two;
            *reinterpret_cast<uint2*>(&m.ud[2][x][t0]) = three;
            __syncwarp();
            asm volatile("bar.arrive 2, %0;" ::"n"(DCH_CHAIN) : "memory");
            if (ch + 1 < chunks) u = first_writes(ch + 1), f = fade(ch + 1);
        }
    } else {
        // ---------------------------------------------------------------- the memory: S^T [16][16 of the key's components] a warp, as an MMA's result lies
        const bool owns = warp * 16 < d;                        // fewer components than 128: the last warps only keep step
        const int d0 = owns ? warp * 16 : 0;
        const int row = lane >> 2, col = (lane & 3) * 2;
        float S[2][4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float* from = st + row * d + d0 + 8 * h + col;
            S[h][0] = from[0], S[h][1] = from[1], S[h][2] = from[8 * d], S[h][3] = from[8 * d + 1];
        }
        // W and queries of a chunk as B operands: rows 16 i .. of either, this warp's 16 components
        uint32_t x[2][3][2][4];
        auto read_rows = [&](int ch, int half) {
            const uint32_t at = dch_saddr(wq + ((ch & 1) * 2 + half) * image + ((lane & 7) + (lane >> 4) * 8) * ld + d0 + ((lane >> 3) & 1) * 8);
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int q = 0; q < 3; ++q) dch_ldmatrix(x[half][q][i], at + (uint32_t)(i * 16 * ld + q * d) * 2u);
        };
        if (!dch_wait(&m.wq_full[0], 0u)) failed = true;
        __syncwarp();
        read_rows(0, 0);
        read_rows(0, 1);
        for (int ch = 0; ch < chunks; ++ch) {
            const int b = ch & 1;
            uint32_t s[3][4];
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    float v = S[h][2 * i], w = S[h][2 * i + 1];
                    cut_pair(v, w, s[0][2 * h + i], s[1][2 * h + i], s[2][2 * h + i]);
                }
            // this warp's share of the inner dimension: (W S)^T, then (Q S)^T while the chunk's writes are made
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                float acc[4][4] = {};
                if (owns) {
#pragma unroll
                    for (int q = 0; q < PIECE_PRODUCTS; ++q)
#pragma unroll
                        for (int i = 0; i < 4; ++i) dch_mma(acc[i], s[piece_a(q)], x[half][piece_b(q)][i >> 1][2 * (i & 1)], x[half][piece_b(q)][i >> 1][2 * (i & 1) + 1]);
                }
                if (half == 1) asm volatile("bar.sync 3, %0;" ::"n"((DCH_WARPS + DCH_READERS) * 32) : "memory");
                if (owns) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        *reinterpret_cast<float2*>(&m.part[half][warp][row][8 * i + col]) = make_float2(acc[i][0], acc[i][1]);
                        *reinterpret_cast<float2*>(&m.part[half][warp][row + 8][8 * i + col]) = make_float2(acc[i][2], acc[i][3]);
                    }
                }
                __syncwarp();
                if (half == 0) {
                    asm volatile("bar.arrive 1, %0;" ::"n"((DCH_WARPS + DCH_WRITERS) * 32) : "memory");
                    if (ch + 1 < chunks && !failed && !dch_wait(&m.wq_full[(ch + 1) & 1], (uint32_t)((ch + 1) >> 1) & 1u)) failed = true;
                    __syncwarp();
                }
                if (ch + 1 < chunks) read_rows(ch + 1, half);
            }
            if (!failed && !dch_wait(&m.k_full[b], (uint32_t)(ch >> 1) & 1u)) failed = true;
            __syncwarp();
            uint32_t u[2][3][4], k[2][3][4];
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int q = 0; q < 3; ++q)
                    dch_ldmatrix_turned(k[h][q], dch_saddr(keys + b * image + (h * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * ld + q * d + d0 + (lane >> 4) * 8));
            const float G = m.within[b][DCH_ALL];
            asm volatile("bar.sync 2, %0;" ::"n"(DCH_CHAIN) : "memory");
            if (owns) {                                         // S^T <- G S^T + (faded U)^T K
                float acc[2][2][4] = {};                        // [16 rows][8 components]
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int q = 0; q < 3; ++q) dch_ldmatrix(u[h][q], dch_saddr(&m.ud[q][(lane & 7) + ((lane >> 3) & 1) * 8][h * 16 + (lane >> 4) * 8]));
#pragma unroll
                for (int q = 0; q < PIECE_PRODUCTS; ++q)
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int i = 0; i < 2; ++i) dch_mma(acc[h][i], u[h][piece_a(q)], k[h][piece_b(q)][2 * i], k[h][piece_b(q)][2 * i + 1]);
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) S[i][j] = fmaf(G, S[i][j], acc[0][i][j] + acc[1][i][j]);
            }
        }
        if (owns)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float* to = st + row * d + d0 + 8 * h + col;
                to[0] = S[h][0], to[1] = S[h][1], to[8 * d] = S[h][2], to[8 * d + 1] = S[h][3];
            }
    }
    if (failed) atomicExch(&g_delta_chain_error, 1);
}

// Keys in whole 32 components, values in whole slices.
bool delta_chunks_take(int d, int e) { return d > 0 && d <= DCH_MAX_D && d % 32 == 0 && e > 0 && e % DCH_E == 0; }

static size_t dch_places(int rows, int entries, int from_rows) { return (size_t)rows / DCH_C + (entries < rows / from_rows ? entries : rows / from_rows) + 1; }
static size_t dch_image_floats(int d) { return (size_t)DCH_C * delta_piece_row(d) / 2; }
long long delta_chunk_floats(int rows, int entries, int from_rows, int heads, int kv_heads, int d, int e) {
    return (long long)(dch_places(rows, entries, from_rows) * (heads * (dch_image_floats(d) + DCH_WITHIN + (size_t)e * DCH_LD_W) + (size_t)kv_heads * 2 * dch_image_floats(d)));
}

int launch_delta_chunks(DeltaChunks p, float* scratch, int rows, int longest, cudaStream_t s) {
    const int chunks = (longest + DCH_C - 1) / DCH_C;
    KB_REQUIRE(p.kv_heads <= 65535 && p.entries <= 65535 && p.heads <= 65535, "delta: too many heads or requests for one launch");
    KB_REQUIRE(((uintptr_t)scratch & 15) == 0, "delta: scratch at %p is not at a multiple of 16 bytes", (void*)scratch);
    const size_t places = dch_places(rows, p.entries, p.from_rows);
    p.w = reinterpret_cast<__nv_bfloat16*>(scratch);
    p.qk = reinterpret_cast<__nv_bfloat16*>(scratch += places * p.heads * dch_image_floats(p.d));
    p.within = scratch += places * p.kv_heads * 2 * dch_image_floats(p.d);
    p.u0 = scratch + places * p.heads * DCH_WITHIN;
    if (cudaFuncSetAttribute(delta_chain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dch_smem(DCH_MAX_D)) != cudaSuccess)
        return fail("delta: cannot have %d bytes of shared memory", dch_smem(DCH_MAX_D));
    delta_chunk_kernel<<<dim3(chunks, p.heads, p.entries), DCH_THREADS, 0, s>>>(p);
    if (int err = check_launch("delta chunks")) return err;
    delta_chain_kernel<<<dim3(p.e / DCH_E, p.heads, p.entries), DCH_CHAIN, dch_smem(p.d), s>>>(p);
    return check_launch("delta chain");
}

}  // namespace kb

using namespace kb;

extern "C" int kb_delta_chain_error() {
    int flag = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&flag, g_delta_chain_error, sizeof(int)) != cudaSuccess) return -1;
    if (flag) cudaMemcpyToSymbol(g_delta_chain_error, &zero, sizeof(int));
    return flag;
}
