// The gated delta rule over long portions of prompts, by chunks of 32 rows: the steps of the scan
//     S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q
// summed in another order. With the memory S_0 before a chunk, G_t the decay from the chunk's start up to and with row t and D_ts the
// decay of the rows s + 1 .. t (products of the rows' decays, never quotients: a decay of 0 is a decay like any other),
//     u_t = beta_t (v_t - G_t S_0^T k_t - sum_{s < t} D_ts (k_s . k_t) u_s)
// so U = U0 - W S_0, where (I + A) [W | U0] = [beta G K | beta V], A_ts = beta_t D_ts (k_t . k_s) below the diagonal: a forward substitution
// that needs no memory, chunk by chunk side by side. Then
//     o_t = G_t S_0^T q_t + sum_{s <= t} D_ts (q_t . k_s) u_s,     S = G_C S_0 + sum_s D_Cs k_s u_s^T.
// `delta_chunk_kernel`, a block a chunk and key head: the keys against the keys and the queries, and for every head of that key head W, U0,
// the weights within the chunk and the decays. `delta_chain_kernel`, a block a head and 16 of its value components of one request: the
// chain over the chunks, the memory's 16 columns in shared memory, the next chunk's inputs fetched meanwhile. Everything is 32-bit
// multiply-adds. What bounds the chain is shared memory's 32 words a clock (0.4 words a product) and the waits between its four parts: 3.9
// us a chunk, where the scan's 32 steps take 9.7. 2,048 rows, 16 heads of 128 over 4 key heads: 54 us for the chunks and 249 us for the chain
// (the scan: 619 us). Sums go by short chains, so that the error against 64 bits stays at the scan's: 1.01 to 1.07 of it where memories fade within
// a row to some twenty rows, 0.99 of it where they hardly do; in one chain over all components it was 1.4 to 1.6.
#include "delta_chunk.cuh"

namespace kb {

constexpr int DCH_THREADS = 256, DCH_E = 16, DCH_MAX_D = 128, DCH_LD = DCH_MAX_D + 4;

__device__ __forceinline__ void dch_copy16(float* dst, const float* src, bool there) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(there ? 16 : 0) : "memory");
}

__global__ void __launch_bounds__(DCH_THREADS, 2)
delta_chunk_kernel(const DeltaChunks p) {
    __shared__ __align__(16) float sk[DCH_C][DCH_LD], sq[DCH_C][DCH_LD];
    __shared__ __align__(16) float kk[DCH_C][DCH_C + 4], qk[DCH_C][DCH_C + 4], decay[DCH_C][DCH_C + 4];      // [t][s]
    __shared__ float sg[DCH_C], sbeta[DCH_C];
    const int entry = blockIdx.z, kvh = blockIdx.y;
    const int r0 = p.entry_start[entry], r1 = p.entry_end[entry];
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
    {   // a thread: row t against four rows s of the chunk
        const int t = tid >> 3, s0 = (tid & 7) * 4;
        float a[4] = {}, b[4] = {};
        for (int x0 = 0; x0 < d; x0 += 32) {                    // 32 components in four chains of eight: the rounding of a warp's sum of lanes
            float4 ka[4] = {}, qa[4] = {};
#pragma unroll 2
            for (int x = x0; x < x0 + 32; x += 4) {
                const float4 k = *reinterpret_cast<const float4*>(&sk[t][x]), q = *reinterpret_cast<const float4*>(&sq[t][x]);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float4 o = *reinterpret_cast<const float4*>(&sk[s0 + j][x]);
                    ka[j].x = fmaf(k.x, o.x, ka[j].x), ka[j].y = fmaf(k.y, o.y, ka[j].y), ka[j].z = fmaf(k.z, o.z, ka[j].z), ka[j].w = fmaf(k.w, o.w, ka[j].w);
                    qa[j].x = fmaf(q.x, o.x, qa[j].x), qa[j].y = fmaf(q.y, o.y, qa[j].y), qa[j].z = fmaf(q.z, o.z, qa[j].z), qa[j].w = fmaf(q.w, o.w, qa[j].w);
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                a[j] += (ka[j].x + ka[j].y) + (ka[j].z + ka[j].w);
                b[j] += (qa[j].x + qa[j].y) + (qa[j].z + qa[j].w);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)                             // a row against itself: as the scan has it, from before the vectors were rounded
            kk[t][s0 + j] = a[j], qk[t][s0 + j] = s0 + j == t && t < n ? p.kq[(size_t)(first + t) * p.kv_heads + kvh] : b[j];
    }
    auto am = sq;                                               // [t][s] the substitution's matrix, once the queries are done with
    const int per = p.heads / p.kv_heads;
    for (int h = kvh * per; h < (kvh + 1) * per; ++h) {
        __syncthreads();                                        // the products are there; the head before is done with the decays
        if (tid < DCH_C) {
            const float2 gb = tid < n ? *reinterpret_cast<const float2*>(p.scal + ((size_t)(first + tid) * p.heads + h) * 2) : make_float2(1.f, 0.f);
            sg[tid] = gb.x, sbeta[tid] = gb.y;
            __syncwarp();
            float D = 0.f, G = 1.f;
#pragma unroll 8
            for (int t = 0; t < DCH_C; ++t) {                   // column s = tid of the decays: zero above the diagonal, 1 on it
                D = t == tid ? 1.f : D * sg[t];
                decay[t][tid] = D;
                G = t <= tid ? G * sg[t] : G;
            }
            if (tid < n) *reinterpret_cast<float2*>(p.fade + ((size_t)(first + tid) * p.heads + h) * 2) = make_float2(G, decay[n - 1][tid]);
        }
        __syncthreads();
        for (int i = tid; i < DCH_C * DCH_C; i += DCH_THREADS) {
            const int t = i / DCH_C, s = i % DCH_C;
            if (t < n) p.within[((size_t)(first + t) * p.heads + h) * DCH_C + s] = s <= t ? decay[t][s] * qk[t][s] : 0.f;
            am[t][s] = s < t ? sbeta[t] * decay[t][s] * kk[t][s] : 0.f;
        }
        __syncthreads();
        // the substitution, a column of [beta G K | beta V] a thread: its 32 values are asked for before the first is needed
        for (int c = tid; c < d + e; c += DCH_THREADS) {
            float x[DCH_C];
            float G = 1.f;
#pragma unroll
            for (int t = 0; t < DCH_C; ++t) {
                G *= sg[t];
                const float v = c < d ? G * sk[t][c] : p.vn[((size_t)(first + min(t, n - 1)) * p.heads + h) * e + (c - d)];
                x[t] = sbeta[t] * v;                            // beta is 0 beyond the last row
            }
#pragma unroll
            for (int t = 1; t < DCH_C; ++t) {
                float sum[2] = {0.f, 0.f};
#pragma unroll
                for (int s = 0; s < t; s += 4) {                // zeros on and above the diagonal
                    const float4 a = *reinterpret_cast<const float4*>(&am[t][s]);
                    sum[0] = fmaf(a.x, x[s], sum[0]);
                    if (s + 1 < t) sum[1] = fmaf(a.y, x[s + 1], sum[1]);
                    if (s + 2 < t) sum[0] = fmaf(a.z, x[s + 2], sum[0]);
                    if (s + 3 < t) sum[1] = fmaf(a.w, x[s + 3], sum[1]);
                }
                x[t] -= sum[0] + sum[1];
            }
#pragma unroll
            for (int t = 0; t < DCH_C; ++t)
                if (t < n) {
                    if (c < d) p.w[((size_t)(first + t) * p.heads + h) * d + c] = x[t];
                    else p.u0[((size_t)(first + t) * p.heads + h) * e + (c - d)] = x[t];
                }
        }
    }
}

// Shared memory of the chain: two sets of a chunk's inputs (W, queries, keys [32][d], weights within [32][32], U0 [32][16], decays), the
// memory's columns [d][16], the chunk's writes (as they are, and faded to the chunk's end), and the eight warps' partial sums.
struct DchBuf {
    float w[DCH_C][DCH_LD], q[DCH_C][DCH_LD], k[DCH_C][DCH_LD], within[DCH_C][DCH_C + 4], u0[DCH_C][DCH_E], fade[DCH_C][2];
};
struct DchSmem {
    DchBuf in[2];
    float S[DCH_MAX_D][DCH_E + 4];
    float u[DCH_C][DCH_E], ud[DCH_C][DCH_E];
    float part[8][2 * DCH_C][DCH_E + 4];
};

__global__ void __launch_bounds__(DCH_THREADS, 1)
delta_chain_kernel(const DeltaChunks p) {
    extern __shared__ __align__(16) unsigned char dch_raw[];
    DchSmem& m = *reinterpret_cast<DchSmem*>(dch_raw);
    const int entry = blockIdx.z, head = blockIdx.y, c0 = blockIdx.x * DCH_E;
    const int r0 = p.entry_start[entry], r1 = p.entry_end[entry];
    const int slot = p.slots[entry];
    if (r1 - r0 < p.from_rows) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, d = p.d, e = p.e, d4 = d >> 2;
    if (slot <= 0 || slot >= p.n_slots) {                       // rows of no request: zeros, no state
        for (int i = tid; i < (r1 - r0) * DCH_E; i += DCH_THREADS) p.out[((size_t)(r0 + i / DCH_E) * p.heads + head) * e + c0 + i % DCH_E] = 0.f;
        return;
    }
    const int kvh = head / (p.heads / p.kv_heads);
    float* st = p.state + (size_t)slot * p.state_floats + p.state_off + ((size_t)head * e + c0) * d;      // [16][d]: a column of the memory lies together
    for (int i = tid; i < DCH_E * d; i += DCH_THREADS) m.S[i % d][i / d] = st[i];
    const int chunks = (r1 - r0 + DCH_C - 1) / DCH_C;
    auto fetch = [&](int chunk) {
        if (chunk < chunks) {
            DchBuf& b = m.in[chunk & 1];
            const int first = r0 + chunk * DCH_C, n = min(DCH_C, r1 - first);
            for (int i = tid; i < DCH_C * d4; i += DCH_THREADS) {
                const int t = i / d4, x = (i - t * d4) * 4;
                const bool there = t < n;                       // rows beyond the last are zeros
                const size_t r = (size_t)(first + (there ? t : 0));
                dch_copy16(&b.w[t][x], p.w + (r * p.heads + head) * d + x, there);
                dch_copy16(&b.q[t][x], p.qn + (r * p.kv_heads + kvh) * d + x, there);
                dch_copy16(&b.k[t][x], p.kn + (r * p.kv_heads + kvh) * d + x, there);
            }
            {
                const int t = tid >> 3, x = (tid & 7) * 4;      // 32 rows x 8 pieces
                const bool there = t < n;
                const size_t r = (size_t)(first + (there ? t : 0));
                dch_copy16(&b.within[t][x], p.within + (r * p.heads + head) * DCH_C + x, there);
                if (x < DCH_E) dch_copy16(&b.u0[t][x], p.u0 + (r * p.heads + head) * e + c0 + x, there);
            }
            if (tid < DCH_C) {
                const float2 f = tid < n ? *reinterpret_cast<const float2*>(p.fade + ((size_t)(first + tid) * p.heads + head) * 2) : make_float2(0.f, 0.f);
                b.fade[tid][0] = f.x, b.fade[tid][1] = f.y;
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0);
    const int rg = lane >> 2, cg = (lane & 3) * 4;              // a thread's rows rg, rg + 8, .. and its four columns
    const int span = d >> 3, k_lo = warp * span;                // a warp's share of the inner dimension
    for (int ch = 0; ch < chunks; ++ch) {
        fetch(ch + 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                                        // the chunk's inputs are there, and the memory behind the chunk before
        const DchBuf& b = m.in[ch & 1];
        const int first = r0 + ch * DCH_C, n = min(DCH_C, r1 - first);
        {   // W S and Q S: 64 rows x 16 columns, a warp an eighth of the inner dimension
            float acc[8][4] = {};
            for (int x = k_lo; x < k_lo + span; x += 4) {
                float4 s[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) s[j] = *reinterpret_cast<const float4*>(&m.S[x + j][cg]);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float4 a = *reinterpret_cast<const float4*>(i < 4 ? &b.w[rg + 8 * i][x] : &b.q[rg + 8 * (i - 4)][x]);
                    acc[i][0] = fmaf(a.x, s[0].x, acc[i][0]), acc[i][1] = fmaf(a.x, s[0].y, acc[i][1]), acc[i][2] = fmaf(a.x, s[0].z, acc[i][2]), acc[i][3] = fmaf(a.x, s[0].w, acc[i][3]);
                    acc[i][0] = fmaf(a.y, s[1].x, acc[i][0]), acc[i][1] = fmaf(a.y, s[1].y, acc[i][1]), acc[i][2] = fmaf(a.y, s[1].z, acc[i][2]), acc[i][3] = fmaf(a.y, s[1].w, acc[i][3]);
                    acc[i][0] = fmaf(a.z, s[2].x, acc[i][0]), acc[i][1] = fmaf(a.z, s[2].y, acc[i][1]), acc[i][2] = fmaf(a.z, s[2].z, acc[i][2]), acc[i][3] = fmaf(a.z, s[2].w, acc[i][3]);
                    acc[i][0] = fmaf(a.w, s[3].x, acc[i][0]), acc[i][1] = fmaf(a.w, s[3].y, acc[i][1]), acc[i][2] = fmaf(a.w, s[3].z, acc[i][2]), acc[i][3] = fmaf(a.w, s[3].w, acc[i][3]);
                }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
                *reinterpret_cast<float4*>(&m.part[warp][rg + 8 * i][cg]) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        }
        __syncthreads();
        // a thread: four columns of one of the 64 rows, the eight shares added up
        const int row = tid >> 2, col = (tid & 3) * 4;
        float4 total = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w8 = 0; w8 < 8; w8 += 2) {
            const float4 v = *reinterpret_cast<const float4*>(&m.part[w8][row][col]), w = *reinterpret_cast<const float4*>(&m.part[w8 + 1][row][col]);
            total.x += v.x + w.x, total.y += v.y + w.y, total.z += v.z + w.z, total.w += v.w + w.w;
        }
        if (row < DCH_C) {                                      // U = U0 - W S
            const float4 v = *reinterpret_cast<const float4*>(&b.u0[row][col]);
            const float f = b.fade[row][1];
            const float4 u = make_float4(v.x - total.x, v.y - total.y, v.z - total.z, v.w - total.w);
            *reinterpret_cast<float4*>(&m.u[row][col]) = u;
            *reinterpret_cast<float4*>(&m.ud[row][col]) = make_float4(f * u.x, f * u.y, f * u.z, f * u.w);
        }
        __syncthreads();
        if (row >= DCH_C) {                                     // the read-outs: G Q S (this thread's sums) + the chunk's own writes
            const int t = row - DCH_C;
            const float G = b.fade[t][0];
            float4 o = make_float4(G * total.x, G * total.y, G * total.z, G * total.w);
            // Up to the row itself: a later row's write may be no finite number, and then a weight of zero does not keep it out. A warp has
            // eight rows, t0 .. t0 + 7: whole pieces of four sources below t0, the eight that lie among its rows each to the rows from it on.
            const int t0 = (t >> 3) << 3;
            float4 below = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int s = 0; s < DCH_C; s += 4) {
                if (s >= t0 + 8) break;                         // the same for the whole warp
                const float4 a = *reinterpret_cast<const float4*>(&b.within[t][s]);
                const float aw[4] = {a.x, a.y, a.z, a.w};
                if (s < t0) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float4 u = *reinterpret_cast<const float4*>(&m.u[s + j][col]);
                        below.x = fmaf(aw[j], u.x, below.x), below.y = fmaf(aw[j], u.y, below.y), below.z = fmaf(aw[j], u.z, below.z), below.w = fmaf(aw[j], u.w, below.w);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float4 u = *reinterpret_cast<const float4*>(&m.u[s + j][col]);
                        const bool takes = s + j <= t;
                        o.x = takes ? fmaf(aw[j], u.x, o.x) : o.x, o.y = takes ? fmaf(aw[j], u.y, o.y) : o.y;
                        o.z = takes ? fmaf(aw[j], u.z, o.z) : o.z, o.w = takes ? fmaf(aw[j], u.w, o.w) : o.w;
                    }
                }
                if (s + 4 == t0) o.x += below.x, o.y += below.y, o.z += below.z, o.w += below.w;
            }
            if (t < n) *reinterpret_cast<float4*>(p.out + ((size_t)(first + t) * p.heads + head) * e + c0 + col) = o;
        } else if ((tid >> 2) < d4) {                           // the memory behind the chunk: four of its rows x four columns a thread
            const int x = (tid >> 2) * 4;
            const float G = b.fade[n - 1][0];
            float s[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 v = *reinterpret_cast<const float4*>(&m.S[x + i][col]);
                s[i][0] = G * v.x, s[i][1] = G * v.y, s[i][2] = G * v.z, s[i][3] = G * v.w;
            }
#pragma unroll 8
            for (int t = 0; t < DCH_C; ++t) {
                const float4 k = *reinterpret_cast<const float4*>(&b.k[t][x]), u = *reinterpret_cast<const float4*>(&m.ud[t][col]);
                const float kx[4] = {k.x, k.y, k.z, k.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    s[i][0] = fmaf(kx[i], u.x, s[i][0]), s[i][1] = fmaf(kx[i], u.y, s[i][1]), s[i][2] = fmaf(kx[i], u.z, s[i][2]), s[i][3] = fmaf(kx[i], u.w, s[i][3]);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(&m.S[x + i][col]) = make_float4(s[i][0], s[i][1], s[i][2], s[i][3]);
        }
        __syncthreads();                                        // the chunk's inputs may be written over, the memory read
    }
    for (int i = tid; i < DCH_E * d; i += DCH_THREADS) st[i] = m.S[i % d][i / d];
}

// Keys in whole eighths of whole 16-byte pieces, values in whole slices.
bool delta_chunks_take(int d, int e) { return d > 0 && d <= DCH_MAX_D && d % 32 == 0 && e > 0 && e % DCH_E == 0; }

int launch_delta_chunks(const DeltaChunks& p, int longest, cudaStream_t s) {
    const int chunks = (longest + DCH_C - 1) / DCH_C;
    KB_REQUIRE(p.kv_heads <= 65535 && p.entries <= 65535 && p.heads <= 65535, "delta: too many heads or requests for one launch");
    static bool attr_set = false;
    if (!attr_set) {
        if (cudaFuncSetAttribute(delta_chain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DchSmem)) != cudaSuccess)
            return fail("delta: cannot have %d bytes of shared memory", (int)sizeof(DchSmem));
        attr_set = true;
    }
    delta_chunk_kernel<<<dim3(chunks, p.kv_heads, p.entries), DCH_THREADS, 0, s>>>(p);
    if (int err = check_launch("delta chunks")) return err;
    delta_chain_kernel<<<dim3(p.e / DCH_E, p.heads, p.entries), DCH_THREADS, sizeof(DchSmem), s>>>(p);
    return check_launch("delta chain");
}

}  // namespace kb
