// The gated delta rule by chunks of rows: what `kb_delta_scan` hands to the kernels of delta_chunk.cu.
#pragma once
#include "common.cuh"

namespace kb {

constexpr int DCH_C = 32;              // rows a chunk
constexpr int DCH_LD_W = DCH_C + 4;    // a row of 32 weights, and four more so that rows begin in different banks
constexpr int DCH_G = DCH_C * DCH_LD_W, DCH_F = DCH_G + DCH_C, DCH_ALL = DCH_F + DCH_C, DCH_WITHIN = DCH_ALL + 4;      // the decays' places behind them

// Where a chunk's inputs lie: the chunk that begins at row `first` of a request with `before` requests by chunks in the rows ahead of it
// (`delta_chunks_before`), whatever the order in which the requests are listed. Requests have rows of their own, so every chunk has a place of its own.
__host__ __device__ inline int delta_chunk_place(int first, int before) { return first / DCH_C + before; }
__host__ __device__ inline int delta_piece_row(int d) { return 3 * d + 8; }             // 8 more: eight rows begin in different banks

struct DeltaChunks {
    const float* qn;            // [rows, kv_heads, d] unit queries times the query scale
    const float* kn;            // [rows, kv_heads, d] unit keys
    const float* vn;            // [rows, heads, e]
    const float* scal;          // [rows, heads, 2] decay, step size
    const float* kq;            // [rows, kv_heads] a row's key times its query
    // A chunk's inputs to the chain as they lie in its shared memory, chunk by chunk (`delta_chunk_place`); rows beyond the last are zeros.
    __nv_bfloat16* w;           // [places, heads, DCH_C, 3 d + 8]: what a row's write owes to the memory before the chunk, in three pieces of d
    __nv_bfloat16* qk;          // [places, kv_heads, 2, DCH_C, 3 d + 8]: unit queries times their scale, then unit keys, likewise
    float* within;              // [places, heads, DCH_WITHIN]: what row t reads of the chunk's row s, [DCH_C][DCH_LD_W]; then the decays from the
                                // chunk's start to the rows, from the rows to its end, over the whole chunk
    float* u0;                  // [places, heads, e, DCH_LD_W]: the writes with an empty memory before, by component
    float* state;               // [slots, state_floats], a head's memory [e, d] at state_off + head e d
    long long state_floats, state_off;
    const int* entry_start;
    const int* entry_end;
    const int* slots;
    int n_slots, entries, heads, kv_heads, d, e, from_rows;
    float* out;                 // [rows, heads, e]
};

// Whether the chunk kernels take these sizes.
bool delta_chunks_take(int d, int e);
// Floats of scratch for a step of `rows` rows whose requests of at least `from_rows` go by chunks.
long long delta_chunk_floats(int rows, int entries, int from_rows, int heads, int kv_heads, int d, int e);
// Requests that bring at least p.from_rows rows, `longest` being the most any brings.
// The inputs' places are taken from `scratch`.
int launch_delta_chunks(DeltaChunks p, float* scratch, int rows, int longest, cudaStream_t s);

}  // namespace kb
