// The gated delta rule by chunks of rows: what `kb_delta_scan` hands to the kernels of delta_chunk.cu.
#pragma once
#include "common.cuh"

namespace kb {

constexpr int DCH_C = 32;              // rows a chunk

struct DeltaChunks {
    const float* qn;            // [rows, kv_heads, d] unit queries times the query scale
    const float* kn;            // [rows, kv_heads, d] unit keys
    const float* vn;            // [rows, heads, e]
    const float* scal;          // [rows, heads, 2] decay, step size
    const float* kq;            // [rows, kv_heads] a row's key times its query
    float* w;                   // [rows, heads, d]: what a chunk's writes owe to the memory before it
    float* u0;                  // [rows, heads, e]: the writes with an empty memory before
    float* within;              // [rows, heads, DCH_C]: what row t reads of the chunk's row s
    float* fade;                // [rows, heads, 2]: decay from the chunk's start to the row, from the row to the chunk's end
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
// Requests that bring at least p.from_rows rows, `longest` being the most any brings.
int launch_delta_chunks(const DeltaChunks& p, int longest, cudaStream_t s);

}  // namespace kb
