// What the kernels of linear attention share: the description of a call, the activation of the projections, the cut of a step's
// packed tokens into chunks, and the tile kernels' launchers.
#pragma once
#include "common.cuh"

#define LA_CHUNK 64

struct LAArgs {
    const void* proj; int ld, q_off, k_off, v_off;
    const void* qk; int qk_ld;                 // the rows q and k are read from (proj itself, or float32 rows of their own)
    const void* z; int z_ld;
    const float* head_decay;
    float inv_tau, q_scale;
    int act_qk, act_v;
    float* state; long long state_stride;
    const int* row_first; const int* row_lens; const int* slots;
    float* out;
    int B, H, D, Dv;
    float* chunk_state;      // [chunks, H, D, Dv]
    float* chunk_decay;      // [chunks, H, D]
    int chunks;              // of the step, at most
    int first_chunk, slab;   // those that this launch takes: from first_chunk on, `slab` of them at most
    float* channel_scratch;  // with a decay per channel: weights, decayed queries and keys of every chunk
    // on the tensor cores (linear_attention_tcgen05.cu):
    unsigned char* chunk_planes;   // the units' queries, keys and weights as bfloat16 parts
    unsigned* chunk_seen;          // [chunks][H]: what cm_watch saw of them
    int2* chunk_rows;              // [chunks]: first packed token and number of tokens
    int* unit_exact;               // [chunks][units]: tokens of a unit's chunk whose outputs come from parts
    int* status;
    int qk_f32, z_f32;
};

// silu of a projection.  FAST (the bfloat16 engine, whose projections carry 8 bits): 2^x and the reciprocal from the
// special-function unit, relative error about 2^-22; else the exact routines.  A block applies it to every q and k entry of
// its head for each of its tokens, so its cost is paid once per 32 columns of the state.
template <bool FAST>
__device__ __forceinline__ float la_act(float v, int act) {
    if (act != 1) return v;
    if (FAST) {
        float e, r;
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(-1.4426950408889634f * v));
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
        return v * r;
    }
    return v / (1.0f + expf(-v));
}

// pw[i] = a^i for i <= 64 (a^0 = 1, also for a = 0)
__device__ __forceinline__ void la_powers(float* pw, float a) {
    const int i = threadIdx.x;
    if (i <= LA_CHUNK) {
        double r = 1.0, b = (double)a;
        for (int e = i; e; e >>= 1) { if (e & 1) r *= b; b *= b; }
        pw[i] = (float)r;
    }
}

// Which sequence chunk `c` of the step belongs to, its first packed token and its number of tokens (0: no such chunk).
__device__ __forceinline__ void la_find_chunk(const int* row_first, const int* row_lens, int B, int c, int& row, int& first, int& count) {
    int base = 0;
    row = -1; first = 0; count = 0;
    for (int b = 0; b < B; ++b) {
        const int n = row_lens[b], nc = (n + LA_CHUNK - 1) / LA_CHUNK;
        if (c < base + nc) {
            const int local = c - base;
            row = b; first = row_first[b] + local * LA_CHUNK;
            count = min(LA_CHUNK, n - local * LA_CHUNK);
            return;
        }
        base += nc;
    }
}

// Prompts with a decay per head, as products of tiles (linear_attention_tiles.cu): every chunk's contribution to the state, and, once
// each chunk's incoming state stands where its contribution was, every chunk's outputs.  `types`: 0 float32; 1 bfloat16 rows;
// 2 bfloat16 rows with float32 queries and keys of their own.
int la_tiles_contributions(const LAArgs& a, int types, cudaStream_t s);
int la_tiles_outputs(const LAArgs& a, int types, cudaStream_t s);
// The same with a decay per channel (linear_attention_channels.cu).
long long la_channels_scratch_floats(int chunks, int H, int D);
int la_channels_contributions(const LAArgs& a, bool f32, bool z_f32, float* scratch, cudaStream_t s);
int la_channels_outputs(const LAArgs& a, bool f32, float* scratch, cudaStream_t s);
// Both on the tensor cores (linear_attention_tcgen05.cu), all of a slab's launches; and the floats of scratch that a chunk takes beside its states and decays.
int la_tensor_chunks(const LAArgs& a, int types, int z_types, cudaStream_t s);
long long la_tensor_chunk_floats(int H, int D, bool values);      // values: they go through an activation
