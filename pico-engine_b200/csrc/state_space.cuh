// What the recurrence of the state-space mixer (state_space.cu) and its form as products of tiles (state_space_tiles.cu) share.
#pragma once
#include "common.cuh"

#define SS_CHUNK 64          // tokens of a chunk of a prompt

#define SS_STEP_FLOATS (4 * 64)               // of a chunk of 64 tokens and a head
#define SS_MATRIX_STEP_FLOATS (20 * 64)       // the same for products on the tensor cores

// Whether prompts' products run on the tensor cores (state_space_tcgen05.cu), and the bytes of a chunk's and group's parts of B (and of C) there.
inline bool ss_on_tensor_cores(int H, int P, int N, int G) { return P == 64 && (N == 64 || N == 128) && H / G % 2 == 0; }
__host__ __device__ __forceinline__ size_t ss_plane_bytes(int N) { return (size_t)(N / 64) * 3 * 8192; }

struct ScanArgs {
    const float* xbc; int xbc_ld;             // [T, inner + 2 G N] float32: x | B | C after the convolution
    const void* proj; int proj_ld, dt_off;    // dt_raw at columns dt_off .. dt_off + H - 1 of proj (the step's dtype)
    const void* dt_bias; int dtb_dtype; const void* a_log; int al_dtype; const void* d_skip; int d_dtype;   // [H] each
    float* state; long long state_stride;     // row slots[b] holds the sequence's state
    const int* row_first; const int* row_lens; const int* slots;
    float* y;                                 // [T, H * P]
    int B, H, P, N, G, NS, NR, NRP, PT;
    float* chunk_state;                       // [chunks][H][N][P]: a chunk's own contribution, then its incoming state
    float* chunk_decay;                       // [chunks][H]: the product of a chunk's decays
    float* chunk_scores;                      // [chunks][G][64 s][64 t]: C_t . B_s (tensor cores: [64 t][64 s])
    float* chunk_steps;                       // [chunks][H][SS_STEP_FLOATS]: 64 x (dt, dt * the decays behind it), then 64 running sums (float64);
                                              // tensor cores: [chunks][H][SS_MATRIX_STEP_FLOATS], SM_WS and on (state_space_tcgen05.cu)
    unsigned char* chunk_planes;              // tensor cores: [chunks][G][B, C][64 state rows at a time]: their bfloat16 parts (chunk_mma.cuh)
    unsigned* chunk_seen;                     // [chunks][G]: whether B has numbers that parts are not made of; from bit 16 on the first token where B or C has an entry that they are not made of (64: none)
    int* unit_exact;                          // [chunks][H / 2]: tokens of a chunk and two heads whose results come from parts
    int2* chunk_rows;                         // [chunks]: first packed token and number of tokens
    int chunks;                               // of the step, at most
    int first_chunk, slab;                    // those that a launch takes: from first_chunk on, `slab` of them at most
};

__device__ __forceinline__ float ss_silu(float v) { return v / (1.0f + expf(-v)); }
__device__ __forceinline__ float ss_softplus(float v) { return fmaxf(v, 0.f) + log1pf(expf(-fabsf(v))); }

// Which sequence chunk `c` belongs to, its first packed token and its number of tokens (0: no such chunk).
__device__ __forceinline__ void ss_find_chunk(const ScanArgs& a, int c, int& first, int& count) {
    first = count = 0;
    for (int b = 0; b < a.B; ++b) {
        const int n = a.row_lens[b], nc = (n + SS_CHUNK - 1) / SS_CHUNK;
        if (c < nc) { first = a.row_first[b] + c * SS_CHUNK; count = min(SS_CHUNK, n - c * SS_CHUNK); return; }
        c -= nc;
    }
}

int ss_tensor_tiles(const ScanArgs& a, int dtype, int* status, cudaStream_t s);
int ss_tiles(const ScanArgs& a, int dtype, cudaStream_t s);     // prompts: contributions, carry, outputs
