// Pieces of float32 products over chunks of 64 tokens (state_space_tiles.cu, linear_attention_channels.cu): vector reads with a ragged end,
// multiply-adds in pairs, slices of a chunk's rows turned in shared memory, and where a thread's results lie.
#pragma once
#include "common.cuh"

#define ST_CHUNK 64                                       // tokens of a chunk
#define ST_THREADS 128
#define ST_SLICE 32                                       // state rows of C and S in shared memory at a time

__device__ __forceinline__ float4 st_load4(const float* p, int left, bool vec) {          // up to four entries, zeros behind `left`
    if (vec && left >= 4) return *reinterpret_cast<const float4*>(p);
    return make_float4(left > 0 ? p[0] : 0.f, left > 1 ? p[1] : 0.f, left > 2 ? p[2] : 0.f, left > 3 ? p[3] : 0.f);
}
__device__ __forceinline__ void st_store4(float* p, int left, bool vec, float4 v) {
    if (vec && left >= 4) { *reinterpret_cast<float4*>(p) = v; return; }
    if (left > 0) p[0] = v.x;
    if (left > 1) p[1] = v.y;
    if (left > 2) p[2] = v.z;
    if (left > 3) p[3] = v.w;
}
typedef unsigned long long st_pair;                        // two float32 numbers
__device__ __forceinline__ void st_fma(st_pair& acc, float a, st_pair b) {
    asm("{\n\t.reg .b64 aa;\n\tmov.b64 aa, {%1, %1};\n\tfma.rn.f32x2 %0, aa, %2, %0;\n\t}" : "+l"(acc) : "f"(a), "l"(b));
}
__device__ __forceinline__ float2 st_two(st_pair v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ float4 st_four(st_pair a, st_pair b) {
    const float2 x = st_two(a), y = st_two(b);
    return make_float4(x.x, x.y, y.x, y.y);
}

// Whether a value is an infinity or no number.  In a product of weights and a chunk's values a token's weight for the tokens in
// front of it is zero, which keeps it out of their sums only while its values are finite: chunks where they are not take the products
// token by token as far as they reach.  st_zero adds zeros of four values to z; z is zero afterwards unless one of them was odd.
// (No branch and no comparison: it stands among loads that are to be asked for together.)
__device__ __forceinline__ void st_zero(float& z, const float4& v) { z = fmaf(v.x, 0.f, fmaf(v.y, 0.f, fmaf(v.z, 0.f, fmaf(v.w, 0.f, z)))); }

// Columns c0 .. c0 + 31 of 64 rows (tokens) into dst[column][token]; entry (column k, token t) lies at k * 64 + (t ^ 4 ((k / 4) % 8)), so
// that neither the four stores of a thread nor the reads of four neighbouring tokens meet in a bank.
__device__ __forceinline__ int st_turned(int k, int t) { return k * ST_CHUNK + (t ^ (((k >> 2) & 7) << 2)); }
struct STSlice {
    float4 v[ST_CHUNK * ST_SLICE / 4 / ST_THREADS];
    __device__ __forceinline__ void load(const float* src, int ld, int n, int left, bool vec) {
#pragma unroll
        for (int e = 0; e < ST_CHUNK * ST_SLICE / 4 / ST_THREADS; ++e) {
            const int i = threadIdx.x + e * ST_THREADS, t = i >> 3, c = (i & 7) * 4;
            v[e] = t < n ? st_load4(src + (size_t)t * ld + c, left - c, vec) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    __device__ __forceinline__ void store_turned(float* dst) const {
#pragma unroll
        for (int e = 0; e < ST_CHUNK * ST_SLICE / 4 / ST_THREADS; ++e) {
            const int i = threadIdx.x + e * ST_THREADS, t = i >> 3, c = (i & 7) * 4;
            dst[st_turned(c, t)] = v[e].x; dst[st_turned(c + 1, t)] = v[e].y;
            dst[st_turned(c + 2, t)] = v[e].z; dst[st_turned(c + 3, t)] = v[e].w;
        }
    }
};
// 8 x 16 threads over 64 x 64 results: a thread the rows ty * 4 + 32 i + 0..3 and columns tx * 4 + 0..3; a warp is four by eight threads.
__device__ __forceinline__ void st_place(int& ty, int& tx) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    ty = (warp >> 1) * 4 + (lane >> 3);
    tx = (warp & 1) * 8 + (lane & 7);
}
// acc += weights x values over a chunk's first `last` tokens: weights [64 s][64 t], values [64 s][64 columns].  guarded: some value is no
// finite number, and a token joins the sums of none in front of it.
__device__ __forceinline__ void st_weighted(st_pair (&acc)[8][2], const float* weights, const float* values, int last, int ty, int tx, bool guarded) {
#pragma unroll 4
    for (int s = 0; s < (guarded ? 0 : last); ++s) {
        float w[8];
        *reinterpret_cast<float4*>(w) = *reinterpret_cast<const float4*>(weights + s * ST_CHUNK + ty * 4);
        *reinterpret_cast<float4*>(w + 4) = *reinterpret_cast<const float4*>(weights + s * ST_CHUNK + ty * 4 + 32);
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(values + s * 64 + tx * 4);
#pragma unroll
        for (int i = 0; i < 8; ++i) { st_fma(acc[i][0], w[i], v.x); st_fma(acc[i][1], w[i], v.y); }
    }
#pragma unroll 1
    for (int s = 0; s < (guarded ? last : 0); ++s) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(values + s * 64 + tx * 4);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int t = ty * 4 + 32 * (i / 4) + i % 4;
            if (s <= t) { st_fma(acc[i][0], weights[s * ST_CHUNK + t], v.x); st_fma(acc[i][1], weights[s * ST_CHUNK + t], v.y); }
        }
    }
}
