// Where linear attention's kernels for the tensor cores (linear_attention_tcgen05.cu) find a chunk's operands, and what the two kernels that work
// them out (there with a decay per head, linear_attention_channels.cu with one per channel) share.
#pragma once
#include "linear_attention.cuh"
#include "chunk_mma.cuh"

// A unit's parts in scratch: queries and keys, [part][two][64 tokens][64 channels] each (two: the channels' halves, or the heads), and weights
// [part][heads][64 t][64 s]; and values behind their activation, [part][half][64 s][64 columns].
template <bool TWO> struct LMUnit {
    static constexpr int ND = TWO ? 64 : 128;             // rows of a head's state
    static constexpr int QUERIES = 0, KEYS = 6 * CM_PLANE, WEIGHTS = 12 * CM_PLANE, W_HEADS = TWO ? 2 : 1, VALUES = (12 + 3 * W_HEADS) * CM_PLANE, BYTES = VALUES + 6 * CM_PLANE;
    // of a head h
    static __device__ __forceinline__ unsigned char* of(const LAArgs& a, int c, int h) { return a.chunk_planes + ((size_t)c * (TWO ? a.H / 2 : a.H) + (TWO ? h / 2 : h)) * BYTES; }
};

// Tiles of a chunk's and head's word: 0 queries, 1 keys (with one decay a head), 2 weights, 3 values, 4 keys times their decays.
// From bit 16 on the first token with an entry that parts do not hold.

// Eight neighbouring numbers of a row, zeros behind the chunk's tokens.
template <typename TQ>
__device__ __forceinline__ void lm_eight(float (&v)[8], const TQ* p, bool there, bool vec) {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = 0.f;
    if (!there) return;
    if (vec) {
        if constexpr (sizeof(TQ) == 4) {
            *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(p);
            *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(p + 4);
        } else {
            const uint4 r = *reinterpret_cast<const uint4*>(p);
            const unsigned w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) { v[2 * i] = __uint_as_float(w[i] << 16); v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = to_f(p[i]);
    }
}
__device__ __forceinline__ void lm_put(unsigned char* to, int stride, const float (&v)[8], unsigned& most) {
    cm_put(to, stride, make_float4(v[0], v[1], v[2], v[3]), make_float4(v[4], v[5], v[6], v[7]), most);
}
__device__ __forceinline__ unsigned lm_value_seen(unsigned most, int act) { return act ? cm_seen(most, 3) : cm_odd(cm_seen(most, 0)) ? 1u << 9 : 2u << 9; }      // (one part holds any finite value)
// Eight values of a token: parts behind their activation; without one they are only looked at.
__device__ __forceinline__ void lm_values(const LAArgs& a, unsigned char* to, const bf16* from, bool there, int row, unsigned* first_odd, unsigned& most) {
    unsigned mine = 0;
    if (a.act_v) {
        float v[8];
        lm_eight(v, from, there, true);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = la_act<true>(v[i], a.act_v);
        lm_put(to, 2 * CM_PLANE, v, mine);
    } else if (there) {
        const uint4 r = *reinterpret_cast<const uint4*>(from);
        cm_watch(mine, r.x); cm_watch(mine, r.y); cm_watch(mine, r.z); cm_watch(mine, r.w);
    }
    if (cm_odd(cm_seen(mine, 0))) atomicMin(first_odd, (unsigned)row);
    cm_watch(most, mine);
}
