// Linear attention of prompts with a decay per key channel and token, as products of tiles in float32 (linear_attention.cu has the
// recurrence itself).
//
// A sequence's tokens are cut into chunks of up to 64, a chunk into four runs of 16.  With A(s, t) = a_(s+1) .. a_t, channel by channel:
//   contribution of a chunk to the state      L = sum_s (A(s, n-1) k_s) v_s^T                                      [D, Dv]
//   its outputs, from the incoming state S    o_t = S^T (A(-1, t) q_t) + sum_{s <= t} (q_t . A(s, t) k_s) v_s      [n, Dv]
// Every product of decays is formed forwards, from factors of at most one: between two runs A(s, t) splits into what follows s in its run,
// the whole runs between, and what leads to t in its run; inside a run it is walked.  (A factored form with 1 / A would overflow: a decay
// may be anything down to zero.)  So a first kernel works out a head's weights q_t . A(s, t) k_s and the queries and keys times their
// decays, and what remains are plain products.
//
// Bound by float32 multiply-adds (fma.rn.f32x2) and, in the first kernel, by the decays' exponentials and logarithms.  2,048 tokens, 16
// heads of 128 x 128, on a B200: 258 us as two walks of every chunk, 160 us here (weights 71, contributions 39, outputs 50); the
// logits come as the product before wrote them (as float32 they were converted first, 10.5 us).  bfloat16 rows of heads of 64 x 64 and 128 x 128 go
// another way (linear_attention_tcgen05.cu).
#include "linear_attention.cuh"
#include "chunk_tiles.cuh"

#define LC_THREADS 256
#define LC_RUN 16
#define LC_LD (ST_CHUNK + 4)                              // entries between two channels in shared memory: neighbours lie four banks apart

// a = sigmoid(z)^(inv_tau), through the logarithm: -softplus(-z) * inv_tau (as the walk has it)
__device__ __forceinline__ float lc_decay(float z, float inv_tau) {
    const float u = -z;
    return expf(-(fmaxf(u, 0.f) + log1pf(expf(-fabsf(u)))) * inv_tau);
}
template <typename T>
__device__ __forceinline__ float4 lc_load4(const T* p, int left, bool vec) {          // up to four entries, zeros behind `left`
    if constexpr (sizeof(T) == 4) return st_load4((const float*)p, left, vec);
    else {
        if (vec && left >= 4) {
            const uint2 r = *reinterpret_cast<const uint2*>(p);
            const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.y));
            return make_float4(a.x, a.y, b.x, b.y);
        }
        return make_float4(left > 0 ? to_f(p[0]) : 0.f, left > 1 ? to_f(p[1]) : 0.f, left > 2 ? to_f(p[2]) : 0.f, left > 3 ? to_f(p[3]) : 0.f);
    }
}

__device__ __forceinline__ void lc_read16(float (&v)[LC_RUN], const float* p) {
#pragma unroll
    for (int t = 0; t < LC_RUN; t += 4) *reinterpret_cast<float4*>(v + t) = *reinterpret_cast<const float4*>(p + t);
}
__device__ __forceinline__ void lc_write16(float* p, const float (&v)[LC_RUN]) {
#pragma unroll
    for (int t = 0; t < LC_RUN; t += 4) *reinterpret_cast<float4*>(p + t) = *reinterpret_cast<const float4*>(v + t);
}

// A chunk and head: weights [64 s][64 t], decayed queries and keys [64][D], and the product of the chunk's decays.
template <typename T, typename TZ>
__global__ void __launch_bounds__(LC_THREADS) lc_prepare_kernel(LAArgs a, float* weights, float* queries, float* keys, int vec_q, int vec_z) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr bool FAST = sizeof(T) == 2;
    extern __shared__ __align__(16) float lc_smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h = blockIdx.y, D = a.D, DP = (D + 3) / 4 * 4;
    float* qt = lc_smem;                                  // [DP][64 + 4]: queries, channel by channel
    float* kt = qt + DP * LC_LD;                          // keys
    float* at = kt + DP * LC_LD;                          // decays; one behind the chunk's tokens
    float* whole = at + DP * LC_LD;                       // [4][DP]: the product of each run's decays
    int row, first, n;
    la_find_chunk(a.row_first, a.row_lens, a.B, a.first_chunk + blockIdx.x, row, first, n);
    if (n <= 0) return;
    // a lane a token: four channels are read as a run and stored to four rows, neighbouring lanes side by side
#pragma unroll 2
    for (int u = warp; u < 2 * (DP / 4); u += LC_THREADS / 32) {
        const int t = (u & 1) * 32 + lane, d = (u >> 1) * 4;
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f), k = q, z = make_float4(1.f, 1.f, 1.f, 1.f);
        if (t < n) {
            const T* p = (const T*)a.qk + (size_t)(first + t) * a.qk_ld + h * D + d;
            q = lc_load4(p + a.q_off, D - d, vec_q);
            k = lc_load4(p + a.k_off, D - d, vec_q);
            z = lc_load4((const TZ*)a.z + (size_t)(first + t) * a.z_ld + h * D + d, D - d, vec_z);
            q = make_float4(la_act<FAST>(q.x, a.act_qk) * a.q_scale, la_act<FAST>(q.y, a.act_qk) * a.q_scale, la_act<FAST>(q.z, a.act_qk) * a.q_scale, la_act<FAST>(q.w, a.act_qk) * a.q_scale);
            k = make_float4(la_act<FAST>(k.x, a.act_qk), la_act<FAST>(k.y, a.act_qk), la_act<FAST>(k.z, a.act_qk), la_act<FAST>(k.w, a.act_qk));
            z = make_float4(lc_decay(z.x, a.inv_tau), lc_decay(z.y, a.inv_tau), lc_decay(z.z, a.inv_tau), lc_decay(z.w, a.inv_tau));
        }
        float* p = qt + d * LC_LD + t;
        p[0] = q.x; p[LC_LD] = q.y; p[2 * LC_LD] = q.z; p[3 * LC_LD] = q.w;
        p = kt + d * LC_LD + t;
        p[0] = k.x; p[LC_LD] = k.y; p[2 * LC_LD] = k.z; p[3 * LC_LD] = k.w;
        p = at + d * LC_LD + t;
        p[0] = z.x; p[LC_LD] = z.y; p[2 * LC_LD] = z.z; p[3 * LC_LD] = z.w;
    }
    __syncthreads();
    float* out = weights + ((size_t)blockIdx.x * a.H + h) * ST_CHUNK * ST_CHUNK;
    // inside a run: thread (run, s, quarter of the channels) walks the decays from s on; four neighbours add up their channels
    {
        const int run = warp >> 1, s = (warp & 1) * 8 + (lane >> 2), part = lane & 3;
        float w[LC_RUN];
#pragma unroll
        for (int t = 0; t < LC_RUN; ++t) w[t] = 0.f;
        for (int d = part; d < DP; d += 4) {
            float q[LC_RUN], c[LC_RUN];
#pragma unroll
            for (int t = 0; t < LC_RUN; t += 4) {
                *reinterpret_cast<float4*>(q + t) = *reinterpret_cast<const float4*>(qt + d * LC_LD + run * LC_RUN + t);
                *reinterpret_cast<float4*>(c + t) = *reinterpret_cast<const float4*>(at + d * LC_LD + run * LC_RUN + t);
            }
            const float k = kt[d * LC_LD + run * LC_RUN + s];
            float x = 0.f;
#pragma unroll
            for (int t = 0; t < LC_RUN; ++t) {
                x = t == s ? k : t > s ? x * c[t] : 0.f;
                w[t] = fmaf(q[t], x, w[t]);
            }
        }
#pragma unroll
        for (int t = 0; t < LC_RUN; ++t) {
            w[t] += __shfl_xor_sync(0xffffffffu, w[t], 1);
            w[t] += __shfl_xor_sync(0xffffffffu, w[t], 2);
        }
        float* dst = out + (run * LC_RUN + s) * ST_CHUNK + run * LC_RUN + 4 * part;
        float4 mine = make_float4(w[0], w[1], w[2], w[3]);
#pragma unroll
        for (int p = 1; p < 4; ++p)
            if (part == p) mine = make_float4(w[4 * p], w[4 * p + 1], w[4 * p + 2], w[4 * p + 3]);
        *reinterpret_cast<float4*>(dst) = mine;
        // runs that s does not reach back to: no weight
        for (int t = part * 4; t < run * LC_RUN; t += 16) *reinterpret_cast<float4*>(out + (run * LC_RUN + s) * ST_CHUNK + t) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    // queries times what leads to them in their run, keys times what follows them there; thread (channel, run)
    for (int i = tid; i < 4 * DP; i += LC_THREADS) {
        const int d = i % DP, run = i / DP;
        const int at_run = d * LC_LD + run * LC_RUN;
        float q[LC_RUN], k[LC_RUN], c[LC_RUN];
        lc_read16(q, qt + at_run); lc_read16(k, kt + at_run); lc_read16(c, at + at_run);
        float x = 1.f;
#pragma unroll
        for (int t = 0; t < LC_RUN; ++t) { x *= c[t]; q[t] *= x; }
        whole[run * DP + d] = x;
        x = 1.f;
#pragma unroll
        for (int t = LC_RUN - 1; t >= 0; --t) { k[t] *= x; x *= c[t]; }
        lc_write16(qt + at_run, q); lc_write16(kt + at_run, k);
    }
    __syncthreads();
    // between runs j < i: 16 threads of 4 x 4 weights for each of the six pairs, two of them sharing the channels
    if (tid < 6 * 16 * 2) {
        const int half = tid & 1, u = (tid >> 1) & 15, pair = tid >> 5;
        const int i = pair < 3 ? pair + 1 : pair < 5 ? pair - 1 : 3, j = pair < 3 ? pair : pair < 5 ? pair - 3 : 0;      // (1,0) (2,1) (3,2) (2,0) (3,1) (3,0)
        const int s0 = j * LC_RUN + (u >> 2) * 4, t0 = i * LC_RUN + (u & 3) * 4;
        float4 w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) w[e] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
        for (int d = half; d < DP; d += 2) {
            const float4 q = *reinterpret_cast<const float4*>(qt + d * LC_LD + t0), k = *reinterpret_cast<const float4*>(kt + d * LC_LD + s0);
            float between = 1.f;
            if (i - j > 1) between = whole[(j + 1) * DP + d];
            if (i - j > 2) between *= whole[(j + 2) * DP + d];
            const float ks[4] = {k.x * between, k.y * between, k.z * between, k.w * between};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                w[e].x = fmaf(ks[e], q.x, w[e].x); w[e].y = fmaf(ks[e], q.y, w[e].y);
                w[e].z = fmaf(ks[e], q.z, w[e].z); w[e].w = fmaf(ks[e], q.w, w[e].w);
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            w[e].x += __shfl_xor_sync(0xffffffffu, w[e].x, 1); w[e].y += __shfl_xor_sync(0xffffffffu, w[e].y, 1);
            w[e].z += __shfl_xor_sync(0xffffffffu, w[e].z, 1); w[e].w += __shfl_xor_sync(0xffffffffu, w[e].w, 1);
            if (e >> 1 == half) *reinterpret_cast<float4*>(out + (s0 + e) * ST_CHUNK + t0) = w[e];
        }
    }
    // queries times all decays from the chunk's start, keys times all to its end, channels side by side
    float* q_out = queries + ((size_t)blockIdx.x * a.H + h) * ST_CHUNK * D;
    float* k_out = keys + ((size_t)blockIdx.x * a.H + h) * ST_CHUNK * D;
    const int r = tid / 64;                               // four groups of threads, a run each
    for (int d = tid % 64; d < D; d += 64) {
        float lead = 1.f, follow = 1.f;
        for (int x = 0; x < r; ++x) lead *= whole[x * DP + d];
        for (int x = 3; x > r; --x) follow *= whole[x * DP + d];
        float q[LC_RUN], k[LC_RUN];
        lc_read16(q, qt + d * LC_LD + r * LC_RUN); lc_read16(k, kt + d * LC_LD + r * LC_RUN);
#pragma unroll
        for (int t = 0; t < LC_RUN; ++t) {
            q_out[(size_t)(r * LC_RUN + t) * D + d] = q[t] * lead;
            k_out[(size_t)(r * LC_RUN + t) * D + d] = k[t] * follow;
        }
        if (r == 0) a.chunk_decay[((size_t)blockIdx.x * a.H + h) * D + d] = follow * whole[d];
    }
}

// Chunk, head, 128 channels x 64 columns of L (blockIdx.z: which): 16 x 8 threads of 8 x 8.
template <typename T>
__global__ void __launch_bounds__(ST_THREADS) lc_contribution_kernel(LAArgs a, const float* keys, int vec_v, int tiles_d) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr bool FAST = sizeof(T) == 2;
    __shared__ __align__(16) float ks[32 * 128], vs[32 * 64];
    const int tid = threadIdx.x, h = blockIdx.y, D = a.D, Dv = a.Dv, d0 = blockIdx.z % tiles_d * 128, c0 = blockIdx.z / tiles_d * 64;
    int row, first, n;
    la_find_chunk(a.row_first, a.row_lens, a.B, a.first_chunk + blockIdx.x, row, first, n);
    if (n <= 0) return;
    const float* k_src = keys + ((size_t)blockIdx.x * a.H + h) * ST_CHUNK * D + d0;
    const T* v_src = (const T*)a.proj + (size_t)first * a.ld + a.v_off + h * Dv + c0;
    const bool vec_k = D % 4 == 0;
    float4 rk[8], rv[4];                                   // 32 tokens of keys (a token of 128 a warp) and values
    auto fetch = [&](int s0) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int i = tid + e * ST_THREADS, s = s0 + (i >> 5), c = (i & 31) * 4;
            rk[e] = s < n ? st_load4(k_src + (size_t)s * D + c, D - d0 - c, vec_k) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int i = tid + e * ST_THREADS, s = s0 + (i >> 4), c = (i & 15) * 4;
            rv[e] = s < n ? lc_load4(v_src + (size_t)s * a.ld + c, Dv - c0 - c, vec_v) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    fetch(0);
    const int lane = tid & 31, warp = tid >> 5, ty = warp * 4 + (lane >> 3), tx = lane & 7;       // rows ty * 4 + 64 i, columns tx * 4 + 32 j
    st_pair acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
    for (int s0 = 0; s0 < n; s0 += 32) {
        if (s0) __syncthreads();
#pragma unroll
        for (int e = 0; e < 8; ++e) *reinterpret_cast<float4*>(ks + 4 * (tid + e * ST_THREADS)) = rk[e];
#pragma unroll
        for (int e = 0; e < 4; ++e)
            *reinterpret_cast<float4*>(vs + 4 * (tid + e * ST_THREADS)) =
                make_float4(la_act<FAST>(rv[e].x, a.act_v), la_act<FAST>(rv[e].y, a.act_v), la_act<FAST>(rv[e].z, a.act_v), la_act<FAST>(rv[e].w, a.act_v));
        if (s0 + 32 < n) fetch(s0 + 32);
        __syncthreads();
        const int m = min(32, n - s0);
#pragma unroll 4
        for (int s = 0; s < m; ++s) {
            float k[8];
            *reinterpret_cast<float4*>(k) = *reinterpret_cast<const float4*>(ks + s * 128 + ty * 4);
            *reinterpret_cast<float4*>(k + 4) = *reinterpret_cast<const float4*>(ks + s * 128 + ty * 4 + 64);
            const ulonglong2 v0 = *reinterpret_cast<const ulonglong2*>(vs + s * 64 + tx * 4), v1 = *reinterpret_cast<const ulonglong2*>(vs + s * 64 + tx * 4 + 32);
#pragma unroll
            for (int i = 0; i < 8; ++i) { st_fma(acc[i][0], k[i], v0.x); st_fma(acc[i][1], k[i], v0.y); st_fma(acc[i][2], k[i], v1.x); st_fma(acc[i][3], k[i], v1.y); }
        }
    }
    float* dst = a.chunk_state + ((size_t)blockIdx.x * a.H + h) * D * Dv;
    const bool vec = Dv % 4 == 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = d0 + ty * 4 + 64 * (i / 4) + i % 4;
        if (r >= D) continue;
        float* to = dst + (size_t)r * Dv + c0 + tx * 4;
        st_store4(to, Dv - c0 - tx * 4, vec, st_four(acc[i][0], acc[i][1]));
        st_store4(to + 32, Dv - c0 - tx * 4 - 32, vec, st_four(acc[i][2], acc[i][3]));
    }
}

// Chunk, head and 64 columns of its outputs.
template <typename T>
__global__ void __launch_bounds__(ST_THREADS) lc_output_kernel(LAArgs a, const float* weights, const float* queries, int vec_v) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr bool FAST = sizeof(T) == 2;
    __shared__ __align__(16) float smem[2 * ST_CHUNK * ST_CHUNK];       // two buffers of a slice of the queries and of S; then weights and values
    const int tid = threadIdx.x, h = blockIdx.y, D = a.D, Dv = a.Dv, c0 = blockIdx.z * 64;
    int row, first, n;
    la_find_chunk(a.row_first, a.row_lens, a.B, a.first_chunk + blockIdx.x, row, first, n);
    if (n <= 0) return;
    int ty, tx;
    st_place(ty, tx);
    const float* q_src = queries + ((size_t)blockIdx.x * a.H + h) * ST_CHUNK * D;
    const float* s_src = a.chunk_state + ((size_t)blockIdx.x * a.H + h) * D * Dv + c0;
    const bool vec_q = D % 4 == 0, vec_s = Dv % 4 == 0;
    STSlice rq;
    float4 rs[4];
    auto fetch = [&](int k0) {
        rq.load(q_src + k0, D, n, D - k0, vec_q);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int i = tid + e * ST_THREADS, k = k0 + (i >> 4), c = (i & 15) * 4;
            rs[e] = k < D ? st_load4(s_src + (size_t)k * Dv + c, Dv - c0 - c, vec_s) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    auto put = [&](float* to) {
        rq.store_turned(to);
#pragma unroll
        for (int e = 0; e < 4; ++e) *reinterpret_cast<float4*>(to + ST_SLICE * ST_CHUNK + 4 * (tid + e * ST_THREADS)) = rs[e];
    };
    fetch(0);
    put(smem);
    __syncthreads();
    st_pair acc[8][2];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = 0ull;
    for (int k0 = 0, b = 0; k0 < D; k0 += ST_SLICE, b ^= 1) {
        const bool more = k0 + ST_SLICE < D;
        if (more) fetch(k0 + ST_SLICE);
        const float* ct = smem + b * ST_CHUNK * ST_CHUNK;
        const float* ss = ct + ST_SLICE * ST_CHUNK;
#pragma unroll 8
        for (int k = 0; k < ST_SLICE; ++k) {
            float c[8];
            *reinterpret_cast<float4*>(c) = *reinterpret_cast<const float4*>(ct + st_turned(k, ty * 4));
            *reinterpret_cast<float4*>(c + 4) = *reinterpret_cast<const float4*>(ct + st_turned(k, ty * 4 + 32));
            const ulonglong2 s = *reinterpret_cast<const ulonglong2*>(ss + k * 64 + tx * 4);
#pragma unroll
            for (int i = 0; i < 8; ++i) { st_fma(acc[i][0], c[i], s.x); st_fma(acc[i][1], c[i], s.y); }
        }
        if (more) put(smem + (b ^ 1) * ST_CHUNK * ST_CHUNK);
        __syncthreads();
    }
    float* pt = smem;                                      // [64 s][64 t]
    float* vs = smem + ST_CHUNK * ST_CHUNK;                // [64 s][64 c]
    const float* w_src = weights + ((size_t)blockIdx.x * a.H + h) * ST_CHUNK * ST_CHUNK;
    const T* v_src = (const T*)a.proj + (size_t)first * a.ld + a.v_off + h * Dv + c0;
    float zero = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int i = tid + e * ST_THREADS, s = i >> 4, c = (i & 15) * 4;
        *reinterpret_cast<float4*>(pt + 4 * i) = *reinterpret_cast<const float4*>(w_src + 4 * i);
        const float4 v = s < n ? lc_load4(v_src + (size_t)s * a.ld + c, Dv - c0 - c, vec_v) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 u = make_float4(la_act<FAST>(v.x, a.act_v), la_act<FAST>(v.y, a.act_v), la_act<FAST>(v.z, a.act_v), la_act<FAST>(v.w, a.act_v));
        st_zero(zero, u);
        *reinterpret_cast<float4*>(vs + 4 * i) = u;
    }
    const bool guarded = __syncthreads_or(zero != 0.f);
    const int last = min(n, 32 + 16 * (tid >> 6) + 16);    // a warp's tokens reach this far: later ones have no weight
    st_weighted(acc, pt, vs, last, ty, tx, guarded);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int t = ty * 4 + 32 * (i / 4) + i % 4;
        if (t < n) st_store4(a.out + (size_t)(first + t) * ((size_t)a.H * Dv) + (size_t)h * Dv + c0 + tx * 4, Dv - c0 - tx * 4, vec_s, st_four(acc[i][0], acc[i][1]));
    }
}

long long la_channels_scratch_floats(int chunks, int H, int D) { return (long long)chunks * H * (ST_CHUNK * ST_CHUNK + 2ll * ST_CHUNK * D); }

template <typename T, typename TZ>
static int lc_prepare_and_contribute(const LAArgs& a, float* scratch, cudaStream_t s) {
    float* weights = scratch;
    float* queries = weights + (size_t)a.slab * a.H * ST_CHUNK * ST_CHUNK;
    float* keys = queries + (size_t)a.slab * a.H * ST_CHUNK * a.D;
    const int DP = (a.D + 3) / 4 * 4, size = sizeof(T);
    const int vec_q = (uintptr_t)a.qk % (4 * size) == 0 && a.qk_ld % 4 == 0 && a.q_off % 4 == 0 && a.k_off % 4 == 0 && a.D % 4 == 0;
    const int vec_z = (uintptr_t)a.z % (4 * sizeof(TZ)) == 0 && a.z_ld % 4 == 0 && a.D % 4 == 0;
    const int vec_v = (uintptr_t)a.proj % (4 * size) == 0 && a.ld % 4 == 0 && a.v_off % 4 == 0 && a.Dv % 4 == 0;
    const size_t smem = sizeof(float) * ((size_t)3 * DP * LC_LD + 4 * DP);
    PE_TRY(cudaFuncSetAttribute(lc_prepare_kernel<T, TZ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    PE_TRY(pe_launch(lc_prepare_kernel<T, TZ>, dim3(a.slab, a.H), LC_THREADS, smem, s, a, weights, queries, keys, vec_q, vec_z));
    PE_LAUNCH_CHECK();
    const int td = (a.D + 127) / 128, tv = (a.Dv + 63) / 64;
    PE_TRY(pe_launch(lc_contribution_kernel<T>, dim3(a.slab, a.H, td * tv), ST_THREADS, 0, s, a, (const float*)keys, vec_v, td));
    PE_LAUNCH_CHECK();
    return 0;
}
template <typename T>
static int lc_outputs(const LAArgs& a, float* scratch, cudaStream_t s) {
    const int vec_v = (uintptr_t)a.proj % (4 * sizeof(T)) == 0 && a.ld % 4 == 0 && a.v_off % 4 == 0 && a.Dv % 4 == 0;
    PE_TRY(pe_launch(lc_output_kernel<T>, dim3(a.slab, a.H, (a.Dv + 63) / 64), ST_THREADS, 0, s, a, (const float*)scratch,
                     (const float*)(scratch + (size_t)a.slab * a.H * ST_CHUNK * ST_CHUNK), vec_v));
    PE_LAUNCH_CHECK();
    return 0;
}

int la_channels_contributions(const LAArgs& a, bool f32, bool z_f32, float* scratch, cudaStream_t s) {
    if (a.D > 256 || a.H > 65535) return PE_ERR_UNSUPPORTED;
    if (f32) return lc_prepare_and_contribute<float, float>(a, scratch, s);
    return z_f32 ? lc_prepare_and_contribute<bf16, float>(a, scratch, s) : lc_prepare_and_contribute<bf16, bf16>(a, scratch, s);
}
int la_channels_outputs(const LAArgs& a, bool f32, float* scratch, cudaStream_t s) { return f32 ? lc_outputs<float>(a, scratch, s) : lc_outputs<bf16>(a, scratch, s); }
