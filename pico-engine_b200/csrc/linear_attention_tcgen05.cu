// Linear attention of prompts as products of tiles on the 5th-generation tensor cores (linear_attention_tiles.cu and
// linear_attention_channels.cu have the same with multiply-adds, and the sums; chunk_mma.cuh how float32 numbers are
// multiplied).  bfloat16 rows, heads of 128 x 128, or an even number of heads of 64 x 64.
//
// A first kernel a kind of decay works out what does not depend on the state and leaves it as bfloat16 parts: the chunk's queries (times their decays
// from the chunk's start, where those are a channel's), its keys times their decays to the chunk's end, and its weights q_t . A(s, t) k_s.
// A unit is a chunk and 128 value columns, one head's or two heads', which stand on the accumulator's lanes:
//   contributions  L^T [v][d] = v^T K          K: the chunk's tokens
//   outputs        o^T [v][t] = S^T Q^T (times the decay to t, where it is a head's) + v^T W^T      K: the state's rows, 64 at a time; then the tokens
// Values that no activation is applied to are bfloat16 numbers as they are: one part, half of the products.  Of two heads the products hold what either's
// columns give with the other's rows too, which is left.
//
// A state in scratch is [half of the unit's columns][D / 8][64 v][8 d], so that a thread writes and reads runs of 32 bytes and a warp whole lines.
//
// Contributions and outputs only copy, multiply and store (outputs cut the state): what bounds them is the parts' way from L2.  Measured on a B200, 2,048
// tokens, 16 heads of 128 x 128, us: a decay a head and silu on queries, keys and values 121 as multiply-adds, 93 here (operands 36,
// contributions 15, carry 10, outputs 29); a decay a channel 174 and 104 (54, 12, 10, 23).  14 heads of 64: 57 and 45, 76 and 49; 200 tokens of those 34 and
// 26, 43 and 29; three prompts of 300, 500 and 33, 16 heads 67 and 49, 91 and 55: steps that go in chunks at all (LinearAttention.chunks_pay) are sooner here.
// Errors against 64 bits, of the outputs' norm: 2.1e-7 as multiply-adds and 6.3e-8 here, with a decay a channel 2.0e-7 and 1.6e-7 (its weights are the same
// sums); of the states 1.0e-7 and 6.1e-8, 1.44e-7 and 1.28e-7.
#include "linear_attention.cuh"
#include "chunk_mma.cuh"

#define LM_THREADS 256
#define LM_SMEM (12 * CM_PLANE + 1024)                    // parts of Q (or of W) and of S (or the values), both halves

// A unit's parts in scratch: queries and keys, [part][two][64 tokens][64 channels] each (two: the channels' halves, or the heads), and weights
// [part][heads][64 t][64 s]; and values behind their activation, if there is one, [part][half][64 s][64 columns].
template <bool TWO> struct LMUnit {
    static constexpr int ND = TWO ? 64 : 128;             // rows of a head's state
    static constexpr int QUERIES = 0, KEYS = 6 * CM_PLANE, WEIGHTS = 12 * CM_PLANE, W_HEADS = TWO ? 2 : 1, VALUES = (12 + 3 * W_HEADS) * CM_PLANE;
    static __host__ __device__ __forceinline__ constexpr size_t bytes(bool values) { return VALUES + (values ? 6 * CM_PLANE : 0); }
    // of a head h
    static __device__ __forceinline__ unsigned char* of(const LAArgs& a, int c, int h) { return a.chunk_planes + ((size_t)c * (TWO ? a.H / 2 : a.H) + (TWO ? h / 2 : h)) * bytes(a.act_v != 0); }
};

// Tiles of a chunk's and head's word: 0 queries, 1 keys (with one decay a head), 2 weights, 3 values; of numbers alone (cm_watch_numbers) 4 keys times their decays, 5 values.
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
template <bool NUMBERS = false>
__device__ __forceinline__ void lm_put(unsigned char* to, int stride, const float (&v)[8], unsigned& most) {
    cm_put<NUMBERS>(to, stride, make_float4(v[0], v[1], v[2], v[3]), make_float4(v[4], v[5], v[6], v[7]), most);
}
// The same with zeros for what parts do not hold; first: the first row that has such a number.
__device__ __noinline__ void lm_mend(unsigned char* to, int stride, float4 a, float4 b, int row, unsigned* first) {
    atomicMin(first, (unsigned)row);
    const auto fit = [](float v) { return fabsf(v) < 0x1p59f ? v : 0.f; };
    unsigned most = 0;
    cm_put(to, stride, make_float4(fit(a.x), fit(a.y), fit(a.z), fit(a.w)), make_float4(fit(b.x), fit(b.y), fit(b.z), fit(b.w)), most);
}
__device__ __forceinline__ void lm_put_mended(unsigned char* to, int stride, const float (&v)[8], unsigned& most, int row, unsigned* first) {
    unsigned mine = 0;
    lm_put(to, stride, v, mine);
    cm_watch(most, mine);
    if (cm_odd(mine)) lm_mend(to, stride, make_float4(v[0], v[1], v[2], v[3]), make_float4(v[4], v[5], v[6], v[7]), row, first);
}
// Eight values of a token: parts behind their activation; without one they are only looked at.
__device__ __forceinline__ void lm_values(const LAArgs& a, unsigned char* to, const bf16* from, bool there, int row, unsigned* first_odd, unsigned& most, unsigned& numbers) {
    unsigned mine = 0;
    if (a.act_v) {
        float v[8];
        lm_eight(v, from, there, true);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = la_act<true>(v[i], a.act_v);
        cm_scale(v, CM_UP);
        lm_put(to, 2 * CM_PLANE, v, mine);
    } else if (there) {
        const uint4 r = *reinterpret_cast<const uint4*>(from);
        cm_watch(mine, r.x); cm_watch(mine, r.y); cm_watch(mine, r.z); cm_watch(mine, r.w);
    }
    cm_watch(most, mine);
    if (!cm_odd(mine, a.act_v ? CM_MOST : CM_MOST_PLAIN)) return;
    atomicMin(first_odd, (unsigned)row);
    for (int i = 0; i < 8; ++i) {                          // (seldom: which of them are numbers)
        const float v = la_act<true>(to_f(from[i]), a.act_v);
        if (fabsf(v) >= 0x1p34f) numbers = CM_MOST;        // (2^34: what is rounded to 2^35 counts)
    }
}

// a = sigmoid(z)^(inv_tau), through the logarithm: -softplus(-z) * inv_tau (as the walk of linear_attention.cu has it)
__device__ __forceinline__ float lm_decay(float z, float inv_tau) {
    const float u = -z;
    return expf(-(fmaxf(u, 0.f) + log1pf(expf(-fabsf(u)))) * inv_tau);
}

// [2][64 t][64] or [64 t][128] numbers of rows, all asked for before any is stored: dst in shared memory.
template <typename T, int ND>
__device__ __forceinline__ void lm_fill(float* dst, const T* src, int ld, int n) {
    float v[2][8];
#pragma unroll 1
    for (int r = 0; r < 4; r += 2) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int i = ((r + e) * LM_THREADS + threadIdx.x) * 8;
            lm_eight(v[e], src + (size_t)min(i / ND % 64, n - 1) * ld + i / (64 * ND) * ND + i % ND, true, ((uintptr_t)src | ld * sizeof(T)) % 16 == 0);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            float* to = dst + ((r + e) * LM_THREADS + threadIdx.x) * 8;
            *reinterpret_cast<float4*>(to) = make_float4(v[e][0], v[e][1], v[e][2], v[e][3]);
            *reinterpret_cast<float4*>(to + 4) = make_float4(v[e][4], v[e][5], v[e][6], v[e][7]);
        }
    }
}
// What parts are not made of: a unit's chunk token after token with multiply-adds, from its incoming state (none: zeros), all threads of a block.  Outputs from
// token `exact` on; the state behind the chunk to `to_state`, if that is asked for.  Queries, keys and decays are worked out once, into the block's shared memory
// (which nobody else uses then).  A state with infinities or huge numbers sends every unit behind it here, a token that is no number those of its chunk.  2,048 tokens with one
// value, one head's keys, all of a token, every token that is none, us:
//   16 heads of 128, a decay a head     144 / 145 / 148 / 164 (96 without; multiply-add tiles 125; entry by entry from memory 4,115 to 8,013)
//   a decay a channel                   155 / 152 / 155 / 171 (110; 180; 5,276 to 9,552)
//   14 heads of 64                      82 / 83 / 84 / 91 (49; 53; 2,000) and 88 / 84 / 89 / 90 (53; 79; 2,600)
// Most of it is one walk's latency, 50 us.
template <bool TWO>
__device__ __noinline__ void lm_walk(const LAArgs& a, int first, int n, int h0, const float* state, int exact, float* to_state) {
    extern __shared__ unsigned char lm_raw[];
    float* smem = reinterpret_cast<float*>(lm_raw + (-at_smem(lm_raw) & 1023u));
    constexpr int ND = LMUnit<TWO>::ND;
    using Walk = CMWalk<ND>;
    const int tid = threadIdx.x, ld_out = a.H * a.Dv, ld = a.ld, act_qk = a.act_qk, act_v = a.act_v, hh = TWO ? Walk::column() >> 6 : 0;
    float *qs = smem, *ks = smem + 64 * 128, *as = smem + 2 * 64 * 128;                     // [head][64 t][ND]
    const bool writes = !(tid & 1);
    float* out = a.out + (size_t)first * ld_out + h0 * a.Dv + Walk::written();
    Walk walk;
    if (__syncthreads_and(walk.begin(state))) {            // no state that is a number: no output is one
        if (writes)
            for (int t = exact; t < n; ++t) out[(size_t)t * ld_out] = __int_as_float(0x7fffffff);
        return;
    }
    // The numbers as they are, then each through its activation.  (Loops of few instructions: what runs here has not run before and comes from L2.)
    const bool pc = a.z != nullptr;
    const float q_scale = a.q_scale, inv_tau = a.inv_tau;    // (loops that store read nothing of the arguments, which they would read again each time)
    const size_t row = (size_t)first * a.qk_ld + h0 * ND;
    if (a.qk_f32) {
        lm_fill<float, ND>(ks, (const float*)a.qk + row + a.k_off, a.qk_ld, n);
        lm_fill<float, ND>(qs, (const float*)a.qk + row + a.q_off, a.qk_ld, n);
    } else {
        lm_fill<bf16, ND>(ks, (const bf16*)a.qk + row + a.k_off, a.qk_ld, n);
        lm_fill<bf16, ND>(qs, (const bf16*)a.qk + row + a.q_off, a.qk_ld, n);
    }
    if (pc && a.z_f32) lm_fill<float, ND>(as, (const float*)a.z + (size_t)first * a.z_ld + h0 * ND, a.z_ld, n);
    if (pc && !a.z_f32) lm_fill<bf16, ND>(as, (const bf16*)a.z + (size_t)first * a.z_ld + h0 * ND, a.z_ld, n);
    __syncthreads();
#pragma unroll 1
    for (int i = tid; i < 64 * 128; i += LM_THREADS) {
        ks[i] = la_act<true>(ks[i], act_qk);
        qs[i] = la_act<true>(qs[i], act_qk) * q_scale;
        if (pc) as[i] = lm_decay(as[i], inv_tau);
    }
    const float fixed = pc ? 0.f : a.head_decay[h0 + hh];
    const bf16* values = (const bf16*)a.proj + (size_t)first * a.ld + a.v_off + h0 * a.Dv + Walk::column();
    auto ask = [&](int t) { return *reinterpret_cast<const uint2*>(values + (size_t)min(t, n - 1) * ld); };
    uint2 next = ask(0), later = ask(1);
    __syncthreads();
#pragma unroll 1
    for (int t = 0; t < n; ++t) {
        const uint2 now = next;
        next = later;
        later = ask(t + 2);
        const int at = (hh * 64 + t) * ND;
        const float v[4] = {la_act<true>(__uint_as_float(now.x << 16), act_v), la_act<true>(__uint_as_float(now.x & 0xffff0000u), act_v),
                            la_act<true>(__uint_as_float(now.y << 16), act_v), la_act<true>(__uint_as_float(now.y & 0xffff0000u), act_v)};
        walk.step(ks + at, pc ? as + at : nullptr, fixed, v);
        if (t < exact) continue;
        const float o = walk.output(qs + at);
        if (writes) out[(size_t)t * ld_out] = o;
    }
    if (to_state) walk.end(to_state);
    __syncthreads();                                       // (the shared memory has been read)
}
// With one decay a head, a chunk and head: queries and keys through their activation, k_s a^(n-1-s), and weights q_t . k_s a^(t-s), from scores by mma.sync.
template <typename TQ, bool TWO>
__global__ void __launch_bounds__(512, 2) lm_prepare_kernel(LAArgs a, int vec_q) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) unsigned char lm_mem[];
    unsigned char *qs = lm_mem, *ks = lm_mem + 3 * CM_PLANE;          // 64 channels at a time; in the end the weights
    __shared__ float pw[LA_CHUNK + 1];
    __shared__ unsigned seen, from;
    using Unit = LMUnit<TWO>;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, row = tid >> 3, group = tid & 7, h = blockIdx.y, D = a.D;
    if (tid == 0) { seen = 0; from = LA_CHUNK; }
    pdl_wait();
    int seq, first, n;
    la_find_chunk(a.row_first, a.row_lens, a.B, a.first_chunk + blockIdx.x, seq, first, n);
    if (tid == 0 && h == 0) a.chunk_rows[blockIdx.x] = make_int2(first, n);
    if (n <= 0) return;
    la_powers(pw, a.head_decay[h]);
    unsigned char* unit = Unit::of(a, blockIdx.x, h);
    const int t0 = (warp & 3) * 16, s0 = warp < 8 ? (warp >> 2) * 32 : LA_CHUNK;
    const bool there = row < n;
    const TQ* src = (const TQ*)a.qk + (size_t)(first + (there ? row : 0)) * a.qk_ld + h * D + 8 * group;
    CMScores acc;
    acc.clear();
    unsigned most_w = 0, most_v = 0, numbers = 0;
    __syncthreads();
    const float follow = there ? pw[n - 1 - row] : 0.f;
    for (int j = 0; j < D / 64; ++j) {
        float q[8], k[8];
        unsigned most[3] = {0, 0, 0};
        lm_eight(q, src + a.q_off + 64 * j, there, vec_q);
        lm_eight(k, src + a.k_off + 64 * j, there, vec_q);
#pragma unroll
        for (int i = 0; i < 8; ++i) { q[i] = la_act<true>(q[i], a.act_qk) * a.q_scale; k[i] = la_act<true>(k[i], a.act_qk); }
        cm_scale(q, CM_UP);
        cm_scale(k, CM_UP);
        if (j) __syncthreads();
        lm_put_mended(qs + cm_at(row, group), CM_PLANE, q, most[0], row, &from);
        lm_put_mended(ks + cm_at(row, group), CM_PLANE, k, most[1], row, &from);
        const int half = (TWO ? h & 1 : j) * CM_PLANE;
#pragma unroll
        for (int p = 0; p < CM_PARTS; ++p)                 // (the thread's own run, a line by eight neighbours)
            *reinterpret_cast<uint4*>(unit + Unit::QUERIES + p * 2 * CM_PLANE + half + cm_at(row, group)) = *reinterpret_cast<const uint4*>(qs + p * CM_PLANE + cm_at(row, group));
#pragma unroll
        for (int i = 0; i < 8; ++i) k[i] *= follow;
        lm_put<true>(unit + Unit::KEYS + half + cm_at(row, group), 2 * CM_PLANE, k, most[2]);
        cm_report(&seen, cm_seen(most[0], 0) | cm_seen(most[1], 1) | cm_seen(most[2], 4));
        __syncthreads();
        if (s0 <= t0) acc.add(at_smem(qs), at_smem(ks), CM_PLANE, t0, s0);
        lm_values(a, unit + Unit::VALUES + half + cm_at(row, group), (const bf16*)a.proj + (size_t)(first + row) * a.ld + a.v_off + h * a.Dv + 64 * j + 8 * group, there, row, &from, most_v, numbers);
    }
    __syncthreads();
    if (warp < 8) {                                        // (later keys have no weight)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 4; e += 2) {
                const int t = t0 + lane / 4 + 4 * e, s = s0 + 8 * j + lane % 4 * 2;
                unsigned hi, mid, lo;
                const float2 scores = cm_scaled(acc.get(j, e), acc.get(j, e + 1), CM_DOWN);      // (times CM_UP once)
                cm_cut(s <= t ? scores.x * pw[t - s] : 0.f, s + 1 <= t ? scores.y * pw[t - s - 1] : 0.f, hi, mid, lo);
                cm_watch(most_w, hi);
                unsigned char* to = qs + cm_at(t, s >> 3) + (s & 7) * 2;
                *reinterpret_cast<unsigned*>(to) = hi;
                *reinterpret_cast<unsigned*>(to + CM_PLANE) = mid;
                *reinterpret_cast<unsigned*>(to + 2 * CM_PLANE) = lo;
            }
    }
    cm_report(&seen, cm_seen(most_w, 2) | cm_seen(most_v, 3, a.act_v ? CM_MOST : CM_MOST_PLAIN) | cm_seen(numbers, 5));
    __syncthreads();
    if (seen >> 2 & 1u) {
        cm_mend(qs, CM_PLANE, CM_PARTS, &from);
        __syncthreads();
    }
#pragma unroll
    for (int p = 0; p < CM_PARTS; ++p)
        *reinterpret_cast<uint4*>(unit + Unit::WEIGHTS + (p * Unit::W_HEADS + (TWO ? h & 1 : 0)) * CM_PLANE + tid * 16) = *reinterpret_cast<const uint4*>(qs + p * CM_PLANE + tid * 16);
    if (tid == 0) a.chunk_seen[(size_t)blockIdx.x * a.H + h] = seen | from << 16;
    if (tid < D) a.chunk_decay[((size_t)blockIdx.x * a.H + h) * D + tid] = pw[n];
}

// With one decay a channel, a chunk and head: queries times all decays from the chunk's start, keys times all to its end, and weights q_t . A(s, t) k_s.
// Every product of decays is formed forwards, from factors of at most one (linear_attention_channels.cu): a chunk is four runs of 16; inside a run the
// decays are walked, between two runs they are what follows s in its run, the whole runs between, and what leads to t in its own.
// Numbers lie channel by channel, [D][64], rows of 68 with four more every eight channels: a token's run of eight channels and a channel's run of tokens
// both meet every bank once.  What bounds it: issue slots, half of them the logarithms and exponentials of the decays and what surrounds the walks.  2,048 tokens, 16
// heads of 128: 54 us; 79 with rows of 68 read a token a lane, walks over whole runs for every key, and parts turned through shared memory.
#define LMC_RUN 16
__device__ __forceinline__ int lmc_row(int d) { return d * 68 + (d >> 3) * 4; }
__host__ __device__ constexpr int lmc_floats(int D) { return D * 68 + D / 8 * 4; }
__device__ __forceinline__ void lmc_read16(float (&v)[LMC_RUN], const float* p) {
#pragma unroll
    for (int t = 0; t < LMC_RUN; t += 4) *reinterpret_cast<float4*>(v + t) = *reinterpret_cast<const float4*>(p + t);
}
// Sums over 16 neighbouring lanes of N (16 or 8) numbers each: lane l is left with number l % N.
template <int N>
__device__ __forceinline__ float lmc_sums(float (&w)[N], int lane) {
#pragma unroll
    for (int o = N / 2; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < o; ++i) {
            const bool upper = lane & o;
            const float keep = upper ? w[i + o] : w[i], give = upper ? w[i] : w[i + o];
            w[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    if (N == 8) w[0] += __shfl_xor_sync(0xffffffffu, w[0], 8);
    return w[0];
}
template <typename TZ, bool TWO>
__global__ void __launch_bounds__(512, 2) lm_channels_kernel(LAArgs a, int vec_q, int vec_z) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) float lmc_smem[];
    __shared__ unsigned seen, from;
    using Unit = LMUnit<TWO>;
    constexpr int D = Unit::ND;
    const int tid = threadIdx.x, lane = tid & 31, row = tid >> 3, group = tid & 7, h = blockIdx.y;
    float *qt = lmc_smem, *kt = qt + lmc_floats(D), *at = kt + lmc_floats(D);
    float *whole = at + lmc_floats(D), *lead = whole + 4 * D, *follow = lead + 4 * D;                       // [4][D]: a run's decays; what leads to it; what follows it
    if (tid == 0) { seen = 0; from = LA_CHUNK; }
    pdl_wait();
    int seq, first, n;
    la_find_chunk(a.row_first, a.row_lens, a.B, a.first_chunk + blockIdx.x, seq, first, n);
    if (tid == 0 && h == 0) a.chunk_rows[blockIdx.x] = make_int2(first, n);
    if (n <= 0) return;
    __syncthreads();                                       // (the words stand before a value that is no number lowers one)
    const bool there = row < n;
    const size_t token = first + (there ? row : 0);
    unsigned char* unit = Unit::of(a, blockIdx.x, h);
    unsigned most_q = 0, most_k = 0, most_w = 0, most_v = 0, numbers = 0;
#pragma unroll 1
    for (int j = 0; j < D / 64; ++j) {
        const int d = 64 * j + 8 * group;
        float q[8], k[8], z[8];
        lm_eight(q, (const bf16*)a.qk + token * a.qk_ld + a.q_off + h * D + d, there, vec_q);
        lm_eight(k, (const bf16*)a.qk + token * a.qk_ld + a.k_off + h * D + d, there, vec_q);
        lm_eight(z, (const TZ*)a.z + token * a.z_ld + h * D + d, there, vec_z);
        lm_values(a, unit + Unit::VALUES + (TWO ? h & 1 : j) * CM_PLANE + cm_at(row, group), (const bf16*)a.proj + token * a.ld + a.v_off + h * a.Dv + d, there, row, &from, most_v, numbers);
        float* to = qt + lmc_row(d) + row;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            to[i * 68] = la_act<true>(q[i], a.act_qk) * a.q_scale;
            to[i * 68 + lmc_floats(D)] = la_act<true>(k[i], a.act_qk);
            to[i * 68 + 2 * lmc_floats(D)] = there ? lm_decay(z[i], a.inv_tau) : 1.f;
        }
    }
    __syncthreads();
    float* weights = a.chunk_state + ((size_t)blockIdx.x * a.H + h) * D * a.Dv;      // [64 s][64 t], until the contribution takes the place
    // inside a run: 16 neighbours share the channels of keys s and s + 8 of a run
    {
        const int part = tid & 15, run = tid >> 7, s = (tid >> 4) & 7;
        float w[16], late[8];                              // weights of s over the run, of s + 8 over its second half
#pragma unroll
        for (int t = 0; t < 16; ++t) w[t] = 0.f;
#pragma unroll
        for (int t = 0; t < 8; ++t) late[t] = 0.f;
#pragma unroll 1
        for (int d = part; d < D; d += 16) {
            float q[LMC_RUN], c[LMC_RUN];
            const float* p = qt + lmc_row(d) + run * LMC_RUN;
            lmc_read16(q, p);
            lmc_read16(c, p + 2 * lmc_floats(D));
            const float k = p[lmc_floats(D) + s], k_late = p[lmc_floats(D) + 8 + s];
            float x = 0.f, y = 0.f;                        // (tokens in front of s: whatever comes of them is not read)
#pragma unroll
            for (int t = 0; t < 8; ++t) { x = t == s ? k : x * c[t]; w[t] = fmaf(q[t], x, w[t]); }
#pragma unroll
            for (int t = 8; t < 16; ++t) {
                x *= c[t]; w[t] = fmaf(q[t], x, w[t]);
                y = t == s + 8 ? k_late : y * c[t]; late[t - 8] = fmaf(q[t], y, late[t - 8]);
            }
        }
        float* to = weights + (run * LMC_RUN + s) * LA_CHUNK + run * LMC_RUN;
        to[part] = lmc_sums(w, lane);
        const float v = lmc_sums(late, lane);
        if (part < 8) to[8 * LA_CHUNK + 8 + part] = v;
    }
    __syncthreads();
    // queries times what leads to them in their run, keys times what follows them there; thread (channel, run)
    if (tid < 4 * D) {
        const int d = tid % D, run = tid / D;
        float q[LMC_RUN], k[LMC_RUN], c[LMC_RUN];
        float* p = qt + lmc_row(d) + run * LMC_RUN;
        lmc_read16(q, p); lmc_read16(k, p + lmc_floats(D)); lmc_read16(c, p + 2 * lmc_floats(D));
        float x = 1.f;
#pragma unroll
        for (int t = 0; t < LMC_RUN; ++t) { x *= c[t]; q[t] *= x; }
        whole[run * D + d] = x;
        x = 1.f;
#pragma unroll
        for (int t = LMC_RUN - 1; t >= 0; --t) { k[t] *= x; x *= c[t]; }
#pragma unroll
        for (int t = 0; t < LMC_RUN; t += 4) {
            *reinterpret_cast<float4*>(p + t) = make_float4(q[t], q[t + 1], q[t + 2], q[t + 3]);
            *reinterpret_cast<float4*>(p + lmc_floats(D) + t) = make_float4(k[t], k[t + 1], k[t + 2], k[t + 3]);
        }
    }
    __syncthreads();
    if (tid < D) {
        const int d = tid;
        const float w[4] = {whole[d], whole[D + d], whole[2 * D + d], whole[3 * D + d]};
        lead[d] = 1.f; lead[D + d] = w[0]; lead[2 * D + d] = w[0] * w[1]; lead[3 * D + d] = (w[0] * w[1]) * w[2];
        follow[3 * D + d] = 1.f; follow[2 * D + d] = w[3]; follow[D + d] = w[3] * w[2]; follow[d] = (w[3] * w[2]) * w[1];
        a.chunk_decay[((size_t)blockIdx.x * a.H + h) * D + d] = ((w[3] * w[2]) * w[1]) * w[0];
    }
    // between runs j < i: 16 threads of 4 x 4 weights for each of the six pairs, four of them sharing the channels
    if (tid < 6 * 16 * 4) {
        const int quarter = tid & 3, u = (tid >> 2) & 15, pair = tid >> 6;
        const int i = pair < 3 ? pair + 1 : pair < 5 ? pair - 1 : 3, j = pair < 3 ? pair : pair < 5 ? pair - 3 : 0;      // (1,0) (2,1) (3,2) (2,0) (3,1) (3,0)
        const int s0 = j * LMC_RUN + (u >> 2) * 4, t0 = i * LMC_RUN + (u & 3) * 4;
        float4 w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) w[e] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
        for (int d = quarter; d < D; d += 4) {
            const float4 q = *reinterpret_cast<const float4*>(qt + lmc_row(d) + t0), k = *reinterpret_cast<const float4*>(kt + lmc_row(d) + s0);
            float between = 1.f;
            if (i - j > 1) between = whole[(j + 1) * D + d];
            if (i - j > 2) between *= whole[(j + 2) * D + d];
            const float ks[4] = {k.x * between, k.y * between, k.z * between, k.w * between};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                w[e].x = fmaf(ks[e], q.x, w[e].x); w[e].y = fmaf(ks[e], q.y, w[e].y);
                w[e].z = fmaf(ks[e], q.z, w[e].z); w[e].w = fmaf(ks[e], q.w, w[e].w);
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                w[e].x += __shfl_xor_sync(0xffffffffu, w[e].x, o); w[e].y += __shfl_xor_sync(0xffffffffu, w[e].y, o);
                w[e].z += __shfl_xor_sync(0xffffffffu, w[e].z, o); w[e].w += __shfl_xor_sync(0xffffffffu, w[e].w, o);
            }
            if (e == quarter) *reinterpret_cast<float4*>(weights + (s0 + e) * LA_CHUNK + t0) = w[e];
        }
    }
    __syncthreads();                                       // (the weights are written, what leads and follows too)
    float weight[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) weight[i] = 8 * group + i <= row ? weights[(8 * group + i) * LA_CHUNK + row] : 0.f;
#pragma unroll 1
    for (int j = 0; j < D / 64; ++j) {
        const int d = 64 * j + 8 * group, place = (TWO ? h & 1 : j) * CM_PLANE + cm_at(row, group), run = row >> 4;
        const float* p = qt + lmc_row(d) + row;
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = p[i * 68] * lead[run * D + d + i];
        cm_scale(v, CM_UP);
        lm_put_mended(unit + Unit::QUERIES + place, 2 * CM_PLANE, v, most_q, row, &from);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = p[i * 68 + lmc_floats(D)] * follow[run * D + d + i];
        cm_scale(v, CM_UP);
        lm_put<true>(unit + Unit::KEYS + place, 2 * CM_PLANE, v, most_k);
    }
    cm_scale(weight, CM_UP);
    lm_put_mended(unit + Unit::WEIGHTS + (TWO ? h & 1 : 0) * CM_PLANE + cm_at(row, group), Unit::W_HEADS * CM_PLANE, weight, most_w, row, &from);
    cm_report(&seen, cm_seen(most_q, 0) | cm_seen(most_k, 4) | cm_seen(most_w, 2) | cm_seen(most_v, 3, a.act_v ? CM_MOST : CM_MOST_PLAIN) | cm_seen(numbers, 5));
    __syncthreads();
    if (tid == 0) a.chunk_seen[(size_t)blockIdx.x * a.H + h] = seen | from << 16;
}

// What stands in the words of a unit's heads (bits from 16 on: the first token that parts do not hold).
template <bool TWO>
__device__ __forceinline__ unsigned lm_known(const LAArgs& a, int c, int h0) {
    const unsigned x = a.chunk_seen[(size_t)c * a.H + h0];
    if (!TWO) return x;
    const unsigned y = a.chunk_seen[(size_t)c * a.H + h0 + 1];
    return ((x | y) & 0xffffu) | (min(x >> 16, y >> 16) << 16);
}
// The values of a unit, [half][64 tokens][64 columns], zeros behind its tokens.
__device__ __forceinline__ void lm_bring_values(unsigned char* dst, const LAArgs& a, int first, int n, int col0) {
    const bf16* src = (const bf16*)a.proj + (size_t)first * a.ld + a.v_off + col0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int u = threadIdx.x + e * LM_THREADS, s = u >> 4, g = u & 15;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(at_smem(dst + (g >> 3) * CM_PLANE + cm_at(s, g & 7))), "l"(src + (size_t)min(s, n - 1) * a.ld + 8 * g), "r"(s < n ? 16 : 0) : "memory");
    }
}

// Chunks of a unit's heads, contributions.  Nothing is cut here: the parts and values of the next unit come while this one's sums leave.
template <bool TWO, int VALUE_PARTS>
__global__ void __launch_bounds__(LM_THREADS, TWO || VALUE_PARTS == 3 ? 3 : 2) lm_contribution_kernel(LAArgs a, int units) {
    extern __shared__ unsigned char lm_raw[];
    __shared__ __align__(8) unsigned long long bar;
    __shared__ unsigned tmem_s;
    using Unit = LMUnit<TWO>;
    constexpr int ND = Unit::ND;
    unsigned char* ks = lm_raw + (-at_smem(lm_raw) & 1023u);          // [part][two][64 s][64 d]
    unsigned char* vs = ks + 6 * CM_PLANE;                            // [part][half][64 s][64 v]
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), per = TWO ? a.H / 2 : a.H;
    const int q = warp & 3, hh = q >> 1, p = (q & 1) * 32 + lane;
    const unsigned tmem = cm_begin(&tmem_s, &bar);
    const unsigned elected = warp == 0 ? pe_elect() : 0u;
    pdl_wait();
    unsigned phase = 0;
    int2 place = a.chunk_rows[blockIdx.x / per];
    unsigned known = 0;
    bool odd = false;
    auto bring = [&](int unit) {
        const int c = unit / per, h0 = unit % per * (TWO ? 2 : 1);
        cm_bring(ks, Unit::of(a, c, h0) + Unit::KEYS, 6 * CM_PLANE);
        if constexpr (VALUE_PARTS == 1) lm_bring_values(vs, a, place.x, place.y, h0 * a.Dv);
        else cm_bring(vs, Unit::of(a, c, h0) + Unit::VALUES, 6 * CM_PLANE);
        known = lm_known<TWO>(a, c, h0);
    };
    if (place.y > 0) bring(blockIdx.x);
    for (int unit = blockIdx.x; unit < units && place.y > 0; unit += gridDim.x) {
        const int next = unit + gridDim.x;
        if (next < units) place = a.chunk_rows[next / per];
        cm_landed();
        cm_ready();
        const bool parts = !(known & (1u << 4 | 1u << 5));            // (every thread has read the same words)
        odd = odd || !parts;
        if (parts) {
            if (warp == 0) {
                if constexpr (VALUE_PARTS == 1) cm_products_one(elected, tmem, tmem + 128, at_desc(at_smem(vs), CM_PLANE, 1024), 128u, cm_across(at_smem(ks), 2 * CM_PLANE, CM_PLANE), cm_idesc(128, true, true));
                else cm_products(elected, tmem, tmem + 128, cm_across(at_smem(vs), 2 * CM_PLANE, CM_PLANE), cm_across(at_smem(ks), 2 * CM_PLANE, CM_PLANE), cm_idesc(128, true, true));
                if (elected) at_commit(at_smem(&bar));
                __syncwarp();
            }
            cm_done(&bar, phase, a.status);
        }
        if (next < units && place.y > 0) bring(next);
        float* state = a.chunk_state + (size_t)unit * 128 * ND;
        if (parts) {
            const int column0 = TWO ? hh * 64 + (warp >> 2) * 32 : (warp >> 2) * 64;
#pragma unroll
            for (int j = 0; j < (TWO ? 2 : 4); ++j) {
                const int column = column0 + 16 * j;
                const unsigned at = tmem + ((unsigned)(q * 32) << 16) + column;
                float acc[16];
                cm_read(acc, at + 128);
                cm_take(acc, at);
                cm_scale(acc, VALUE_PARTS == 1 ? CM_DOWN : CM_DOWN * CM_DOWN);
                float* to = state + (size_t)hh * ND * 64 + ((size_t)((TWO ? column & 63 : column) / 8) * 64 + p) * 8;
                cm_store8(to, *reinterpret_cast<const float (*)[8]>(acc));
                cm_store8(to + 512, *reinterpret_cast<const float (*)[8]>(acc + 8));
            }
        }
    }
    cm_end(tmem);
    if (!odd) return;                                      // (the walks behind the loop: inside they cost its registers)
    __shared__ LAArgs args;
    if (tid == 0) args = a;
    __syncthreads();
#pragma unroll 1
    for (int unit = blockIdx.x; unit < units; unit += gridDim.x) {
        const int c = unit / per, h0 = unit % per * (TWO ? 2 : 1);
        const int2 at = a.chunk_rows[c];
        if (at.y <= 0) break;
        if (lm_known<TWO>(a, c, h0) & (1u << 4 | 1u << 5)) lm_walk<TWO>(args, at.x, at.y, h0, nullptr, at.y, a.chunk_state + (size_t)unit * 128 * ND);
    }
}

// A block eight columns of a head's state, 2 D threads: a thread four rows of a column walks the sequence's chunks in order, leaves every chunk its
// incoming state where its own contribution was, and stores the sequence's new state.  Reads in whole runs of eight chunks and what is left apart
// (one loop whose reads ask whether there is a chunk took twice as long in state_space_tcgen05.cu's pass of the same kind).
__global__ void __launch_bounds__(256) lm_carry_kernel(LAArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    const int b = blockIdx.y, tid = threadIdx.x, D = a.D, eights = a.Dv / 8, h = blockIdx.x / eights, v = blockIdx.x % eights * 8 + tid / 2 % 8, d0 = tid / 16 * 8 + tid % 2 * 4;
    int base = 0;
    for (int i = 0; i < b; ++i) base += (a.row_lens[i] + LA_CHUNK - 1) / LA_CHUNK;
    int nc = (a.row_lens[b] + LA_CHUNK - 1) / LA_CHUNK;
    const int end = min(base + nc - a.first_chunk, a.slab);           // the sequence's chunks of this slab, by their places in it
    base = max(base - a.first_chunk, 0);
    nc = end - base;
    if (nc <= 0) return;
    const size_t per = (size_t)a.H * D * a.Dv / 4;
    float4* chunks = reinterpret_cast<float4*>(a.chunk_state + ((size_t)h * a.Dv + v / 64 * 64) * D + ((size_t)(d0 / 8) * 64 + v % 64) * 8 + d0 % 8) + (size_t)base * per;
    const float4* decay = reinterpret_cast<const float4*>(a.chunk_decay + ((size_t)base * a.H + h) * D + d0);
    const size_t per_decay = (size_t)a.H * D / 4;
    float4 own[8], dec[8];
    auto ask = [&](int m) {
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (u < m) { own[u] = chunks[u * per]; dec[u] = decay[u * per_decay]; }
    };
    if (nc >= 8) ask(8);
    else ask(nc);
    float* sp = a.state + (size_t)a.slots[b] * a.state_stride + ((size_t)h * D + d0) * a.Dv + v;
    float4 carry = make_float4(sp[0], sp[a.Dv], sp[2 * a.Dv], sp[3 * a.Dv]);
    auto step = [&](int m) {
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (u < m) {
                chunks[u * per] = carry;
                carry = make_float4(fmaf(dec[u].x, carry.x, own[u].x), fmaf(dec[u].y, carry.y, own[u].y), fmaf(dec[u].z, carry.z, own[u].z), fmaf(dec[u].w, carry.w, own[u].w));
            }
    };
    while (nc >= 8) {
        step(8);
        nc -= 8; chunks += 8 * per; decay += 8 * per_decay;
        if (nc >= 8) ask(8);
        else ask(nc);
    }
    step(nc);
    sp[0] = carry.x; sp[a.Dv] = carry.y; sp[2 * a.Dv] = carry.z; sp[3 * a.Dv] = carry.w;
}

// Chunks of a unit's heads, outputs: the next unit's first rows of the state are asked for while this one's last products run, its queries come when
// these have ended.
template <bool TWO, int VALUE_PARTS>
__global__ void __launch_bounds__(LM_THREADS, 2) lm_output_kernel(LAArgs a, int units) {
    extern __shared__ unsigned char lm_raw[];
    __shared__ __align__(8) unsigned long long bar;
    __shared__ unsigned tmem_s, odd_state, from_s, odd;
    __shared__ __align__(16) float es[TWO ? 2 : 1][LA_CHUNK];
    using Unit = LMUnit<TWO>;
    constexpr int ND = Unit::ND, SLABS = TWO ? 1 : 2;
    unsigned char* ss = lm_raw + (-at_smem(lm_raw) & 1023u);          // [part][half][64 v][64 d] of the state; then the values, [part][half][64 s][64 v]
    unsigned char* qs = ss + 6 * CM_PLANE;                            // [part][two][64 t][64 d]; then the weights, [part][heads][64 t][64 s]
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), per = TWO ? a.H / 2 : a.H, ld_out = a.H * a.Dv;
    const int q = warp & 3, hh = q >> 1, p = (q & 1) * 32 + lane, column = (warp >> 2) * 32;
    const bool scaled = a.z == nullptr;                               // one decay a head: the decay to a token behind the products
    if (tid == 0) odd = 0;
    const unsigned tmem = cm_begin(&tmem_s, &bar), mine = tmem + ((unsigned)(q * 32) << 16) + column + (TWO ? hh * 64 : 0);
    const unsigned elected = warp == 0 ? pe_elect() : 0u;
    pdl_wait();
    unsigned phase = 0, known = 0;
    int2 place = a.chunk_rows[blockIdx.x / per];
    float4 v[4][2];
    auto fetch_state = [&](int unit, int slab) {
        const float* state = a.chunk_state + (size_t)unit * 128 * ND + ((size_t)(slab * 8 + (tid >> 6)) * 64 + (tid & 63)) * 8;
#pragma unroll
        for (int e = 0; e < 4; ++e) cm_load8(v[e][0], v[e][1], state + (size_t)(e >> 1) * ND * 64 + (e & 1) * 4 * 512);
    };
    auto bring_queries = [&](int unit) {
        const int c = unit / per, h0 = unit % per * (TWO ? 2 : 1);
        cm_bring(qs, Unit::of(a, c, h0) + Unit::QUERIES, 6 * CM_PLANE);
        known = lm_known<TWO>(a, c, h0);
    };
    fetch_state(blockIdx.x, 0);
    if (place.y > 0) bring_queries(blockIdx.x);
    for (int unit = blockIdx.x; unit < units && place.y > 0; unit += gridDim.x) {
        const int c = unit / per, h0 = unit % per * (TWO ? 2 : 1), next = unit + gridDim.x, first = place.x, n = place.y;
        if (next < units) place = a.chunk_rows[next / per];
        const unsigned from = known >> 16;
        const bool odd_values = known >> 3 & 1u;
        if (tid == 0) { odd_state = 0; from_s = from; }
        if (scaled && tid < (TWO ? 2 : 1) * LA_CHUNK) {
            double r = 1.0, by = (double)a.head_decay[h0 + (tid >> 6)];
            for (int e = (tid & 63) + 1; e; e >>= 1) { if (e & 1) r *= by; by *= by; }
            es[tid >> 6][tid & 63] = (float)r;
        }
        unsigned most = 0;
        for (int slab = 0; slab < SLABS; ++slab) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float s[8] = {v[e][0].x, v[e][0].y, v[e][0].z, v[e][0].w, v[e][1].x, v[e][1].y, v[e][1].z, v[e][1].w};
                cm_scale(s, CM_UP);
                lm_put<true>(ss + (e >> 1) * CM_PLANE + cm_at(tid & 63, (e & 1) * 4 + (tid >> 6)), 2 * CM_PLANE, s, most);
            }
            if (slab == 0) cm_landed();
            cm_ready();
            if (warp == 0) {
                if constexpr (TWO) cm_products(elected, tmem, tmem + 128, cm_along(at_smem(ss), 2 * CM_PLANE), cm_along(at_smem(qs), 2 * CM_PLANE), cm_idesc(128, false, false));
                else cm_products(elected, tmem + 128 * slab, tmem + 128 * slab + 64, cm_along(at_smem(ss), 2 * CM_PLANE), cm_along(at_smem(qs) + slab * CM_PLANE, 2 * CM_PLANE), cm_idesc(64, false, false));
                if (elected) at_commit(at_smem(&bar));
                __syncwarp();
            }
            if (slab + 1 < SLABS) fetch_state(unit, 1);
            cm_done(&bar, phase, a.status);
        }
        cm_report(&odd_state, cm_seen(most, 0));
        if constexpr (VALUE_PARTS == 1) lm_bring_values(ss, a, first, n, h0 * a.Dv);
        else cm_bring(ss, Unit::of(a, c, h0) + Unit::VALUES, 6 * CM_PLANE);
        cm_bring(qs, Unit::of(a, c, h0) + Unit::WEIGHTS, 3 * Unit::W_HEADS * CM_PLANE);
        float acc[32];
        cm_read(acc, mine + (TWO ? 128 : 64));
        cm_take(acc, mine);
        if constexpr (!TWO) { cm_take(acc, mine + 192); cm_take(acc, mine + 128); }
        if constexpr (VALUE_PARTS == 1) cm_scale(acc, CM_DOWN);       // (as the sums over the values come: one of their operands is cut)
        if (scaled) {
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
                const float4 d = *reinterpret_cast<const float4*>(&es[TWO ? hh : 0][column + i]);
                acc[i] *= d.x; acc[i + 1] *= d.y; acc[i + 2] *= d.z; acc[i + 3] *= d.w;
            }
        }
        cm_landed();
        cm_ready();
        const int exact = odd_state ? 0 : min(n, (int)from);      // tokens in front of it have their outputs from the parts
        if (odd_values) {
            constexpr unsigned LIMIT = VALUE_PARTS == 1 ? CM_MOST_PLAIN : CM_MOST;
            cm_mend(ss, 2 * CM_PLANE, VALUE_PARTS, &from_s, LIMIT);
            cm_mend(ss + CM_PLANE, 2 * CM_PLANE, VALUE_PARTS, &from_s, LIMIT);
            cm_ready();
        }
        if (warp == 0) {
            constexpr int SUM = TWO ? 128 : 64;
            const CMOperand weights = cm_along(at_smem(qs), Unit::W_HEADS * CM_PLANE);
            if constexpr (VALUE_PARTS == 1) cm_products_one(elected, tmem, tmem + SUM, at_desc(at_smem(ss), CM_PLANE, 1024), 128u, weights, cm_idesc(SUM, true, false));
            else cm_products(elected, tmem, tmem + SUM, cm_across(at_smem(ss), 2 * CM_PLANE, CM_PLANE), weights, cm_idesc(SUM, true, false));
            if (elected) at_commit(at_smem(&bar));
            __syncwarp();
        }
        if (next < units) fetch_state(next, 0);
        cm_done(&bar, phase, a.status);
        if (next < units && place.y > 0) bring_queries(next);
        cm_take(acc, mine + (TWO ? 128 : 64));
        cm_take(acc, mine);
        cm_scale(acc, VALUE_PARTS == 1 ? CM_DOWN : CM_DOWN * CM_DOWN);
        float* out = a.out + (size_t)(first + column) * ld_out + h0 * a.Dv + hh * 64 + p;
        if (exact == LA_CHUNK) {
#pragma unroll
            for (int i = 0; i < 32; ++i) out[i * ld_out] = acc[i];
        } else {
#pragma unroll
            for (int i = 0; i < 32; ++i)
                if (column + i < exact) out[i * ld_out] = acc[i];
        }
        if (tid == 0) {
            a.unit_exact[unit] = exact;
            if (exact < n) odd = 1;
        }
    }
    cm_end(tmem);
    if (!odd) return;                                      // (the walks behind the loop: inside they cost its registers)
    __shared__ LAArgs args;
    if (tid == 0) args = a;
    __syncthreads();
#pragma unroll 1
    for (int unit = blockIdx.x; unit < units; unit += gridDim.x) {
        const int2 at = a.chunk_rows[unit / per];
        if (at.y <= 0) break;
        const int exact = a.unit_exact[unit];
        if (exact < at.y) lm_walk<TWO>(args, at.x, at.y, unit % per * (TWO ? 2 : 1), a.chunk_state + (size_t)unit * 128 * ND, exact, nullptr);
    }
}

template <bool TWO, int VP>
static int lm_run(LAArgs a, int types, int z_types, cudaStream_t s) {
    const int units = a.slab * (TWO ? a.H / 2 : a.H), blocks = units < 2 * pe_sm_count() ? units : 2 * pe_sm_count();
    PE_TRY(cudaFuncSetAttribute(lm_contribution_kernel<TWO, VP>, cudaFuncAttributeMaxDynamicSharedMemorySize, LM_SMEM));
    PE_TRY(cudaFuncSetAttribute(lm_output_kernel<TWO, VP>, cudaFuncAttributeMaxDynamicSharedMemorySize, LM_SMEM));
    const int size = types == 2 ? 4 : 2;
    if (a.z) {
        const int z_size = z_types == 0 ? 4 : 2, smem = 4 * (3 * lmc_floats(a.D) + 12 * a.D);
        const int vec_q = (uintptr_t)a.qk % 16 == 0 && a.qk_ld % 8 == 0 && a.q_off % 8 == 0 && a.k_off % 8 == 0, vec_z = (uintptr_t)a.z % 16 == 0 && a.z_ld * z_size % 16 == 0;
        auto kernel = z_types == 0 ? lm_channels_kernel<float, TWO> : lm_channels_kernel<bf16, TWO>;
        PE_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        PE_TRY(pe_launch(kernel, dim3(a.slab, a.H), 512, smem, s, a, vec_q, vec_z));
        PE_LAUNCH_CHECK();
    } else {
        const int vec_q = (uintptr_t)a.qk % 16 == 0 && a.qk_ld * size % 16 == 0 && a.q_off * size % 16 == 0 && a.k_off * size % 16 == 0;
        auto kernel = types == 2 ? lm_prepare_kernel<float, TWO> : lm_prepare_kernel<bf16, TWO>;
        PE_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 6 * CM_PLANE));
        PE_TRY(pe_launch(kernel, dim3(a.slab, a.H), 512, 6 * CM_PLANE, s, a, vec_q));
        PE_LAUNCH_CHECK();
    }
    PE_TRY(pe_launch(lm_contribution_kernel<TWO, VP>, blocks, LM_THREADS, LM_SMEM, s, a, units));
    PE_LAUNCH_CHECK();
    PE_TRY(pe_launch(lm_carry_kernel, dim3(a.H * a.Dv / 8, a.B), 2 * a.D, 0, s, a));
    PE_LAUNCH_CHECK();
    PE_TRY(pe_launch(lm_output_kernel<TWO, VP>, blocks, LM_THREADS, LM_SMEM, s, a, units));
    PE_LAUNCH_CHECK();
    return 0;
}

long long la_tensor_chunk_floats(int H, int D, bool values) {         // a chunk's parts, words and place
    const long long parts = D == 128 ? (long long)H * LMUnit<false>::bytes(values) : (long long)H / 2 * LMUnit<true>::bytes(values);
    return parts / 4 + 2 * H + 2;
}
int la_tensor_chunks(const LAArgs& a, int types, int z_types, cudaStream_t s) {
    if (a.act_v) return a.D == 64 ? lm_run<true, 3>(a, types, z_types, s) : lm_run<false, 3>(a, types, z_types, s);
    return a.D == 64 ? lm_run<true, 1>(a, types, z_types, s) : lm_run<false, 1>(a, types, z_types, s);
}
