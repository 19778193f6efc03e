// Softmax attention of any number of tokens over the paged key/value cache, for every head
// size up to 256 and either dtype: the attention of the true 32-bit path, and the one that
// takes the shapes the tensor-core kernels refuse.
//
// A query at position p of its sequence sees the keys lo..p of that sequence, lo = 0 or
// p - window + 1.  Keys are visited in increasing position, page by page (the kernel of one block a
// (token, head): in chunks that start at lo), so the arithmetic of one (sequence, position, head) is the
// same whether the token came in a long prompt, alone, or beside other sequences.
//
// Scores, softmax and the weighted sum are float32 (pico-engine: src/pico_engine/kernels.py:
// 108-125; its result is stored through float16 at kernels.py:126, which is not done here).
#include "common.cuh"

#define AG_THREADS 128
#define AG_MAX_HD 256

template <typename T>
__global__ void __launch_bounds__(AG_THREADS) attention_generic_kernel(
    const T* q, int q_stride, T* out, const T* k_pool,
    const T* v_pool, const int* block_table, int table_stride,
    const int* tok_pos, const int* tok_row, int nh, int nkv, int hd, int window,
    float scale) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float q_s[AG_MAX_HD];
    __shared__ float p_s[AG_THREADS];
    __shared__ long long base_s[AG_THREADS];
    __shared__ float scratch[33];

    const int t = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
    const int pos = tok_pos[t];
    const int* table = block_table + (size_t)tok_row[t] * table_stride;
    const int kvh = h / (nh / nkv);
    const int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;

    const T* qp = q + (size_t)t * q_stride + (size_t)h * hd;
    for (int d = tid; d < hd; d += AG_THREADS) q_s[d] = to_f(qp[d]);
    __syncthreads();

    float m = -INFINITY, l = 0.f;
    float acc0 = 0.f, acc1 = 0.f;                       // dims tid and tid + AG_THREADS
    for (int c0 = lo; c0 <= pos; c0 += AG_THREADS) {
        const int j = c0 + tid;
        float s = -INFINITY;
        long long base = -1;
        if (j <= pos) {
            const int page = table[j / PE_PAGE];
            if (page >= 0) {
                base = ((long long)page * nkv + kvh) * PE_PAGE * hd + (long long)(j % PE_PAGE) * hd;
                const T* kp = k_pool + base;
                float dot = 0.f;
                for (int d = 0; d < hd; ++d) dot = fmaf(q_s[d], to_f(kp[d]), dot);
                s = dot * scale;
            }
        }
        const float m_new = fmaxf(m, block_max(s, scratch));
        const float alpha = (m == -INFINITY) ? 0.f : expf(m - m_new);
        const float p = (s == -INFINITY) ? 0.f : expf(s - m_new);
        p_s[tid] = p;
        base_s[tid] = base;
        l = l * alpha + block_sum(p, scratch);          // block_sum synchronises: p_s and base_s are visible after it
        m = m_new;
        acc0 *= alpha; acc1 *= alpha;
        const int n = min(AG_THREADS, pos - c0 + 1);
        for (int jj = 0; jj < n; ++jj) {
            const long long b = base_s[jj];
            if (b < 0) continue;
            const float pj = p_s[jj];
            const T* vp = v_pool + b;
            if (tid < hd) acc0 = fmaf(pj, to_f(vp[tid]), acc0);
            if (tid + AG_THREADS < hd) acc1 = fmaf(pj, to_f(vp[tid + AG_THREADS]), acc1);
        }
        __syncthreads();                                 // p_s and base_s are rewritten by the next chunk
    }
    T* op = out + ((size_t)t * nh + h) * hd;
    const float inv = l > 0.f ? 1.0f / l : 0.f;
    if (tid < hd) op[tid] = from_f<T>(acc0 * inv);
    if (tid + AG_THREADS < hd) op[tid + AG_THREADS] = from_f<T>(acc1 * inv);
}

// ---------------------------------------------------------------------------- tiles of rows
// A block: R rows, each a (token, query head); the rows of neighbouring tokens and of the heads that share a key/value head, so that a
// page is read once for all of them.  A step is a page: thread (ty, tx) of 16 x 16 has the scores of R / 16 rows and four keys, then
// R / 16 rows and hd / 16 columns of the outputs.  Tokens of several sequences in a block are served one after the other, each run of
// neighbouring tokens of one sequence by itself (tokens of two sequences may come in any order).
// Whatever R is, a row's scores are sums over the entries in order, its weights are added in the same tree, its outputs in the order of
// the keys of a segment (AG_SEGMENT pages, counted from the sequence's start), and the segments are joined in their order: R = 16 (single
// tokens) and R = 64 (prompts) give the same bits, and so do blocks of one sequence whose segments are dealt out to a cluster
// of CTAs, which join them in shared memory (few rows over a long context, which one CTA walks at 2 to 4 us a page).  A key that a row does not see adds nothing to it, not even
// a value that is no number.  Bound by float32 multiply-adds and the reads from shared memory that feed them.  14 heads of 64 on 2, prompts
// of 301 and 207 tokens, on a B200: 322 us by the kernel above (a block a token and head, which read every key and value once a head), 35 us
// here (34 without segments).  One token behind 700 / 4,000 others 47 / 258 us in one CTA, 12 / 39 as segments over a cluster; twelve
// tokens behind 50 to 1,500 99 and 27; segments of 4 pages 19 / 35 and 30.
#define AT_THREADS 256
#define AG_SEGMENT 2                                      // pages whose sums have a maximum of their own
#define AG_RUN 128                                        // tokens of a run at most

struct AttentionTileArgs {
    const void* q; int q_stride; void* out; const void* k_pool; const void* v_pool;
    const int* table; int table_stride; const int* tok_pos; const int* tok_row;
    int T, nh, nkv, hd, window; float scale;
    int heads, slices, tokens;                     // query heads and tokens of a block's rows; blocks that share a key/value head's heads
    int cluster, buffers;                          // CTAs that share a block's segments; places for a segment's sums
    const int4* runs; int parts;                   // null: blocks of neighbouring packed tokens; else runs (row, first packed token, tokens, ..), `parts` blocks each
};

__device__ __forceinline__ float4 ag_load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 ag_load4(const bf16* p) {
    const uint2 r = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void ag_store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void ag_store4(bf16* p, float4 v) {
    __nv_bfloat162 h[2] = {__floats2bfloat162_rn(v.x, v.y), __floats2bfloat162_rn(v.z, v.w)};
    *reinterpret_cast<uint2*>(p) = *reinterpret_cast<const uint2*>(h);
}
// acc += a * b on four entries, two multiply-adds an instruction (each half rounds as a plain one does)
__device__ __forceinline__ void ag_fma4(float4& acc, float a, const float4& b) {
    asm("{\n\t.reg .b64 pa, b0, b1, c0, c1;\n\t"
        "mov.b64 pa, {%4, %4};\n\tmov.b64 b0, {%5, %6};\n\tmov.b64 b1, {%7, %8};\n\tmov.b64 c0, {%0, %1};\n\tmov.b64 c1, {%2, %3};\n\t"
        "fma.rn.f32x2 c0, pa, b0, c0;\n\tfma.rn.f32x2 c1, pa, b1, c1;\n\t"
        "mov.b64 {%0, %1}, c0;\n\tmov.b64 {%2, %3}, c1;\n\t}"
        : "+f"(acc.x), "+f"(acc.y), "+f"(acc.z), "+f"(acc.w) : "f"(a), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w));
}
// entry d of key (or row) j in a turned tile [hd][64]: neither a thread's four stores nor the reads of four neighbours meet in a bank
__device__ __forceinline__ int ag_turned(int d, int j) { return d * 64 + (j ^ (((d >> 2) & 7) << 2)); }
// (m, l) of what came before joined with the (ms, ls) of a segment; before and now: what the outputs of either are multiplied by.  Nothing
// seen (a maximum of -infinity) changes no bit of the other.
__device__ __forceinline__ void ag_join(float& m, float& l, float ms, float ls, float& before, float& now) {
    const float m_new = fmaxf(m, ms), less = expf(fminf(m, ms) - m_new);       // (one of the two is the new maximum)
    before = m == m_new ? 1.f : m == -INFINITY ? 0.f : less;
    now = ms == m_new ? 1.f : ms == -INFINITY ? 0.f : less;
    l = fmaf(l, before, ls * now);
    m = m_new;
}
__device__ __forceinline__ void ag_join4(float4& acc, float before, const float4& v, float now) {
    acc.x = fmaf(acc.x, before, v.x * now); acc.y = fmaf(acc.y, before, v.y * now); acc.z = fmaf(acc.z, before, v.z * now); acc.w = fmaf(acc.w, before, v.w * now);
}
__device__ __forceinline__ void ag_cluster_sync() { asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ unsigned ag_peer(const float* mine, int rank) {
    unsigned at = (unsigned)__cvta_generic_to_shared(mine), peer;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(at), "r"(rank));
    return peer;
}
__device__ __forceinline__ float ag_peer1(const float* mine, int rank) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(ag_peer(mine, rank)) : "memory");
    return v;
}
__device__ __forceinline__ float4 ag_peer4(const float* mine, int rank) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(ag_peer(mine, rank)) : "memory");
    return v;
}
struct ag_yes { static constexpr bool value = true; };
struct ag_no { static constexpr bool value = false; };

template <typename T, int R, int NJ>
__global__ void __launch_bounds__(AT_THREADS, R == 16 && NJ == 1 ? 2 : 1) attention_tile_kernel(AttentionTileArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int RT = R / 16;                             // rows a thread
    extern __shared__ __align__(16) float ag_smem[];
    __shared__ int pos_s[R], row_s[R], run_s[R], last_s;
    const int hd = a.hd, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, per4 = hd / 4;
    float* qt = ag_smem;                                   // [hd][64]: the rows' queries, turned (R of 64 places used)
    float* kt = qt + hd * 64;                              // [hd][64]: a page's keys, turned
    float* vs = kt + hd * 64;                              // [64][hd]
    float* ps = vs + hd * 64;                              // [64 keys][R]: weights, rows in groups of four exchanged by the key
    float* joint = ps + 64 * R;                            // a cluster: one or two buffers of a segment's maxima [R], sums [R] and outputs [R][hd]
    const int C = R == 16 ? a.cluster : 1, member = C > 1 ? blockIdx.x % C : 0, block = C > 1 ? blockIdx.x / C : blockIdx.x;
    const int per = a.nh / a.nkv, kvh = blockIdx.y / a.slices, h0 = kvh * per + blockIdx.y % a.slices * a.heads;
    int t0 = block * a.tokens, left = a.T - t0;
    if (a.runs) {
        const int4 run = a.runs[block / a.parts];
        const int behind = block % a.parts * a.tokens;
        t0 = run.y + behind; left = run.z - behind;
        if (left <= 0) return;
    }
    const int n_heads = min(a.heads, kvh * per + per - h0), n_tok = min(a.tokens, left);
    if (member > 0) {                                      // one segment is the first member's: nobody waits for anybody
        int lowest = a.tok_pos[t0], highest = lowest;
        for (int t = 1; t < n_tok; ++t) { lowest = min(lowest, a.tok_pos[t0 + t]); highest = max(highest, a.tok_pos[t0 + t]); }
        if ((a.window > 0 ? max(lowest - a.window + 1, 0) : 0) / (PE_PAGE * AG_SEGMENT) == highest / (PE_PAGE * AG_SEGMENT)) return;
    }
    const int rows = n_heads * n_tok;                      // row r: token t0 + r / n_heads, head h0 + r % n_heads
    if (tid < R) {
        const int t = t0 + min(tid, rows - 1) / n_heads;
        pos_s[tid] = a.tok_pos[t];
        row_s[tid] = tid < rows ? a.tok_row[t] : -1;
    }
    // a row's run: the first of the rows of its sequence that stand together with it
    const bool one = a.runs || a.tokens == 1;              // (one sequence: the first row)
    if (!one) __syncthreads();
    if (!one && tid < (R < 32 ? 32 : R)) {
        const unsigned begins = __ballot_sync(0xffffffffu, tid < R && (tid == 0 || row_s[tid] != row_s[tid - 1])) & (0xffffffffu >> (31 - (tid & 31)));
        if (tid < R) run_s[tid] = begins ? (tid & ~31) + 31 - __clz(begins) : -1;
        if (tid == 31) last_s = 31 - __clz(begins);        // (of the first 32 rows' runs: the first row always begins one)
    }
    for (int i = tid; i < R * per4; i += AT_THREADS) {
        const int r = i / per4, c = i % per4 * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < rows) v = ag_load4((const T*)a.q + (size_t)(t0 + r / n_heads) * a.q_stride + (size_t)(h0 + r % n_heads) * hd + c);
        qt[ag_turned(c, r)] = v.x; qt[ag_turned(c + 1, r)] = v.y; qt[ag_turned(c + 2, r)] = v.z; qt[ag_turned(c + 3, r)] = v.w;
    }
    __syncthreads();
    float m[RT], l[RT], m_all[RT], l_all[RT];              // of a segment, and of those before it
    float4 acc[RT][NJ], all[RT][NJ];
    float joined_m[NJ], joined_l[NJ];                      // a cluster: of the rows whose columns this thread joins
#pragma unroll
    for (int j = 0; j < NJ; ++j) { joined_m[j] = -INFINITY; joined_l[j] = 0.f; }
    int my_pos[RT], my_run[RT];
#pragma unroll
    for (int i = 0; i < RT; ++i) {
        m[i] = m_all[i] = -INFINITY; l[i] = l_all[i] = 0.f;
        my_pos[i] = pos_s[ty * RT + i]; my_run[i] = one ? (ty * RT + i < rows ? 0 : -1) : run_s[ty * RT + i] >= 0 ? run_s[ty * RT + i] : last_s;
#pragma unroll
        for (int j = 0; j < NJ; ++j) acc[i][j] = all[i][j] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    // Where a page's rows are few enough registers (PRE: a thread's share of up to PU vectors of keys and of values), the next page
    // travels while this one is used.  A thread's vectors are AT_THREADS apart: their (key, entry) advance by fixed steps.
    constexpr int PU = 4 * NJ;
    constexpr bool PRE = NJ == 1 || (NJ == 2 && RT == 1);
    float4 pk[PRE ? PU : 1], pv[PRE ? PU : 1];
    const int j_first = tid / per4, c_first = tid % per4 * 4, j_step = AT_THREADS / per4, c_step = AT_THREADS % per4 * 4;
    auto fetch = [&](size_t base) {
#pragma unroll
        for (int u = 0; u < PU; ++u) {
            const int i = tid + u * AT_THREADS;
            if (i < PE_PAGE * per4) {
                pk[PRE ? u : 0] = ag_load4((const T*)a.k_pool + base + (size_t)i * 4);
                pv[PRE ? u : 0] = ag_load4((const T*)a.v_pool + base + (size_t)i * 4);
            }
        }
    };
    auto turn = [&](int j, int c, const float4& k) { kt[ag_turned(c, j)] = k.x; kt[ag_turned(c + 1, j)] = k.y; kt[ag_turned(c + 2, j)] = k.z; kt[ag_turned(c + 3, j)] = k.w; };
    bool alone = true;                                     // no other CTA has a part in this block's rows
    for (int from = 0; from < rows;) {                     // the rows of one sequence that stand together, after them the next ones
        const int seq = row_s[from];
        int to = from + n_heads, lowest = pos_s[from], highest = lowest;
        while (to < rows && row_s[to] == seq) { lowest = min(lowest, pos_s[to]); highest = max(highest, pos_s[to]); to += n_heads; }
        const int* table = a.table + (size_t)seq * a.table_stride;
        const int page_lo = a.window > 0 && lowest - a.window + 1 > 0 ? (lowest - a.window + 1) / PE_PAGE : 0;
        const int page_hi = highest / PE_PAGE;
        const auto base_of = [&](int pg) { return ((size_t)pg * a.nkv + kvh) * PE_PAGE * hd; };
        int page = -1;                                     // the one whose keys and values are on their way (PRE)
        const auto visit = [&](int pg, int here) {         // a page's keys
            __syncthreads();                               // the page before has been used
            int j = j_first, c = c_first;
            if constexpr (PRE) {
#pragma unroll
                for (int u = 0; u < PU; ++u) {
                    if (j < PE_PAGE) {
                        turn(j, c, pk[u]);
                        *reinterpret_cast<float4*>(vs + j * hd + c) = pv[u];
                    }
                    j += j_step; c += c_step;
                    if (c >= hd) { c -= hd; ++j; }
                }
                if (page >= 0) fetch(base_of(page));
            } else {
                const size_t base = base_of(here);
#pragma unroll 4
                while (j < PE_PAGE) {
                    turn(j, c, ag_load4((const T*)a.k_pool + base + (size_t)j * hd + c));
                    *reinterpret_cast<float4*>(vs + j * hd + c) = ag_load4((const T*)a.v_pool + base + (size_t)j * hd + c);
                    j += j_step; c += c_step;
                    if (c >= hd) { c -= hd; ++j; }
                }
            }
            __syncthreads();
            float4 s[RT];
#pragma unroll
            for (int i = 0; i < RT; ++i) s[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
            for (int d = 0; d < hd; ++d) {
                const float4 k = *reinterpret_cast<const float4*>(kt + ag_turned(d, tx * 4));
                if constexpr (RT == 4) {
                    const float4 q = *reinterpret_cast<const float4*>(qt + ag_turned(d, ty * 4));
                    ag_fma4(s[0], q.x, k); ag_fma4(s[1], q.y, k); ag_fma4(s[2], q.z, k); ag_fma4(s[3], q.w, k);
                } else ag_fma4(s[0], qt[ag_turned(d, ty)], k);
            }
            // which of the four keys a row sees; the rows' new maxima and weights
            const int key0 = pg * PE_PAGE + tx * 4;
            bool whole = true;                             // this thread's rows see the whole page
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                const int first_key = pg * PE_PAGE;
                whole = whole && my_run[i] == from && my_pos[i] >= first_key + PE_PAGE - 1 && (a.window <= 0 || my_pos[i] - first_key < a.window);
            }
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                s[i].x *= a.scale; s[i].y *= a.scale; s[i].z *= a.scale; s[i].w *= a.scale;
                if (whole) continue;
                const int hi = my_run[i] == from ? my_pos[i] - key0 : -1, lo = a.window > 0 ? hi - a.window + 1 : 0;      // keys lo .. hi of the four
                s[i].x = hi >= 0 && lo <= 0 ? s[i].x : -INFINITY;
                s[i].y = hi >= 1 && lo <= 1 ? s[i].y : -INFINITY;
                s[i].z = hi >= 2 && lo <= 2 ? s[i].z : -INFINITY;
                s[i].w = hi >= 3 && lo <= 3 ? s[i].w : -INFINITY;
            }
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                float mx = fmaxf(fmaxf(s[i].x, s[i].y), fmaxf(s[i].z, s[i].w));
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                const float m_new = fmaxf(m[i], mx), alpha = m[i] == -INFINITY ? 0.f : expf(m[i] - m_new);
                s[i].x = s[i].x == -INFINITY ? 0.f : expf(s[i].x - m_new); s[i].y = s[i].y == -INFINITY ? 0.f : expf(s[i].y - m_new);
                s[i].z = s[i].z == -INFINITY ? 0.f : expf(s[i].z - m_new); s[i].w = s[i].w == -INFINITY ? 0.f : expf(s[i].w - m_new);
                float sum = (s[i].x + s[i].y) + (s[i].z + s[i].w);
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                if (my_run[i] == from) {
                    l[i] = l[i] * alpha + sum;
                    m[i] = m_new;
#pragma unroll
                    for (int j = 0; j < NJ; ++j) { acc[i][j].x *= alpha; acc[i][j].y *= alpha; acc[i][j].z *= alpha; acc[i][j].w *= alpha; }
                }
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const auto at = [e](const float4& v) { return e == 0 ? v.x : e == 1 ? v.y : e == 2 ? v.z : v.w; };
                float* p = ps + (tx * 4 + e) * R;
                if constexpr (RT == 4) *reinterpret_cast<float4*>(p + ((ty * 4) ^ ((tx & 7) << 2))) = make_float4(at(s[0]), at(s[1]), at(s[2]), at(s[3]));
                else p[ty] = at(s[0]);
            }
            __syncthreads();
            // guarded: a row adds nothing of a key whose weight is zero (a weight that is no number joins)
            const auto add_values = [&](int keys, auto guarded) {
#pragma unroll 8
                for (int k = 0; k < keys; ++k) {
                    float p[RT];
                    if constexpr (RT == 4) *reinterpret_cast<float4*>(p) = *reinterpret_cast<const float4*>(ps + k * R + ((ty * 4) ^ (((k >> 2) & 7) << 2)));
                    else p[0] = ps[k * R + ty];
#pragma unroll
                    for (int j = 0; j < NJ; ++j) {
                        const int c = tx * 4 + 64 * j;
                        const float4 v = *reinterpret_cast<const float4*>(vs + k * hd + (c < hd ? c : 0));      // (columns that are none are not stored)
#pragma unroll
                        for (int i = 0; i < RT; ++i)
                            if (!decltype(guarded)::value || p[i] != 0.f) ag_fma4(acc[i][j], p[i], v);
                    }
                }
            };
            if (__all_sync(0xffffffffu, whole)) add_values(PE_PAGE, ag_no());
            else add_values(min(PE_PAGE, highest - pg * PE_PAGE + 1), ag_yes());
        };
        const auto fresh = [&]() {
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                if (my_run[i] != from) continue;
                m[i] = -INFINITY; l[i] = 0.f;
#pragma unroll
                for (int j = 0; j < NJ; ++j) acc[i][j] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        };
        alone = C == 1 || page_lo / AG_SEGMENT == page_hi / AG_SEGMENT;
        if (alone) {
            int segment = -1;
            const auto join = [&]() {                      // the segment joins those before it
#pragma unroll
                for (int i = 0; i < RT; ++i) {
                    float before, now;
                    if (my_run[i] != from) continue;
                    ag_join(m_all[i], l_all[i], m[i], l[i], before, now);
#pragma unroll
                    for (int j = 0; j < NJ; ++j) ag_join4(all[i][j], before, acc[i][j], now);
                }
                fresh();
            };
            page = table[page_lo];
            if (PRE && page >= 0) fetch(base_of(page));
            for (int pg = page_lo; pg <= page_hi; ++pg) {
                const int here = page;
                page = pg < page_hi ? table[pg + 1] : -1;
                if (here < 0) {
                    if (PRE && page >= 0) fetch(base_of(page));
                    continue;
                }
                if (pg / AG_SEGMENT != segment) {
                    if (segment >= 0) join();
                    segment = pg / AG_SEGMENT;
                }
                visit(pg, here);
            }
            join();
        } else {
            // a member of a cluster has every C-th segment; all of them take as many turns
            const auto following = [&](int pg) { return ++pg % AG_SEGMENT ? pg : pg + (C - 1) * AG_SEGMENT; };
            const auto page_at = [&](int pg) { return pg >= page_lo && pg <= page_hi ? table[pg] : -1; };
            const int past = (page_hi / AG_SEGMENT + 1 + member) * AG_SEGMENT;
            int pg = (page_lo / AG_SEGMENT + member) * AG_SEGMENT, turns = 0;
            page = page_at(pg);
            if (PRE && page >= 0) fetch(base_of(page));
            for (; pg < past; pg = following(pg)) {
                const int here = page;
                page = page_at(following(pg));
                if (here >= 0) visit(pg, here);
                else if (PRE && page >= 0) fetch(base_of(page));
                if (pg % AG_SEGMENT != AG_SEGMENT - 1) continue;
                // C segments join those before them, each of its CTA: a thread four columns of a row
                float* mine = joint + (turns & (a.buffers - 1)) * R * (hd + 2);
                if (tx == 0) { mine[ty] = m[0]; mine[R + ty] = l[0]; }
    #pragma unroll
                for (int j = 0; j < NJ; ++j)
                    if (tx * 4 + 64 * j < hd) *reinterpret_cast<float4*>(mine + 2 * R + ty * hd + tx * 4 + 64 * j) = acc[0][j];
                ag_cluster_sync();
                const int here_now = min(C, page_hi / AG_SEGMENT - page_lo / AG_SEGMENT + 1 - turns * C);
    #pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    const int i = member + C * (tid + j * AT_THREADS), r = i / per4, c = i % per4 * 4;
                    if (r >= rows) break;
    #pragma unroll 1
                    for (int p0 = 0; p0 < here_now; p0 += 2) {     // (C is a power of two; who has no segment has seen nothing)
                        float ms[2], ls[2], before, now;
                        float4 vs2[2];
    #pragma unroll
                        for (int p = 0; p < 2; ++p) { ms[p] = ag_peer1(mine + r, p0 + p); ls[p] = ag_peer1(mine + R + r, p0 + p); vs2[p] = ag_peer4(mine + 2 * R + r * hd + c, p0 + p); }
    #pragma unroll
                        for (int p = 0; p < 2; ++p) {
                            ag_join(joined_m[j], joined_l[j], ms[p], ls[p], before, now);
                            ag_join4(all[0][j], before, vs2[p], now);
                        }
                    }
                }
                if (a.buffers == 1) ag_cluster_sync();         // (with two, nobody is two turns ahead of a reader)
                ++turns;
                fresh();
            }
        }
        from = to;
    }
    const auto store = [&](int r, int c, const float4& v, float sum) {
        const float inv = sum > 0.f ? 1.0f / sum : 0.f;
        ag_store4((T*)a.out + ((size_t)(t0 + r / n_heads) * a.nh + h0 + r % n_heads) * hd + c, make_float4(v.x * inv, v.y * inv, v.z * inv, v.w * inv));
    };
    if (!alone) {
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const int i = member + C * (tid + j * AT_THREADS);
            if (i / per4 < rows) store(i / per4, i % per4 * 4, all[0][j], joined_l[j]);
        }
        ag_cluster_sync();                                 // nobody leaves while its sums are being read
        return;
    }
#pragma unroll
    for (int i = 0; i < RT; ++i) {
        const int r = ty * RT + i;
        if (r >= rows) continue;
#pragma unroll
        for (int j = 0; j < NJ; ++j)
            if (tx * 4 + 64 * j < hd) store(r, tx * 4 + 64 * j, all[i][j], l_all[i]);
    }
}

template <typename T, int R, int NJ>
static int attention_tile_as(AttentionTileArgs a, int n_runs, int most, cudaStream_t s) {
    const int per = a.nh / a.nkv;
    a.heads = per < R ? per : R;
    a.slices = (per + a.heads - 1) / a.heads;
    a.tokens = R / a.heads < most ? R / a.heads : most;
    a.parts = (AG_RUN + a.tokens - 1) / a.tokens;
    if (a.runs) a.tokens = (AG_RUN + a.parts - 1) / a.parts;          // a whole run in equal parts
    const int blocks = a.runs ? n_runs * a.parts : (a.T + a.tokens - 1) / a.tokens;
    // A cluster for each block of one sequence's rows where those leave SMs idle: as many CTAs as a context that fills its row of the page table
    // has segments (how long contexts are is on the device; a captured step's tables are as wide as contexts may become).
    // All of them fit at once, two an SM of heads of up to 64 and one of larger ones: eight tokens behind 200, 16 heads of 128 on 4, 46 us with clusters
    // of eight, which do not.
    a.cluster = 1;
    if (R == 16 && (a.runs || a.tokens == 1))
        while (a.cluster < 8 && (long long)2 * a.cluster * blocks * a.nkv * a.slices <= (NJ == 1 ? 2 * 148 : 148) && a.cluster * AG_SEGMENT < a.table_stride) a.cluster *= 2;
    a.buffers = a.hd > 192 ? 1 : 2;
    const size_t smem = sizeof(float) * ((size_t)3 * a.hd * 64 + 64 * R + (a.cluster > 1 ? a.buffers * R * (a.hd + 2) : 0));
    auto kernel = attention_tile_kernel<T, R, NJ>;
    PE_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    PE_TRY(pe_launch_cluster(kernel, dim3(blocks * a.cluster, a.nkv * a.slices), AT_THREADS, smem, s, a.cluster, a));
    PE_LAUNCH_CHECK();
    return 0;
}
template <typename T>
static int attention_tile(const AttentionTileArgs& a, int n_runs, int sequences, cudaStream_t s) {
    const int per = a.nh / a.nkv, few = per < 16 ? 16 / per : 1;      // tokens of a block of 16 rows
    // Which blocks: 16 rows while those fill half of the SMs at most, else 64 (14 heads of 64 on 2, before rows of few blocks were dealt out to clusters: 60
    // tokens alone 7.6 / 10.5 us, 20 behind 4,000 261 / 363, 100 behind 4,000 418 / 373).  Where no runs are known a block may get tokens of several sequences, which
    // it serves one after the other: no more of them than a quarter of what a sequence brings on average, and so single ones where they bring few.
    // One prompt of 40 tokens beside 30 single tokens at 600, float32, on a B200, a block a token and head / 64 rows of neighbouring tokens
    // / runs: 14 heads of 64 on 2 255 / 506 / 71 us, 4 of 256 on one 275 / 3,801 / 173.
    const int most = a.runs ? AG_RUN : sequences > 0 && a.T / sequences >= 16 ? a.T / sequences / 4 : 1;
    const int blocks16 = (a.T + min(few, most) - 1) / min(few, most);
    const bool wide = (long long)most * per > 16 && (long long)blocks16 * a.nkv * ((per + 15) / 16) > 74;
    if (a.hd <= 64) return wide ? attention_tile_as<T, 64, 1>(a, n_runs, most, s) : attention_tile_as<T, 16, 1>(a, n_runs, most, s);
    if (a.hd <= 128) return wide ? attention_tile_as<T, 64, 2>(a, n_runs, most, s) : attention_tile_as<T, 16, 2>(a, n_runs, most, s);
    return wide ? attention_tile_as<T, 64, 4>(a, n_runs, most, s) : attention_tile_as<T, 16, 4>(a, n_runs, most, s);
}

// runs: null, or [n_runs] of (batch row, first packed token, number of tokens (<= 128), ..): the step's tokens, each in one of them
extern "C" int pe_attention_generic(const void* q, int q_stride, void* out, const void* k_pool, const void* v_pool,
                                    int dtype, const int* block_table, int table_stride, const int* tok_pos,
                                    const int* tok_row, int T, int nh, int nkv, int hd, int window, float scale, int sequences,
                                    const void* runs, int n_runs, void* stream) {
    if (T <= 0) return 0;
    if (hd <= 0 || hd > AG_MAX_HD || nkv <= 0 || nh % nkv || nh > 65535) return PE_ERR_UNSUPPORTED;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t size = dtype == PE_F32 ? 4 : 2;
    if ((dtype == PE_F32 || dtype == PE_BF16) && hd % 4 == 0 && q_stride % 4 == 0 && !(((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_pool | (uintptr_t)v_pool) % (4 * size))) {
        // rows of four entries that can be read at once: tiles of rows
        const AttentionTileArgs a = {q, q_stride, out, k_pool, v_pool, block_table, table_stride, tok_pos, tok_row, T, nh, nkv, hd, window, scale, 0, 0, 0, 1, 1,
                                     (const int4*)runs, 0};
        return dtype == PE_F32 ? attention_tile<float>(a, n_runs, sequences, s) : attention_tile<bf16>(a, n_runs, sequences, s);
    }
    dim3 grid(T, nh);
    if (dtype == PE_F32)
        PE_TRY(pe_launch(attention_generic_kernel<float>, grid, AG_THREADS, 0, s, (const float*)q, q_stride, (float*)out,
            (const float*)k_pool, (const float*)v_pool, block_table, table_stride, tok_pos, tok_row, nh, nkv, hd, window, scale));
    else if (dtype == PE_BF16)
        PE_TRY(pe_launch(attention_generic_kernel<bf16>, grid, AG_THREADS, 0, s, (const bf16*)q, q_stride, (bf16*)out,
            (const bf16*)k_pool, (const bf16*)v_pool, block_table, table_stride, tok_pos, tok_row, nh, nkv, hd, window, scale));
    else return PE_ERR_UNSUPPORTED;
    PE_LAUNCH_CHECK();
    return 0;
}
