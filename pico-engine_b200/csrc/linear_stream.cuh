// The decode products of linear_fused.cu (up to 16 rows, the same prologues and epilogues) for weights of more than a few megabytes.
//
// What bounds such a product is how many bytes of W are on their way at any time, from the kernel's first to its last moment.  A CTA of
// linear_fused.cu owns one tile of W: it fills its stages, works them off and ends, and an SM's next CTA starts empty.  Here a CTA has
// groups of up to 32 rows of W one after the other (blockIdx.x, + gridDim.x, ..), and its eight warps share a group's columns, 64 at a time in turn, each with
// a ring of its own of three or four pairs of boxes (TMA tiled loads, 128-byte swizzle) that it refills as soon as it has used one: the next group's
// columns are on their way while a group's sums are added up, and no warp waits for another in between.  96 to 128 KB an SM are in flight
// (two pairs of boxes a warp, so that two kernels fit an SM: gate/up of 37888 x 3584 49 us instead of 45, down 24.5 instead of 23.2).
//
// A group is two boxes of `height` rows: for SWIGLU matching gate and up rows, for ROPE the two halves of a head that rotate together
// (heights divide a head's half), else neighbouring rows; one box where a CTA has no more than 16 rows.  Heights are chosen so that all CTAs have
// nearly the same number of rows.  Activations: float32 rows are normed, rounded and kept in shared memory for all groups
// (the row's 1/rms is applied to the sums); of bfloat16 rows 64 columns come with each pair of boxes.
//
// A row's sums do not depend on its neighbours: columns are added in the order of the warps that have them, whatever M is.
//
// A wait that runs out sets *status to 10.  The whole CTA leaves before it writes anything of that group or of a later one, when what it has
// under way has landed (a wait with a limit again).
#pragma once
#include "tcgen05_attention.cuh"

#define LS_WARPS 8
#define LS_BOX (16 * 128)
// Bytes of a box's place: two boxes of W, and one of the activations where these come with them.
template <int NT, int PRO> constexpr int ls_slot_bytes() { return 2 * LS_BOX + (PRO == LF_RMSNORM ? 0 : NT * 1024); }
template <int NT, int PRO, int SLOTS> constexpr int ls_ring_bytes() { return LS_WARPS * SLOTS * ls_slot_bytes<NT, PRO>(); }

struct LsArgs {
    LfArgs f;
    int units, height, groups;       // row pairs (SWIGLU, ROPE) or rows; rows of a box; groups of boxes
    int pair;                        // a group is two boxes
};

__device__ __forceinline__ uint4 ls_lds16(unsigned at) { return lf_lds16(at); }

// SLOTS: boxes of a group that a warp has under way
template <int NT, int PRO, int EPI, int SLOTS>
__global__ void __launch_bounds__(32 * LS_WARPS, 1) linear_stream_kernel(const __grid_constant__ CUtensorMap map, const __grid_constant__ CUtensorMap map_a, const LsArgs a, int* status) {
    constexpr int SLOT = ls_slot_bytes<NT, PRO>();
    constexpr bool PAIRS = EPI == LF_SWIGLU || EPI == LF_ROPE;
    extern __shared__ unsigned char ls_smem[];              // ring, then (RMSNORM) the rows [8 NT][K + 8] bfloat16
    __shared__ __align__(8) unsigned long long bars[LS_WARPS * SLOTS];
    __shared__ float red[LS_WARPS][2 * NT * 4][32], ssq[LS_WARPS][NT * 8];
    const LfArgs& p = a.f;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int M = p.M, K = p.K, chunks = (K + 63) / 64;
    const unsigned ring = ((at_smem(ls_smem) + 1023u) & ~1023u) + warp * SLOTS * SLOT, bar = at_smem(bars + warp * SLOTS);
    const unsigned rows_at = ((at_smem(ls_smem) + 1023u) & ~1023u) + ls_ring_bytes<NT, PRO, SLOTS>(), row_bytes = (unsigned)(K + 8) * 2u;
    const int half = EPI == LF_ROPE ? p.hd >> 1 : 0;
    // first row of W of a group's boxes
    const auto lo_row = [&](int group) {
        if (EPI == LF_ROPE) { const int u = group * a.height; return u / half * p.hd + u % half; }
        return EPI == LF_SWIGLU ? group * a.height : group * a.height * (a.pair ? 2 : 1);
    };
    const auto hi_row = [&](int group) { return lo_row(group) + (EPI == LF_ROPE ? half : EPI == LF_SWIGLU ? p.I : a.height); };
    const unsigned bytes = (unsigned)(a.pair ? 2 : 1) * a.height * 128u + (PRO == LF_PLAIN ? NT * 1024u : 0u);

    if (lane == 0) {
        for (int s = 0; s < SLOTS; ++s) lf_bar_init(bar + 8 * s, 1u);
        asm volatile("fence.mbarrier_init.release.cluster;\n\tfence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    pdl_launch_dependents();
    // this warp's boxes in order: groups, and of each the columns warp * 64, + 512, ..
    int next_group = blockIdx.x, next_chunk = warp, sent = 0;
    const auto send = [&]() {
        if (next_chunk >= chunks || next_group >= a.groups) return;
        if (lane == 0) {
            const unsigned s = sent % SLOTS, to = ring + s * SLOT;
            lf_bar_expect(bar + 8 * s, bytes);
            at_tma_2d(to, &map, next_chunk * 64, lo_row(next_group), bar + 8 * s);
            if (a.pair) at_tma_2d(to + LS_BOX, &map, next_chunk * 64, hi_row(next_group), bar + 8 * s);
            if (PRO == LF_PLAIN && sent >= SLOTS) at_tma_2d(to + 2 * LS_BOX, &map_a, next_chunk * 64, 0, bar + 8 * s);      // (the first ones' follow the wait)
        }
        ++sent;
        next_chunk += LS_WARPS;
        if (next_chunk >= chunks) { next_chunk = warp; next_group += gridDim.x; }
    };
    for (int s = 0; s < SLOTS; ++s) send();                 // weights: no kernel writes them
    if (PRO == LF_RMSNORM) {                                // the norm's weights too, into L1
        const unsigned n = (unsigned)K * (p.norm_w_dtype == PE_BF16 ? 2u : 4u);
        for (unsigned o = tid * 128u; o < n; o += 32u * LS_WARPS * 128u) asm volatile("prefetch.global.L1 [%0];" ::"l"((const char*)p.norm_w + o) : "memory");
    }
    pdl_wait();
    if (PRO == LF_PLAIN && lane == 0)
        for (int s = 0, c = warp; s < sent; ++s) {
            at_tma_2d(ring + s * SLOT + 2 * LS_BOX, &map_a, c * 64, 0, bar + 8 * s);
            c += LS_WARPS;
            if (c >= chunks) c = warp;
        }

    if (PRO == LF_RMSNORM) {
        // bfloat16(x * w) of every row, a warp an eighth of the columns; rows that are none read as zeros
        const int per = ((K / 8 + LS_WARPS - 1) / LS_WARPS) * 8, from = warp * per, to = min(K, from + per);
        float sums[NT * 8];
#pragma unroll
        for (int m = 0; m < NT * 8; ++m) sums[m] = 0.f;
        for (int k = from + lane * 8; k < to; k += 256) {
            float w[8];
            if (p.norm_w_dtype == PE_BF16) {
                const uint4 wv = *reinterpret_cast<const uint4*>((const bf16*)p.norm_w + k);
                const __nv_bfloat162* w2 = reinterpret_cast<const __nv_bfloat162*>(&wv);
#pragma unroll
                for (int e = 0; e < 4; ++e) { const float2 f = __bfloat1622float2(w2[e]); w[2 * e] = f.x; w[2 * e + 1] = f.y; }
            } else {
                const float4 w0 = *reinterpret_cast<const float4*>((const float*)p.norm_w + k), w1 = *reinterpret_cast<const float4*>((const float*)p.norm_w + k + 4);
                w[0] = w0.x; w[1] = w0.y; w[2] = w0.z; w[3] = w0.w; w[4] = w1.x; w[5] = w1.y; w[6] = w1.z; w[7] = w1.w;
            }
#pragma unroll
            for (int m = 0; m < NT * 8; ++m) {               // (all rows' loads are asked for together)
                float4 x0 = make_float4(0.f, 0.f, 0.f, 0.f), x1 = x0;
                if (m < M) { x0 = *reinterpret_cast<const float4*>(p.X + (size_t)m * K + k); x1 = *reinterpret_cast<const float4*>(p.X + (size_t)m * K + k + 4); }
                sums[m] += x0.x * x0.x + x0.y * x0.y + x0.z * x0.z + x0.w * x0.w + x1.x * x1.x + x1.y * x1.y + x1.z * x1.z + x1.w * x1.w;
                asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(rows_at + m * row_bytes + k * 2), "r"(lf_pack(x0.x * w[0], x0.y * w[1])),
                             "r"(lf_pack(x0.z * w[2], x0.w * w[3])), "r"(lf_pack(x1.x * w[4], x1.y * w[5])), "r"(lf_pack(x1.z * w[6], x1.w * w[7])));
            }
        }
#pragma unroll
        for (int m = 0; m < NT * 8; ++m) {
            const float sum = warp_sum(sums[m]);
            if (lane == 0) ssq[warp][m] = sum;
        }
        __syncthreads();
    }

    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    int used = 0;
    bool late = false;                                      // a box of this warp's has not come
    for (int group = blockIdx.x; group < a.groups; group += gridDim.x) {
        // ROPE: what the epilogue needs of the step's description and of the rotation tables is asked for now
        const int ep_r = (lane >> 2) + 8 * ((warp >> 1) & 1), ep_m = (warp >> 2) * 8 + 2 * (lane & 3) + (warp & 1);      // this thread's row and token (256 threads: two tokens' groups)
        int ep_pos = 0, ep_page = -1;
        float ep_cos = 1.f, ep_sin = 0.f;
        const int unit = PAIRS ? group * a.height + ep_r : 0, head = EPI == LF_ROPE ? unit / half : 0, d = EPI == LF_ROPE ? unit % half : 0;
        if (EPI == LF_ROPE && ep_m < M && ep_r < a.height && unit < a.units) {
            ep_pos = p.tok_pos[ep_m];
            if (head < p.n_q + p.n_kv && p.cos_t) { ep_cos = p.cos_t[(size_t)ep_pos * half + d]; ep_sin = p.sin_t[(size_t)ep_pos * half + d]; }
            if (head >= p.n_q && p.store) ep_page = p.block_table[(size_t)p.tok_row[ep_m] * p.table_stride + ep_pos / PE_PAGE];
        }
        float acc[2][NT][4];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.f;
        for (int c = warp; c < chunks; c += LS_WARPS) {
            const unsigned s = used % SLOTS, w_at = ring + s * SLOT;
            if (!lf_bar_wait(bar + 8 * s, (used / SLOTS) & 1)) {      // (the warp asks as one: a vote here costs a twentieth of the time)
                late = true;
                break;
            }
            ++used;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const unsigned at = w_at + g * 128 + (((4 * k + t) ^ g) << 4);       // rows g and g + 8 of a box: eight rows a turn of the swizzle
                const uint4 l0 = lf_lds16(at), l1 = lf_lds16(at + 1024), h0 = a.pair ? lf_lds16(at + LS_BOX) : zero, h1 = a.pair ? lf_lds16(at + LS_BOX + 1024) : zero;
#pragma unroll
                for (int j = 0; j < NT; ++j) {               // rows of activations: entries 8 t .. 8 t + 7 of these 32 (behind the last column: zeros)
                    const int col = c * 64 + 32 * k + 8 * t;
                    const uint4 v = PRO == LF_PLAIN ? lf_lds16(w_at + 2 * LS_BOX + j * 1024 + g * 128 + (((4 * k + t) ^ g) << 4))
                                                    : col < K ? lf_lds16(rows_at + (j * 8 + g) * row_bytes + col * 2) : zero;
                    lf_mma(acc[0][j], l0.x, l1.x, l0.y, l1.y, v.x, v.y);
                    lf_mma(acc[0][j], l0.z, l1.z, l0.w, l1.w, v.z, v.w);
                    lf_mma(acc[1][j], h0.x, h1.x, h0.y, h1.y, v.x, v.y);
                    lf_mma(acc[1][j], h0.z, h1.z, h0.w, h1.w, v.z, v.w);
                }
            }
            __syncwarp();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");             // the slot's reads precede its refill
            send();
        }
        // acc[i][j][e] of lane (g, t): row g (+ 8 if e & 2) of box i, token j * 8 + 2 t + (e & 1)
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) red[warp][(i * NT + j) * 4 + e][lane] = acc[i][j][e];
        if (__syncthreads_or(late)) {
            if (late && lane == 0) atomicExch(status, 10);
            for (int s = used; s < sent; ++s) at_wait(bar + 8 * (s % SLOTS), (s / SLOTS) & 1);
            break;
        }
        if (tid < NT * 128 && ep_m < M && ep_r < a.height) {
            float lo = 0.f, hi = 0.f;
#pragma unroll
            for (int w = 0; w < LS_WARPS; ++w) { lo += red[w][warp][lane]; hi += red[w][NT * 4 + warp][lane]; }
            if (PRO == LF_RMSNORM) {
                float sum = 0.f;
#pragma unroll
                for (int w = 0; w < LS_WARPS; ++w) sum += ssq[w][ep_m];
                const float rstd = 1.0f / sqrtf(sum / (float)K + p.eps);
                lo *= rstd; hi *= rstd;
            }
            if (EPI == LF_SWIGLU) {
                if (unit < a.units) {
                    // the unfused path rounds gate and up to bfloat16 before the activation; so does this one
                    lo = __bfloat162float(__float2bfloat16_rn(lo)); hi = __bfloat162float(__float2bfloat16_rn(hi));
                    const float act = p.relu ? fmaxf(lo, 0.f) : lo * (1.0f / (1.0f + expf(-lo)));
                    ((bf16*)p.out)[(size_t)ep_m * p.I + unit] = __float2bfloat16_rn(act * hi);
                }
            } else if (EPI == LF_ROPE) {
                if (unit < a.units) {
                    const int n_lo = head * p.hd + d, n_hi = n_lo + half;
                    if (p.bias) { lo += load_as_f(p.bias, p.bias_dtype, n_lo); hi += load_as_f(p.bias, p.bias_dtype, n_hi); }
                    // the unfused path rounds the projection to bfloat16 before it rotates; so does this one
                    lo = __bfloat162float(__float2bfloat16_rn(lo)); hi = __bfloat162float(__float2bfloat16_rn(hi));
                    if (head < p.n_q + p.n_kv && p.cos_t) {
                        const float u = lo * ep_cos - hi * ep_sin, v = lo * ep_sin + hi * ep_cos;
                        lo = u; hi = v;
                    }
                    const bf16 o_lo = __float2bfloat16_rn(lo), o_hi = __float2bfloat16_rn(hi);
                    if (head < p.n_q) {
                        bf16* q = (bf16*)p.out + (size_t)ep_m * p.n_q * p.hd + (size_t)head * p.hd;
                        q[d] = o_lo; q[d + half] = o_hi;
                    } else if (p.store && ep_page >= 0) {
                        const bool is_k = head < p.n_q + p.n_kv;
                        const int kvh = head - p.n_q - (is_k ? 0 : p.n_kv);
                        bf16* dst = (is_k ? p.k_pool : p.v_pool) + (((size_t)ep_page * p.n_kv + kvh) * PE_PAGE + (ep_pos % PE_PAGE)) * p.hd;
                        dst[d] = o_lo; dst[d + half] = o_hi;
                    }
                }
            } else {
                const int n_lo = lo_row(group) + ep_r, n_hi = n_lo + a.height;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int n = h ? n_hi : n_lo;
                    if (n >= p.N || (h && !a.pair)) continue;
                    float v = h ? hi : lo;
                    if (p.bias) v += load_as_f(p.bias, p.bias_dtype, n);
                    const size_t o = (size_t)ep_m * p.N + n;
                    if (EPI == LF_STORE_F32) ((float*)p.out)[o] = v;
                    else if (EPI == LF_STORE_BF16) ((bf16*)p.out)[o] = __float2bfloat16_rn(v);
                    else atomicAdd((float*)p.out + o, p.out_scale * v);     // the only sum into this element: a reduction in memory, no read to wait for
                }
            }
        }
        __syncthreads();                                    // the sums have been read
    }
}

template <int NT, int PRO, int EPI, int SLOTS>
static int ls_launch_nt(const CUtensorMap& map, const CUtensorMap& map_a, const LsArgs& a, int* status, cudaStream_t s) {
    auto kernel = linear_stream_kernel<NT, PRO, EPI, SLOTS>;
    const size_t smem = 1024 + ls_ring_bytes<NT, PRO, SLOTS>() + (PRO == LF_RMSNORM ? (size_t)NT * 8 * (a.f.K + 8) * 2 : 0);
    PE_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    PE_TRY(pe_launch(kernel, dim3(a.groups < 148 ? a.groups : 148), 32 * LS_WARPS, smem, s, map, map_a, a, status));
    PE_LAUNCH_CHECK();
    return 0;
}

// Which products come here: by what they are and by N and K alone, so that a row's sums are the same in every step.  Measured on a B200, weights
// from memory, us at 1, 8 and 16 rows, linear_fused.cu's kernel / here:
//   normed rows        gate/up 16384 x 2048   25.1 28.3 34.4 / 15.1 15.6 17.6    q/k/v 3072 x 2048   7.3 7.7 9.9 / 5.2 5.6 7.3
//                      gate/up  9728 x 1536    9.6 10.2 13.5 /  9.8 10.2 11.6    q/k/v 1152 x 896    3.7 3.8 4.9 / 3.5 3.7 4.5
//                      gate/up  9728 x 896     5.7  6.2  8.4 /  7.6  7.8  9.0    1152 x 512 stored   3.4 3.4 3.6 / 2.9 3.0 3.8
//                      100 x 2080 stored       3.5  3.9  4.9 /  4.8  5.5  7.5    (few rows: there K is cut over a cluster)
//   bfloat16 rows      2048 x 8192  12.9 12.2 19.2 / 9.0 9.2 11.8                3584 x 3584         7.8 7.6 9.9 / 6.6 6.8 8.1
//                      1536 x 8960  13.2 12.9 21.0 / 9.3 9.5 12.5                896 x 4864          6.0 5.6 7.8 / 5.9 6.1 7.3
//                      5120 x 5120  12.9 13.1 16.5 / 13.4 13.8 17.7              18944 x 1536        20.2 19.2 21.7 / 12.1 12.2 13.7
//                      gate/up 9728 x 1536  7.8 7.8 8.9 / 8.9 8.9 10.5           gate/up 16384 x 2048  20.0 19.8 22.3 / 13.5 14.0 16.5
// and of more than 100 MB, the library's product with the passes around it / here: gate/up 37888 x 3584 51.9 52.3 52.6 / 44.0 45.4 49.8,
// 3584 x 18944 30.4 30.9 30.9 / 22.9 23.2 30.9.
// The lines of the rule lie where a grid of 152 shapes changes sides: normed rows, 33 rows of W a CTA or more (a second group of few rows keeps
// too little under way), 6144 x 512 5.1 6.1 4.4 / 5.0 5.2 6.1, x 768 6.5 7.6 6.1 / 6.5 6.7 7.7, x 1024 7.6 8.8 7.3 / 7.3 7.4 8.4, x 3072 16.0 17.1 18.4 /
// 15.7 16.4 18.4; fewer rows a CTA win from 1024 x 512 (3.2 3.6 3.8 / 2.6 2.7 3.5) to 4608 x 1024 (6.9 8.2 6.7 / 4.2 4.3 5.2).  bfloat16 rows: gate/up 4736 x 1024
// 2.8 3.5 3.8 / 3.5 3.4 3.7, 2368 x 2048 3.9 4.0 4.9 / 4.6 4.5 5.2, 4736 x 1536 5.3 5.1 6.1 / 4.6 4.5 5.1; stored, 1280 x 512 2.6 2.3 2.5 / 1.8 1.7 1.8 to 4736 x 512
// 3.1 3.2 3.0 / 2.3 2.3 2.4.  Taken although one row is slower: 4736 x 1024 2.9 3.0 4.3 / 3.5 3.4 3.7, 9500 x 512 3.7 3.7 5.7 / 4.5 4.4 5.0.
static bool ls_takes(const LfArgs& p, bool norm, int epi) {
    const bool pairs = epi == LF_SWIGLU || epi == LF_ROPE;
    const long long entries = (long long)p.N * p.K;
    if (p.K < 512 || (norm && p.K > 4096) || (epi == LF_ROPE && p.hd % 8)) return false;
    const int rows = ((pairs ? p.N / 2 : p.N) + 147) / 148 * (pairs ? 2 : 1);      // of W, a CTA: up to 32 are one group
    if (epi == LF_SWIGLU) return norm ? p.K >= 1024 || rows <= 32 : entries >= 25000000 || (rows <= 32 && entries >= 6000000);
    if (norm) return p.N >= 1024 && (rows <= 32 || p.K >= 1024);
    return rows >= 9 && (rows <= 32 || rows >= 64);        // (two groups of few rows keep too little under way)
}

template <int PRO, int EPI>
static int ls_launch(const LfArgs& f, int* status, cudaStream_t s) {
    LsArgs a = {};
    a.f = f;
    a.pair = 1;
    a.units = EPI == LF_SWIGLU ? f.I : EPI == LF_ROPE ? f.N / 2 : f.N;
    if (EPI == LF_ROPE) {
        a.height = 16;                                       // whole boxes of a head's half, 48 CTAs and more
        while (a.height > 4 && ((f.hd / 2) % a.height || a.units / a.height < 48)) a.height /= 2;
        if ((f.hd / 2) % a.height) return PE_ERR_UNSUPPORTED;
    } else {
        const int boxes = EPI == LF_SWIGLU ? 1 : 2;          // boxes a group's units fill
        long long least = -1;
        for (int h = 16; h >= 7; --h) {
            const long long groups = (a.units + boxes * h - 1) / (boxes * h), rows = (groups + 147) / 148 * h * boxes;
            if (least < 0 || rows < least) { least = rows; a.height = h; }
        }
        if (EPI != LF_SWIGLU && (a.units + 147) / 148 <= 16) { a.pair = 0; a.height = (a.units + 147) / 148; }
    }
    const int per_group = a.height * (EPI == LF_SWIGLU || EPI == LF_ROPE || !a.pair ? 1 : 2);
    a.groups = (a.units + per_group - 1) / per_group;
    at_encode_fn enc = at_encoder();
    if (!enc) return PE_ERR_UNSUPPORTED;
    const auto boxes_of = [&](CUtensorMap* map, const bf16* base, int rows, int height) {      // boxes of 64 columns; what lies outside reads as zero
        const cuuint64_t dims[2] = {(cuuint64_t)f.K, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)f.K * 2};
        const cuuint32_t box[2] = {64, (cuuint32_t)height}, elem[2] = {1, 1};
        const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        return r == CUDA_SUCCESS ? 0 : 20000 + (int)r;
    };
    CUtensorMap map = {}, map_a = {};
    if (const int e = boxes_of(&map, f.W, f.N, a.height)) return e;
    if (PRO == LF_PLAIN)
        if (const int e = boxes_of(&map_a, f.A, f.M, f.M <= 8 ? 8 : 16)) return e;
    constexpr int SLOTS = PRO == LF_RMSNORM ? 3 : 4;
    if (f.M <= 8) return ls_launch_nt<1, PRO, EPI, SLOTS>(map, map_a, a, status, s);
    if (PRO == LF_RMSNORM && f.K > 3584) return ls_launch_nt<2, PRO, EPI, 2>(map, map_a, a, status, s);      // (16 longer rows leave room for two)
    return ls_launch_nt<2, PRO, EPI, SLOTS>(map, map_a, a, status, s);
}
