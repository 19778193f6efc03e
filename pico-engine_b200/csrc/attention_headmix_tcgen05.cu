// Attention with mixed heads for prompts on the 5th-generation tensor cores.
//
// The mixing is linear, so it can follow the product with the values:
//     o_h(i) = sum_j (sum_g mix[h, g] p_g(i, j)) v_c(h)(j) = sum_g mix[h, g] O_g,c(h)(i),    O_g,c(i) = sum_j p_g(i, j) v_c(j).
// The first kernel is flash attention whose every head g keeps an output for every key/value head c of a group, both products as
// tcgen05.mma with their accumulators in tensor memory; it divides by the softmax denominator (with exp(sink_g) in it) and leaves O_g,c
// in float32.  The second kernel mixes: a thread has a value column of a key/value head and the heads that read it.
//
//   one CTA   = a run of up to 128 consecutive tokens of one sequence x one query head x a group of value heads
//   a step    = two pages of the cache (128 keys)
//   warp 0      loader: TMA tiled loads (128-byte swizzle) of the run's queries and of the pages' keys and the group's values into a ring
//               of stages; it alone reads the page table and tells the others through flags which pages are there
//   warp 1      allocates tensor memory; an elected thread issues S = Q K^T (128 x 128) into one of two buffers and O_c += P V_c for the group's
//               heads: S of the next step before P V of this one
//   warps 2-9   softmax, two threads a query row, one for each page of the step; P goes as bfloat16 back into the S buffer's own columns,
//               from where it is the A operand of P V.  O is rescaled only when a row's reference point has moved by more than 2^8.
//
// Tensor memory has 256 columns for S and 256 for O: two value heads of 128 or four of 64 a CTA; more are further CTAs, which make S again.
// Bound by a step's chain (scores, maximum, exponentials, P) rather than by the tensor cores.
// Measured on a B200, 1,024 tokens, 16 heads of 128 on four key/value heads: 33 + 6 us (40 + 7 with rows of O stored by their own lanes, 32
// lines an instruction, a chain of comparisons a score and the first loads behind the block's meeting), where the mma.sync kernel and its merge
// (attention_headmix_flash.cu) take 198 + 83.
// Head sizes: D a multiple of 16, Dv of 16.  Every mbarrier wait is bounded by the clock; a wait that runs out sets *status to 5, the
// roles leave their loops, tensor memory is freed and the CTA returns (status 6: shared memory did not start on a 1024-byte boundary).
#include "tcgen05_attention.cuh"

#define HT_QTILE 128
#define HT_KTILE PE_PAGE
#define HT_MAX_STAGES 4
#define HT_THREADS 320                             // loader, MMA issuer, and two softmax warps for each 32 rows
#define HT_PANEL (2 * HT_KTILE * 128)              // 128 rows of 64 columns: one swizzled panel, of the queries or of a step's keys or values
#define HT_BAR_WORDS (13 + 2 * HT_MAX_STAGES)
#define HT_TMEM_COLS 512                           // S (then P) at columns 0 and 128, O of the group's heads from column 256
#define HT_O_COL 256
#define HT_LAZY 8.0f
#define HT_SMALL_BYTES (8 * HT_BAR_WORDS + 8 * HT_MAX_STAGES + 2 * 2 * HT_QTILE * 4)
#define HT_SMEM_LIMIT 232448

struct HeadmixArgs {
    float* o; const int* block_table; int table_stride; const int4* tiles;      // o [tokens][H][G][Dv]
    int H, G, D, Dv, cg, window; float scale_log2e;
    const float* sink;                             // [H] or null
    int qp, vp, stages;                            // 64-column panels of a query (and key) row and of a value row; stages of the ring
    int pool_rows;                                 // rows of the pools seen as matrices [rows][D] and [rows][Dv]
};

// tiles[i] = (batch row, first packed token, number of tokens (<= 128), position of the first token)
__global__ void __launch_bounds__(HT_THREADS, 1) attention_headmix_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q,
                                                                                  const __grid_constant__ CUtensorMap map_k,
                                                                                  const __grid_constant__ CUtensorMap map_v,
                                                                                  const HeadmixArgs p, int* status) {
    extern __shared__ __align__(1024) unsigned char ht_mem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned stage_bytes = (unsigned)(p.qp + p.cg * p.vp) * HT_PANEL;
    const unsigned q_s = at_smem(ht_mem), kv_s = q_s + p.qp * HT_PANEL;
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(ht_mem + (size_t)p.qp * HT_PANEL + (size_t)p.stages * stage_bytes);
    unsigned long long &q_full = bars[0];
    unsigned long long *p_full = bars + 2, *pv_done = bars + 4, *s_full = bars + 6, *kv_full = bars + 8, *kv_empty = bars + 8 + HT_MAX_STAGES;
    unsigned long long* pair_bar = bars + 8 + 2 * HT_MAX_STAGES;   // one for the two softmax warps of each 32 rows
    unsigned& tmem_base_s = *reinterpret_cast<unsigned*>(bars + 12 + 2 * HT_MAX_STAGES);
    volatile unsigned* stage_flags = reinterpret_cast<volatile unsigned*>(bars + HT_BAR_WORDS);   // bit g: page g of the stage exists
    float* exchange = reinterpret_cast<float*>(bars + HT_BAR_WORDS + HT_MAX_STAGES);    // [meeting parity][half][row]: what the halves of a row tell each other
    if (q_s & 1023u) {                                              // every thread alike: nothing is allocated yet
        if (threadIdx.x == 0) atomicExch(status, 6);
        return;
    }
    // (the step's description and the page table are inputs like any other: the kernel in front may have written them)
    pdl_wait();
    const int4 info = p.tiles[blockIdx.y];                          // heads vary fastest: the runs that see the most keys start first
    const int brow = info.x, tok0 = info.y, n = info.z, pos0 = info.w;
    const int groups = p.G / p.cg, h = blockIdx.x / groups, c_lo = blockIdx.x % groups * p.cg, kvh = h / (p.H / p.G);
    const int first_key = (p.window > 0 && pos0 - p.window + 1 > 0) ? pos0 - p.window + 1 : 0;
    const int page_lo = first_key / HT_KTILE, page_hi = (pos0 + n - 1) / HT_KTILE;
    const int n_pages = page_hi - page_lo + 1, n_steps = (n_pages + 1) / 2;
    const int* table = p.block_table + (size_t)brow * p.table_stride;
    auto bring = [&](int s, const int (&page)[2]) {                  // a stage: two pages
        const unsigned bar = at_smem(&kv_full[s]), k_dst = kv_s + s * stage_bytes, v_dst = k_dst + p.qp * HT_PANEL;
        stage_flags[s] = (page[0] >= 0 ? 1u : 0u) | (page[1] >= 0 ? 2u : 0u);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(stage_bytes) : "memory");
        for (int g = 0; g < 2; ++g) {
            // a page that is not there is read from beyond the pool's end, which gives zeros: its scores are masked and its
            // values add nothing; so are a row's entries behind its size (the queries hold the next head's there)
            const unsigned at = g * (HT_KTILE * 128);
            for (int c = 0; c < p.qp; ++c)
                at_tma_2d(k_dst + c * HT_PANEL + at, &map_k, 64 * c, page[g] >= 0 ? (page[g] * p.G + kvh) * HT_KTILE : p.pool_rows, bar);
            for (int v = 0; v < p.cg; ++v)
                for (int c = 0; c < p.vp; ++c)
                    at_tma_2d(v_dst + (v * p.vp + c) * HT_PANEL + at, &map_v, 64 * c,
                              page[g] >= 0 ? (page[g] * p.G + c_lo + v) * HT_KTILE : p.pool_rows, bar);
        }
    };
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(at_smem(&q_full)) : "memory");
        for (int q = 0; q < 4; ++q) asm volatile("mbarrier.init.shared::cta.b64 [%0], 2;" ::"r"(at_smem(&pair_bar[q])) : "memory");
        for (int s = 0; s < HT_MAX_STAGES; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(at_smem(&kv_full[s])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(at_smem(&kv_empty[s])) : "memory");
        }
        for (int b = 0; b < 2; ++b) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(at_smem(&s_full[b])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 8;" ::"r"(at_smem(&p_full[b])) : "memory");      // the eight softmax warps
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(at_smem(&pv_done[b])) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n\tfence.proxy.async.shared::cta;" ::: "memory");
        // the queries and the first step are asked for before the block meets
        const int first[2] = {table[page_lo], 1 < n_pages ? table[page_lo + 1] : -1};
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(at_smem(&q_full)), "r"((unsigned)(p.qp * HT_PANEL)) : "memory");
        for (int c = 0; c < p.qp; ++c) at_tma_2d(q_s + c * HT_PANEL, &map_q, h * p.D + 64 * c, tok0, at_smem(&q_full));
        bring(0, first);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(at_smem(&tmem_base_s)), "r"((unsigned)HT_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = tmem_base_s;
    // only now may the next kernel of the stream be scheduled: it could take tensor memory that a CTA of this grid still waits for
    pdl_launch_dependents();

    if (warp == 0) {
        if (lane == 0) {                                            // ---------------- loader
            int page[2] = {2 < n_pages ? table[page_lo + 2] : -1, 3 < n_pages ? table[page_lo + 3] : -1};
            int s = p.stages > 1 ? 1 : 0;
            unsigned round = p.stages > 1 ? 0 : 1;                                     // how often the ring has been filled
            for (int it = 1; it < n_steps; ++it) {
                int next[2] = {-1, -1};                             // the step after this one: its entries travel during the wait
                if (2 * it + 2 < n_pages) next[0] = table[page_lo + 2 * it + 2];
                if (2 * it + 3 < n_pages) next[1] = table[page_lo + 2 * it + 3];
                if (round > 0 && !at_wait(at_smem(&kv_empty[s]), (round - 1) & 1u)) { atomicExch(status, 5); break; }
                bring(s, page);
                page[0] = next[0]; page[1] = next[1];
                if (++s == p.stages) { s = 0; ++round; }
            }
        }
    } else if (warp == 1) {
        {                                                           // ---------------- MMA issuer: the warp waits, one thread issues
            const unsigned elected = pe_elect();
            // instruction descriptors: float32 accumulator, bfloat16 operands, M = 128; S: A and B K-major, N = 128 keys;
            // O: A from tensor memory, B MN-major (bit 16), N = Dv
            const unsigned idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)((2 * HT_KTILE) >> 3) << 17) | ((unsigned)(HT_QTILE >> 4) << 24);
            const unsigned idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((unsigned)(p.Dv >> 3) << 17) | ((unsigned)(HT_QTILE >> 4) << 24);
            const unsigned long long dq = at_desc(q_s, 0, 1024), dk = at_desc(kv_s, 0, 1024), dv = at_desc(kv_s + p.qp * HT_PANEL, HT_PANEL, 1024);
            const int k_steps = p.D / 16;
            bool ok = at_wait_warp(at_smem(&q_full), 0u);
            int s_next = 0, s_here = 0;                             // the stages of the S issued next and of the P V issued next
            unsigned s_round = 0;
            auto issue_s = [&](int it) -> bool {                    // S of step `it` into buffer it & 1, when P V has read the P that lay there
                const int b = it & 1;
                if (it >= 2 && !at_wait_warp(at_smem(&pv_done[b]), (unsigned)((it >> 1) - 1) & 1u)) return false;
                if (!at_wait_warp(at_smem(&kv_full[s_next]), s_round & 1u)) return false;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned long long dks = dk + (unsigned long long)(s_next * (stage_bytes >> 4));
                for (int kk = 0; kk < k_steps; ++kk) {              // 16 columns = 32 bytes inside the swizzle atom; 64 columns = one panel
                    const unsigned off = ((kk / 4) * HT_PANEL + (kk % 4) * 32) >> 4;
                    at_mma(elected, tmem + b * (2 * HT_KTILE), dq + off, dks + off, idesc_s, kk > 0 ? 1u : 0u);
                }
                at_commit_by(elected, at_smem(&s_full[b]));
                if (++s_next == p.stages) { s_next = 0; ++s_round; }
                return true;
            };
            if (ok) ok = issue_s(0);
            for (int it = 0; it < n_steps && ok; ++it) {
                if (it + 1 < n_steps && !issue_s(it + 1)) { ok = false; break; }
                const int b = it & 1;
                if (!at_wait_warp(at_smem(&p_full[b]), (unsigned)(it >> 1) & 1u)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int v = 0; v < p.cg; ++v) {
                    const unsigned long long dvs = dv + (unsigned long long)(s_here * (stage_bytes >> 4) + v * p.vp * (HT_PANEL >> 4));
#pragma unroll
                    for (int kk = 0; kk < 2 * HT_KTILE / 16; ++kk)  // 16 keys: 8 columns further in P, 16 rows further in the panels
                        at_mma_ts(elected, tmem + HT_O_COL + v * p.Dv, tmem + b * (2 * HT_KTILE) + kk * 8, dvs + ((kk * 16 * 128) >> 4), idesc_o, (it > 0 || kk > 0) ? 1u : 0u);
                }
                at_commit_by(elected, at_smem(&kv_empty[s_here]));   // the stage's keys and values have been read
                at_commit_by(elected, at_smem(&pv_done[b]));   // and O holds this step's share
                if (++s_here == p.stages) s_here = 0;
            }
            if (!ok) atomicExch(status, 5);
        }
    } else {                                                        // ---------------- softmax, warps 2..9
        // Two threads a query row: thread (row, g) has the scores of the step's page g (64 keys) and half of the row of O.  The two tell
        // each other their maxima, and at the end their sums, through shared memory.
        const int quarter = warp & 3;                               // the 32 lanes of tensor memory this warp may touch
        const int g = (warp - 2) >> 2;
        const int r = quarter * 32 + lane, p_r = pos0 + r;          // this thread's query row
        const unsigned lane_addr = tmem + ((unsigned)(quarter * 32) << 16);
        const int half = p.cg * p.Dv / 2;
        const unsigned o_addr = lane_addr + HT_O_COL + g * half;
        const unsigned pair = at_smem(&pair_bar[quarter]);
        const unsigned long long scale2 = at_two(p.scale_log2e, p.scale_log2e);
        float m_run = -INFINITY, l_run = 0.f;
        bool ok = true;
        int it = 0, met = 0, st = 0;                                // met: how often the row's two threads have met; st: the step's stage
        unsigned st_round = 0;
        auto swap = [&](float mine, float& theirs) -> bool {        // tell the other half `mine`, learn what it tells
            float* slot = exchange + (met & 1) * (2 * HT_QTILE);
            slot[g * HT_QTILE + r] = mine;
            __syncwarp();
            if (lane == 0) at_arrive(pair);
            if (!at_wait_warp(pair, (unsigned)met & 1u)) return false;
            theirs = slot[(g ^ 1) * HT_QTILE + r];
            ++met;
            return true;
        };
        for (; it < n_steps; ++it) {
            const int b = it & 1;
            if (!at_wait_warp(at_smem(&s_full[b]), (unsigned)(it >> 1) & 1u)) { ok = false; break; }
            // (S of the step exists, so its rows have landed; the flags were written before they were asked for)
            if (!at_wait_warp(at_smem(&kv_full[st]), st_round & 1u)) { ok = false; break; }
            const bool there = (stage_flags[st] >> g) & 1u;
            if (it + 1 == n_steps)
                at_clear_rows(kv_s + st * stage_bytes + p.qp * HT_PANEL, p.cg * p.vp, HT_PANEL, pos0 + n - (page_lo + 2 * it) * HT_KTILE, threadIdx.x - 64, HT_THREADS - 64);
            if (++st == p.stages) { st = 0; ++st_round; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int key0 = (page_lo + 2 * it + g) * HT_KTILE;
            unsigned raw[HT_KTILE];
            at_ld32_start(lane_addr + b * (2 * HT_KTILE) + g * HT_KTILE, raw);
            at_ld32_start(lane_addr + b * (2 * HT_KTILE) + g * HT_KTILE + 32, raw + 32);
            at_ld_wait();
            at_pin32(raw); at_pin32(raw + 32);
            // the row sees the keys up to its own position and inside its window
            float s[HT_KTILE];
#pragma unroll
            for (int c = 0; c < HT_KTILE; ++c) s[c] = __uint_as_float(raw[c]);
            const int hi = there ? p_r - key0 : -1;                 // the last of the page's keys that the row sees
            if (p.window <= 0) {
                if (hi < HT_KTILE - 1) at_mask_behind<HT_KTILE>(s, hi);
            } else if (const int lo = p_r - p.window + 1 - key0; hi < HT_KTILE - 1 || lo > 0) {      // lo: the window's first one
#pragma unroll
                for (int c = 0; c < HT_KTILE; ++c)
                    if (c > hi || c < lo) s[c] = -INFINITY;
            }
            float mx[4] = {s[0], s[1], s[2], s[3]};                 // four chains: a warp has little else to hide their latency
#pragma unroll
            for (int c = 4; c < HT_KTILE; ++c) mx[c & 3] = fmaxf(mx[c & 3], s[c]);
            const float m_mine = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            float m_theirs;
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            if (!swap(m_mine, m_theirs)) { ok = false; break; }     // (after this the other half has read its scores too: their columns take P)
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // The reference point of the exponentials follows the row's maximum only when that has grown by more than HT_LAZY (in powers
            // of two).  Both threads of a row compute the same from the same numbers.
            const float m_tile = fmaxf(m_mine, m_theirs) * p.scale_log2e;
            const float m_new = (m_run != -INFINITY && m_tile <= m_run + HT_LAZY) ? m_run : fmaxf(m_run, m_tile);
            const float m_use = m_new == -INFINITY ? 0.f : m_new;
            const float alpha = m_run == -INFINITY ? 1.0f : at_exp2(m_run - m_use);
            m_run = m_new;
            unsigned long long sum[2] = {0ull, 0ull};
            const unsigned long long off = at_two(-m_use, -m_use);
            float packed[HT_KTILE / 2];
#pragma unroll
            for (int c = 0; c < HT_KTILE; c += 2) packed[c >> 1] = __uint_as_float(at_exp2_pair(s[c], s[c + 1], scale2, off, sum[(c >> 1) & 1]));
            l_run = l_run * alpha + at_sum_four(sum[0], sum[1]);
            at_st32(lane_addr + b * (2 * HT_KTILE) + g * (HT_KTILE / 2), packed);
            if (it > 0 && __any_sync(0xffffffffu, alpha != 1.0f)) { // a row's reference point moved: rescale this half of the warp's rows of O
                if (!at_wait_warp(at_smem(&pv_done[b ^ 1]), (unsigned)((it - 1) >> 1) & 1u)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
                for (int c = 0; c < half; c += 32) {
                    float o[32];
                    at_ld32(o_addr + c, o);
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] *= alpha;
                    at_st32(o_addr + c, o);
                }
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) at_arrive(at_smem(&p_full[b]));
        }
        // the row's sum, and the last P V (products complete in the order they were issued)
        float l_theirs = 0.f;
        if (ok && !swap(l_run, l_theirs)) ok = false;
        if (ok && it > 0 && !at_wait_warp(at_smem(&pv_done[(it - 1) & 1]), (unsigned)((it - 1) >> 1) & 1u)) ok = false;
        if (ok && it > 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float l = g == 0 ? l_run + l_theirs : l_theirs + l_run;         // the same sum in both threads
            if (p.sink) l += at_exp2(fmaf(p.sink[h], 1.4426950408889634f, -m_run));       // (a row that saw no key: 2^inf, and 1 / l = 0)
            const float inv = l > 0.f ? 1.0f / l : 0.f;
            // the group's heads lie side by side; through the place of the queries and stages (the last products have read them), 4 KB a warp
            const unsigned tile = q_s + (warp - 2) * 4096;
            const size_t row_floats = (size_t)p.H * p.G * p.Dv;
            float* out = p.o + (size_t)(tok0 + quarter * 32) * row_floats + ((size_t)h * p.G + c_lo) * p.Dv + g * half;
#pragma unroll 1
            for (int c = 0; c < half; c += 32) {
                float o[32];
                unsigned bits[32];
                at_ld32(o_addr + c, o);
#pragma unroll
                for (int i = 0; i < 32; ++i) bits[i] = __float_as_uint(o[i] * inv);
                at_put_row<64>(tile, 128, lane, 0, bits);           // 32 numbers of 4 bytes
                at_store_rows<64>(tile, 128, 0, 0, n - quarter * 32, reinterpret_cast<bf16*>(out + c), 2 * row_floats, lane);
                __syncwarp();
            }
        }
        if (!ok) atomicExch(status, 5);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((unsigned)HT_TMEM_COLS) : "memory");
    }
}

// out[t][h][d] = sum_g mix[h, g] o[t][g][c(h)][d].  A thread has four columns of key/value head c and HEADS of the heads that read it
// (blockIdx.y: which): a head's outputs are read once for all of them, neighbouring threads side by side, and no read waits for another.
// The weights of one g lie side by side in shared memory, so that one read serves them all.  Bound by reading o: 7.2 us at
// 1,024 tokens of 16 heads over 4 x 128 columns (34 MB), against 15.1 with a column and eight heads a thread.
#define HT_MIX_HEADS 8                                              // at most
template <int HEADS>
__global__ void __launch_bounds__(256) headmix_mix_kernel(const float* o, const float* mix, bf16* out, int T, int H, int G, int Dv) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) float ht_mix[];                 // [G][H][HEADS]: the weights of this block's heads of every c
    pdl_wait();
    const int per = H / G, cols = G * Dv;
    for (int i = threadIdx.x; i < G * H * HEADS; i += blockDim.x) {
        const int h = blockIdx.y * HEADS + i % HEADS, g = i / HEADS % H, c = i / HEADS / H;
        ht_mix[i] = h < per ? mix[(c * per + h) * H + g] : 0.f;
    }
    __syncthreads();
    const long long e = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (e >= (long long)T * cols) return;
    const int t = (int)(e / cols), col = (int)(e % cols), c = col / Dv, d = col % Dv;
    const float* src = o + (size_t)t * H * cols + col;
    const float* w = ht_mix + c * H * HEADS;
    float4 acc[HEADS];
#pragma unroll
    for (int i = 0; i < HEADS; ++i) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int g = 0; g < H; ++g) {
        const float4 v = *reinterpret_cast<const float4*>(src + (size_t)g * cols);
#pragma unroll
        for (int i = 0; i < HEADS; ++i) {
            const float x = w[g * HEADS + i];
            acc[i].x = fmaf(x, v.x, acc[i].x); acc[i].y = fmaf(x, v.y, acc[i].y); acc[i].z = fmaf(x, v.z, acc[i].z); acc[i].w = fmaf(x, v.w, acc[i].w);
        }
    }
    const int h0 = c * per + blockIdx.y * HEADS, n_h = min(HEADS, per - (int)blockIdx.y * HEADS);
#pragma unroll
    for (int i = 0; i < HEADS; ++i) {
        if (i >= n_h) break;
        uint2 r;
        *reinterpret_cast<__nv_bfloat162*>(&r.x) = __floats2bfloat162_rn(acc[i].x, acc[i].y);
        *reinterpret_cast<__nv_bfloat162*>(&r.y) = __floats2bfloat162_rn(acc[i].z, acc[i].w);
        *reinterpret_cast<uint2*>(out + ((size_t)t * H + h0 + i) * Dv + d) = r;
    }
}

template <int HEADS>
static int ht_mix_launch(const float* o, const float* mix, bf16* out, int T, int H, int G, int Dv, cudaStream_t s) {
    const size_t smem = sizeof(float) * G * H * HEADS;              // HEADS < 2 H / G: less than 128 KB
    if (smem > 48 * 1024) PE_TRY(cudaFuncSetAttribute(headmix_mix_kernel<HEADS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const dim3 grid((unsigned)(((long long)T * G * Dv / 4 + 255) / 256), (H / G + HEADS - 1) / HEADS);
    PE_TRY(pe_launch(headmix_mix_kernel<HEADS>, grid, 256, smem, s, o, mix, out, T, H, G, Dv));
    PE_LAUNCH_CHECK();
    return 0;
}

// How the sizes are laid out: value heads a CTA and stages of the ring; false: not taken.
static bool ht_plan(int H, int G, int D, int Dv, HeadmixArgs& a) {
    if (H < 1 || G < 1 || H % G || H > 128 || D < 16 || D % 16 || D > 256 || Dv < 16 || Dv % 16 || Dv > 256) return false;
    a.qp = (D + 63) / 64;
    a.vp = (Dv + 63) / 64;
    for (int cg = G; cg >= 1; --cg) {
        if (G % cg || cg * Dv > 256 || cg * Dv % 64) continue;
        const int stage = (a.qp + cg * a.vp) * HT_PANEL;
        int stages = (HT_SMEM_LIMIT - HT_SMALL_BYTES - a.qp * HT_PANEL) / stage;
        if (stages > HT_MAX_STAGES) stages = HT_MAX_STAGES;
        if (stages < 2) continue;                                   // S of a step is made before P V of the step before: two stages at least
        a.cg = cg;
        a.stages = stages;
        return true;
    }
    return false;
}
extern "C" int pe_attention_headmix_tcgen05_takes(int H, int G, int D, int Dv) {
    HeadmixArgs a;
    return ht_plan(H, G, D, Dv, a) ? 1 : 0;
}

// q: [T][q_stride] with head h at columns h * D; pools: [pool_pages][G][64][D] and [..][Dv]; scratch: float32 [T][H][G][Dv]; out [T][H * Dv]
extern "C" int pe_attention_headmix_tcgen05(const void* q, int q_stride, void* out, const void* k_pool, const void* v_pool, long long pool_pages,
                                            const int* block_table, int table_stride, const void* tiles, int n_tiles, int T, int H, int G, int D,
                                            int Dv, int window, float scale, const float* sink, const float* mix, float* scratch, int* status, void* stream) {
    if (n_tiles <= 0) return 0;
    HeadmixArgs a = {scratch, block_table, table_stride, (const int4*)tiles, H, G, D, Dv, 0, window, scale * 1.4426950408889634f, sink, 0, 0, 0,
                     (int)(pool_pages * G * HT_KTILE)};
    if (!ht_plan(H, G, D, Dv, a) || n_tiles > 65535 || q_stride % 8 || !(scale > 0.f) || !status || !mix) return PE_ERR_UNSUPPORTED;
    if (((uintptr_t)q | (uintptr_t)k_pool | (uintptr_t)v_pool | (uintptr_t)tiles | (uintptr_t)scratch) & 15) return PE_ERR_UNSUPPORTED;
    if (pool_pages * G * HT_KTILE > 0x7fffff00ll) return PE_ERR_UNSUPPORTED;         // TMA coordinates are 32-bit
    CUtensorMap mq, mk, mv;
    int rc = at_make_map(&mq, q, T, (long long)H * D, q_stride, HT_QTILE);
    if (rc) return rc;
    rc = at_make_map(&mk, k_pool, pool_pages * G * HT_KTILE, D, D, HT_KTILE);
    if (rc) return rc;
    rc = at_make_map(&mv, v_pool, pool_pages * G * HT_KTILE, Dv, Dv, HT_KTILE);
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    size_t smem = (size_t)a.qp * HT_PANEL + (size_t)a.stages * (a.qp + a.cg * a.vp) * HT_PANEL + HT_SMALL_BYTES;
    if (smem < 120 * 1024) smem = 120 * 1024;                       // one CTA an SM: it takes all of tensor memory
    PE_TRY(cudaFuncSetAttribute(attention_headmix_tcgen05_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, HT_SMEM_LIMIT));
    PE_TRY(pe_launch(attention_headmix_tcgen05_kernel, dim3(H * (G / a.cg), n_tiles), HT_THREADS, smem, s, mq, mk, mv, a, status));
    PE_LAUNCH_CHECK();
    const int per = H / G;
    const auto launch = per == 1 ? ht_mix_launch<1> : per == 2 ? ht_mix_launch<2> : per <= 4 ? ht_mix_launch<4> : ht_mix_launch<HT_MIX_HEADS>;
    return launch((const float*)scratch, mix, (bf16*)out, T, H, G, Dv, s);
}
