// Attention of prompts over low-rank rows on the 5th-generation tensor cores: one key head whose rows [rank | rotated part] all query
// heads read, and whose first `rank` entries are also the value (latent_ops.cu makes queries and rows).  Both products of flash
// attention run as tcgen05.mma with their accumulators in tensor memory.
//
//   one CTA   = a run of up to 128 consecutive tokens of one sequence x one query head
//   a step    = two pages of the cache (128 keys); a page's rows are in shared memory once and serve as keys (K-major) and, their first
//               64-column panels, as values (MN-major)
//   warp 0      loader: TMA tiled loads (128-byte swizzle) of the run's queries and of the pages' rows into a ring of two stages; it
//               alone reads the page table and tells the others through flags which pages are there
//   warp 1      allocates tensor memory; an elected thread issues S = Q K^T (128 x 128) into one of two buffers and O += P V: S of the next step
//               before P V of this one
//   warps 2-9   softmax, two threads a query row, one for each page of the step.  P goes as bfloat16 back into the S buffer's own
//               columns, from where it is the A operand of P V: with queries of 64 KB and two stages of 64 KB there is no room for it
//               in shared memory.  O is rescaled only when a row's reference point has moved by more than 2^8.
//
// Rows of up to 256 entries, a multiple of 16, values of 64, 128 or 192 of them.  At 16 heads of 192 + 64 a step is 1,024 tensor-core
// cycles for Q K^T and 768 for P V against 1,024 of the special-function units for its exponentials: the tensor core bounds it.
// Measured on a B200, 2,048 tokens, 16 heads of 192 + 64: 40 us (45 before the first loads went out ahead of the block's meeting, the mask
// became one comparison a score, sums took two numbers at a time and rows left through shared memory), where the mma.sync kernel (attention_headmix_flash.cu) takes 667.
// A head's gate is one number a token and commutes with the product behind this kernel: it joins the division by the row's sum.
// Every mbarrier wait is bounded by the clock; a wait that runs out sets *status to 5, the roles leave their loops, tensor memory is
// freed and the CTA returns (status 6: shared memory did not start on a 1024-byte boundary, nothing was done).
#include "tcgen05_attention.cuh"

#define LT_QTILE 128
#define LT_KTILE PE_PAGE
#define LT_STAGES 2
#define LT_THREADS 320                             // loader, MMA issuer, and two softmax warps for each 32 rows
#define LT_PANEL (2 * LT_KTILE * 128)              // 128 rows of 64 columns: one swizzled panel, of the queries or of a step's keys
#define LT_BAR_WORDS (13 + 2 * LT_STAGES)
#define LT_TMEM_COLS 512                           // S (then P) at columns 0 and 128, O from column 256
#define LT_O_COL 256
#define LT_LAZY 8.0f
#define LT_USED_BYTES(KP) ((1 + LT_STAGES) * (KP) * LT_PANEL + 8 * LT_BAR_WORDS + 8 * LT_STAGES + 2 * 2 * LT_QTILE * 4)
#define LT_SMEM_BYTES(KP) (LT_USED_BYTES(KP) > 120 * 1024 ? LT_USED_BYTES(KP) : 120 * 1024)     // one CTA an SM: it takes all of tensor memory

struct LatentArgs {
    bf16* out; const int* block_table; int table_stride; const int4* tiles;
    int H, width, rank, window; float scale_log2e;
    int pool_rows;                                 // rows of the pool seen as a matrix [rows][width]
    const bf16* gate; int gate_ld;                 // null, or: head h of token t leaves times sigmoid(gate[t * gate_ld + h])
};

// tiles[i] = (batch row, first packed token, number of tokens (<= 128), position of the first token); KP: 64-column panels of a row
template <int KP>
__global__ void __launch_bounds__(LT_THREADS, 1) attention_latent_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q,
                                                                                 const __grid_constant__ CUtensorMap map_k,
                                                                                 const LatentArgs p, int* status) {
    extern __shared__ __align__(1024) unsigned char lt_mem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int STAGE = KP * LT_PANEL;
    const unsigned q_s = at_smem(lt_mem), kv_s = q_s + KP * LT_PANEL;
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(lt_mem + (1 + LT_STAGES) * STAGE);
    unsigned long long &q_full = bars[0];
    unsigned long long *p_full = bars + 2, *pv_done = bars + 4, *s_full = bars + 6, *kv_full = bars + 8, *kv_empty = bars + 8 + LT_STAGES;
    unsigned long long* pair_bar = bars + 8 + 2 * LT_STAGES;       // one for the two softmax warps of each 32 rows
    unsigned& tmem_base_s = *reinterpret_cast<unsigned*>(bars + 12 + 2 * LT_STAGES);
    volatile unsigned* stage_flags = reinterpret_cast<volatile unsigned*>(bars + LT_BAR_WORDS);   // bit g: page g of the stage exists
    float* exchange = reinterpret_cast<float*>(bars + LT_BAR_WORDS + LT_STAGES);    // [meeting parity][half][row]: what the halves of a row tell each other
    if (q_s & 1023u) {                                              // every thread alike: nothing is allocated yet
        if (threadIdx.x == 0) atomicExch(status, 6);
        return;
    }
    // (the step's description and the page table are inputs like any other: the kernel in front may have written them)
    pdl_wait();
    const int4 info = p.tiles[blockIdx.y];                          // heads vary fastest: the runs that see the most keys start first
    const int brow = info.x, tok0 = info.y, n = info.z, pos0 = info.w, h = blockIdx.x;
    const int first_key = (p.window > 0 && pos0 - p.window + 1 > 0) ? pos0 - p.window + 1 : 0;
    const int page_lo = first_key / LT_KTILE, page_hi = (pos0 + n - 1) / LT_KTILE;
    const int n_pages = page_hi - page_lo + 1, n_steps = (n_pages + 1) / 2;
    const int* table = p.block_table + (size_t)brow * p.table_stride;
    auto bring = [&](int s, const int (&page)[2]) {                  // a stage: two pages
        const unsigned bar = at_smem(&kv_full[s]), dst = kv_s + s * STAGE;
        stage_flags[s] = (page[0] >= 0 ? 1u : 0u) | (page[1] >= 0 ? 2u : 0u);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((unsigned)STAGE) : "memory");
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            // a page that is not there is read from beyond the pool's end, which gives zeros: its scores are masked and its
            // values add nothing; so are a row's entries behind its width (the queries hold the next head's there)
            const int y = page[g] >= 0 ? page[g] * LT_KTILE : p.pool_rows;
#pragma unroll
            for (int c = 0; c < KP; ++c) at_tma_2d(dst + c * LT_PANEL + g * (LT_KTILE * 128), &map_k, 64 * c, y, bar);
        }
    };
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(at_smem(&q_full)) : "memory");
        for (int q = 0; q < 4; ++q) asm volatile("mbarrier.init.shared::cta.b64 [%0], 2;" ::"r"(at_smem(&pair_bar[q])) : "memory");
        for (int s = 0; s < LT_STAGES; ++s) {
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
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(at_smem(&q_full)), "r"((unsigned)STAGE) : "memory");
#pragma unroll
        for (int c = 0; c < KP; ++c) at_tma_2d(q_s + c * LT_PANEL, &map_q, h * p.width + 64 * c, tok0, at_smem(&q_full));
        bring(0, first);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(at_smem(&tmem_base_s)), "r"((unsigned)LT_TMEM_COLS) : "memory");
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
            for (int it = 1; it < n_steps; ++it) {
                const int s = it % LT_STAGES;
                int next[2] = {-1, -1};                             // the step after this one: its entries travel during the wait
                if (2 * it + 2 < n_pages) next[0] = table[page_lo + 2 * it + 2];
                if (2 * it + 3 < n_pages) next[1] = table[page_lo + 2 * it + 3];
                if (it >= LT_STAGES && !at_wait(at_smem(&kv_empty[s]), (unsigned)((it / LT_STAGES) - 1) & 1u)) { atomicExch(status, 5); break; }
                bring(s, page);
                page[0] = next[0]; page[1] = next[1];
            }
        }
    } else if (warp == 1) {
        {                                                           // ---------------- MMA issuer: the warp waits, one thread issues
            const unsigned elected = pe_elect();
            // instruction descriptors: float32 accumulator, bfloat16 operands, M = 128; S: A and B K-major, N = 128 keys;
            // O: A from tensor memory, B MN-major (bit 16), N = rank
            const unsigned idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)((2 * LT_KTILE) >> 3) << 17) | ((unsigned)(LT_QTILE >> 4) << 24);
            const unsigned idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((unsigned)(p.rank >> 3) << 17) | ((unsigned)(LT_QTILE >> 4) << 24);
            const unsigned long long dq = at_desc(q_s, 0, 1024), dk = at_desc(kv_s, 0, 1024), dv = at_desc(kv_s, LT_PANEL, 1024);
            const int k_steps = p.width / 16;
            bool ok = at_wait_warp(at_smem(&q_full), 0u);
            auto issue_s = [&](int it) -> bool {                    // S of step `it` into buffer it & 1, when P V has read the P that lay there
                const int s = it % LT_STAGES, b = it & 1;
                if (it >= 2 && !at_wait_warp(at_smem(&pv_done[b]), (unsigned)((it >> 1) - 1) & 1u)) return false;
                if (!at_wait_warp(at_smem(&kv_full[s]), (unsigned)(it / LT_STAGES) & 1u)) return false;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned long long dks = dk + (unsigned long long)(s * (STAGE >> 4));
                for (int kk = 0; kk < k_steps; ++kk) {              // 16 columns = 32 bytes inside the swizzle atom; 64 columns = one panel
                    const unsigned off = ((kk / 4) * LT_PANEL + (kk % 4) * 32) >> 4;
                    at_mma(elected, tmem + b * (2 * LT_KTILE), dq + off, dks + off, idesc_s, kk > 0 ? 1u : 0u);
                }
                at_commit_by(elected, at_smem(&s_full[b]));
                return true;
            };
            if (ok) ok = issue_s(0);
            for (int it = 0; it < n_steps && ok; ++it) {
                if (it + 1 < n_steps && !issue_s(it + 1)) { ok = false; break; }
                const int s = it % LT_STAGES, b = it & 1;
                if (!at_wait_warp(at_smem(&p_full[b]), (unsigned)(it >> 1) & 1u)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned long long dvs = dv + (unsigned long long)(s * (STAGE >> 4));
#pragma unroll
                for (int kk = 0; kk < 2 * LT_KTILE / 16; ++kk)      // 16 keys: 8 columns further in P, 16 rows further in the panels
                    at_mma_ts(elected, tmem + LT_O_COL, tmem + b * (2 * LT_KTILE) + kk * 8, dvs + ((kk * 16 * 128) >> 4), idesc_o, (it > 0 || kk > 0) ? 1u : 0u);
                at_commit_by(elected, at_smem(&kv_empty[s]));   // the stage's rows have been read
                at_commit_by(elected, at_smem(&pv_done[b]));   // and O holds this step's share
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
        const int half = p.rank / 2;
        const unsigned o_addr = lane_addr + LT_O_COL + g * half;
        const unsigned pair = at_smem(&pair_bar[quarter]);
        const unsigned long long scale2 = at_two(p.scale_log2e, p.scale_log2e);
        float m_run = -INFINITY, l_run = 0.f;
        bool ok = true;
        int it = 0, met = 0;                                        // met: how often the row's two threads have met
        auto swap = [&](float mine, float& theirs) -> bool {        // tell the other half `mine`, learn what it tells
            float* slot = exchange + (met & 1) * (2 * LT_QTILE);
            slot[g * LT_QTILE + r] = mine;
            __syncwarp();
            if (lane == 0) at_arrive(pair);
            if (!at_wait_warp(pair, (unsigned)met & 1u)) return false;
            theirs = slot[(g ^ 1) * LT_QTILE + r];
            ++met;
            return true;
        };
        for (; it < n_steps; ++it) {
            const int b = it & 1, st = it % LT_STAGES;
            if (!at_wait_warp(at_smem(&s_full[b]), (unsigned)(it >> 1) & 1u)) { ok = false; break; }
            // (S of the step exists, so its rows have landed; the flags were written before they were asked for)
            if (!at_wait_warp(at_smem(&kv_full[st]), (unsigned)(it / LT_STAGES) & 1u)) { ok = false; break; }
            const bool there = (stage_flags[st] >> g) & 1u;
            // (S of the last step exists: its rows are read as values only from here on)
            if (it + 1 == n_steps) at_clear_rows(kv_s + st * STAGE, p.rank / 64, LT_PANEL, pos0 + n - (page_lo + 2 * it) * LT_KTILE, threadIdx.x - 64, LT_THREADS - 64);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int key0 = (page_lo + 2 * it + g) * LT_KTILE;
            unsigned raw[LT_KTILE];
            at_ld32_start(lane_addr + b * (2 * LT_KTILE) + g * LT_KTILE, raw);
            at_ld32_start(lane_addr + b * (2 * LT_KTILE) + g * LT_KTILE + 32, raw + 32);
            at_ld_wait();
            at_pin32(raw); at_pin32(raw + 32);
            // the row sees the keys up to its own position and inside its window
            float s[LT_KTILE];
#pragma unroll
            for (int c = 0; c < LT_KTILE; ++c) s[c] = __uint_as_float(raw[c]);
            const int hi = there ? p_r - key0 : -1;                 // the last of the page's keys that the row sees
            if (p.window <= 0) {
                if (hi < LT_KTILE - 1) at_mask_behind<LT_KTILE>(s, hi);
            } else if (const int lo = p_r - p.window + 1 - key0; hi < LT_KTILE - 1 || lo > 0) {      // lo: the window's first one
#pragma unroll
                for (int c = 0; c < LT_KTILE; ++c)
                    if (c > hi || c < lo) s[c] = -INFINITY;
            }
            float mx[4] = {s[0], s[1], s[2], s[3]};                 // four chains: a warp has little else to hide their latency
#pragma unroll
            for (int c = 4; c < LT_KTILE; ++c) mx[c & 3] = fmaxf(mx[c & 3], s[c]);
            const float m_mine = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            float m_theirs;
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            if (!swap(m_mine, m_theirs)) { ok = false; break; }     // (after this the other half has read its scores too: their columns take P)
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // The reference point of the exponentials follows the row's maximum only when that has grown by more than LT_LAZY (in powers
            // of two).  Both threads of a row compute the same from the same numbers.
            const float m_tile = fmaxf(m_mine, m_theirs) * p.scale_log2e;
            const float m_new = (m_run != -INFINITY && m_tile <= m_run + LT_LAZY) ? m_run : fmaxf(m_run, m_tile);
            const float m_use = m_new == -INFINITY ? 0.f : m_new;
            const float alpha = m_run == -INFINITY ? 1.0f : at_exp2(m_run - m_use);
            m_run = m_new;
            unsigned long long sum[2] = {0ull, 0ull};
            const unsigned long long off = at_two(-m_use, -m_use);
            float packed[LT_KTILE / 2];
#pragma unroll
            for (int c = 0; c < LT_KTILE; c += 2) packed[c >> 1] = __uint_as_float(at_exp2_pair(s[c], s[c + 1], scale2, off, sum[(c >> 1) & 1]));
            l_run = l_run * alpha + at_sum_four(sum[0], sum[1]);
            at_st32(lane_addr + b * (2 * LT_KTILE) + g * (LT_KTILE / 2), packed);
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
            const float l = g == 0 ? l_run + l_theirs : l_theirs + l_run;   // the same sum in both threads
            float inv = l > 0.f ? 1.0f / l : 0.f;
            if (p.gate && r < n) inv *= 1.0f / (1.0f + expf(-to_f(p.gate[(size_t)(tok0 + r) * p.gate_ld + h])));
            // through the queries' place (the last products have read them), 32 columns at a time
            const int row_bytes = p.rank * 2, group0 = g * (half / 8);
            bf16* out = p.out + ((size_t)tok0 * p.H + h) * p.rank + g * half;
#pragma unroll 1
            for (int c = 0; c < half; c += 32) {
                float o[32];
                unsigned packed[16];
                at_ld32(o_addr + c, o);
#pragma unroll
                for (int i = 0; i < 16; ++i) packed[i] = at_pack(o[2 * i] * inv, o[2 * i + 1] * inv);
                at_put_row<32>(q_s, row_bytes, r, group0 + c / 8, packed);
                at_store_rows<32>(q_s, row_bytes, quarter * 32, group0 + c / 8, n, out + c, (size_t)p.H * p.rank, lane);
            }
        }
        if (!ok) atomicExch(status, 5);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((unsigned)LT_TMEM_COLS) : "memory");
    }
}

template <int KP>
static int latent_run(const void* q, int q_stride, const void* pool, long long pool_pages, int n_tiles, int n_tokens, LatentArgs p, int* status, cudaStream_t s) {
    CUtensorMap mq, mk;
    int rc = at_make_map(&mq, q, n_tokens, (long long)p.H * p.width, q_stride, LT_QTILE);
    if (rc) return rc;
    rc = at_make_map(&mk, pool, pool_pages * LT_KTILE, p.width, p.width, LT_KTILE);
    if (rc) return rc;
    PE_TRY(cudaFuncSetAttribute(attention_latent_tcgen05_kernel<KP>, cudaFuncAttributeMaxDynamicSharedMemorySize, LT_SMEM_BYTES(KP)));
    PE_TRY(pe_launch(attention_latent_tcgen05_kernel<KP>, dim3(p.H, n_tiles), LT_THREADS, LT_SMEM_BYTES(KP), s, mq, mk, p, status));
    PE_LAUNCH_CHECK();
    return 0;
}

// Whether the kernel takes these sizes.
extern "C" int pe_attention_latent_tcgen05_takes(int width, int rank) {
    return width % 16 == 0 && width <= 256 && rank % 64 == 0 && rank > 0 && rank <= 192 && rank <= width;
}

// q: [n_tokens][q_stride] with head h at columns h * width; pool: [pool_pages][1][64][width]; out [n_tokens][H * rank];
// gate: null, or a logit a head at gate[t * gate_ld + h]
extern "C" int pe_attention_latent_tcgen05(const void* q, int q_stride, void* out, const void* pool, long long pool_pages, const int* block_table,
                                           int table_stride, const void* tiles, int n_tiles, int n_tokens, int H, int width, int rank,
                                           int window, float scale, const void* gate, int gate_ld, int* status, void* stream) {
    if (n_tiles <= 0) return 0;
    if (!pe_attention_latent_tcgen05_takes(width, rank) || n_tiles > 65535 || q_stride % 8 || !(scale > 0.f) || !status) return PE_ERR_UNSUPPORTED;
    if (((uintptr_t)q | (uintptr_t)pool | (uintptr_t)out | (uintptr_t)tiles) & 15) return PE_ERR_UNSUPPORTED;
    if (pool_pages * LT_KTILE > 0x7fffff00ll) return PE_ERR_UNSUPPORTED;             // TMA coordinates are 32-bit
    const LatentArgs p = {(bf16*)out, block_table, table_stride, (const int4*)tiles, H, width, rank, window, scale * 1.4426950408889634f,
                          (int)(pool_pages * LT_KTILE), (const bf16*)gate, gate_ld};
    cudaStream_t s = (cudaStream_t)stream;
    if (width <= 64) return latent_run<1>(q, q_stride, pool, pool_pages, n_tiles, n_tokens, p, status, s);
    if (width <= 128) return latent_run<2>(q, q_stride, pool, pool_pages, n_tiles, n_tokens, p, status, s);
    if (width <= 192) return latent_run<3>(q, q_stride, pool, pool_pages, n_tiles, n_tokens, p, status, s);
    return latent_run<4>(q, q_stride, pool, pool_pages, n_tiles, n_tokens, p, status, s);
}
