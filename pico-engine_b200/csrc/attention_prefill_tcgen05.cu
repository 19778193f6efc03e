// Causal attention of many tokens per sequence over the paged bfloat16 cache on the
// 5th-generation tensor cores, for head sizes 64 and 128 (PE_HEAD_DIM): both products of flash
// attention run as tcgen05.mma with their accumulators in tensor memory.
//
//   one CTA   = a run of up to 128 consecutive tokens of one sequence x one query head
//   a step    = two pages of the cache (128 keys): products this small cost the tensor core more in
//               fixed latency than in work, so fewer and larger ones are issued
//   warp 0      loader: TMA tiled loads (cp.async.bulk.tensor.2d, 128-byte swizzle) of the run's
//               queries and, step after step, of the pages' keys and values into a ring
//   warp 1      allocates tensor memory; an elected thread issues S = Q.K^T (128 x 128, K = head size) into
//               one of three S buffers and O += P.V (128 x head size, K = 128 keys); S runs three
//               steps ahead of P.V.  A stage's keys are free for the next ones when S has read them,
//               its values when P.V has
//   warps 2-9   softmax, two warpgroups that take the steps in turn, a thread a query row: tcgen05.ld
//               of its 128 scores, mask, maximum, P = 2^(s - reference) rounded to bfloat16 back into
//               the S buffer's own columns (tcgen05.st), where it is the A operand of P.V, and a row sum
//               in float32 a warpgroup.  From step to step only a row's reference point goes from one
//               warpgroup to the other (through shared memory, before the exponentials), so that one
//               group's waits, loads and maxima lie under the other's exponentials.  When a reference
//               point moves, the row of O in tensor memory is rescaled (tcgen05.ld / tcgen05.st) before P.V.
//
// What bounds a step: its 16,384 exponentials take 1,024 cycles of the special-function units.  With all
// eight warps on one step (two threads a row that told each other their maxima) a step was a chain of
// 2,480 cycles (clock stamps: waits 370, maxima 430, exponentials 1,100, P through shared memory 350);
// with the warpgroups in turn it is 1,430 (head size 64; 1,560 with 128).  Beside the steps a CTA has about 8,000 cycles: barriers, tensor
// memory and the first loads (asked for before the block meets), the first step's chain, the end of the row.  What the softmax
// warps do besides exponentials counts: scale and sums go two numbers at a time (fma / add .f32x2), a page's mask is one comparison
// a score against the last key the row sees, and rows leave through shared memory (at_store_rows).  2,048 tokens, 14 heads of 64,
// on a B200, in a graph of nothing else: 23.8 us with a chain of comparisons a score, single sums and rows stored by their own lanes, 19.3 us here (18.9 if runs and
// page table were read before the kernel in front has ended); 28 heads of 128, prompts of 5,001 / 1,807 / 700 / 33 tokens: 271 us, 228 us here.
//
// Values lie in the cache as [key][head size], which is the MN-major form of the B operand of
// P.V: its shared-memory descriptor steps 8 keys by 1024 bytes and 64 columns by one panel.
// Every mbarrier wait is bounded by the clock; a wait that runs out sets *status to 5, the roles
// leave their loops, tensor memory is freed and the CTA returns.
//
// pico-engine hands this to torch's fused attention after copying keys and values out of the
// cache (src/pico_engine/model.py:201-209).
#ifndef PE_HEAD_DIM
#error "compile with -DPE_HEAD_DIM=<head size>"
#endif
#include "tcgen05_attention.cuh"

#if PE_HEAD_DIM == 64 || PE_HEAD_DIM == 128

#define AT_HD PE_HEAD_DIM
#define AT_QTILE 128
#define AT_KTILE PE_PAGE
#define AT_PANELS (AT_HD / 64)                     // 64-column panels of a row: one 128-byte swizzle atom each
#define AT_STAGES (AT_HD == 64 ? 5 : 3)            // steps in flight or in use; a step is two pages (128 keys)
#define AT_AHEAD 3                                 // steps that S is issued ahead of P.V (no more than stages or S buffers)
#define AT_THREADS 320                             // loader, MMA issuer, and two softmax warpgroups
#define AT_Q_BYTES (AT_QTILE * AT_HD * 2)
#define AT_STAGE_BYTES (2 * 2 * AT_KTILE * AT_HD * 2)   // keys, then values, of two pages and one head
#define AT_TILE_BYTES (AT_Q_BYTES + AT_STAGES * AT_STAGE_BYTES)
#define AT_BUFFERS 3                               // S buffers
#define AT_BAR_WORDS (2 + 3 * AT_BUFFERS + 4 * AT_STAGES + 12)
#define AT_SMEM_BYTES (AT_TILE_BYTES + 8 * AT_BAR_WORDS + 2 * 2 * AT_QTILE * 4)
#define AT_TMEM_COLS 512                           // S buffers (then P) at columns 0, 128 and 256, O from column 384
#define AT_O_COL (AT_BUFFERS * 2 * AT_KTILE)
#define AT_LAZY 8.0f

struct AtArgs {
    bf16* out; const int* block_table; int table_stride; const int4* tiles;
    int nh, nkv, window; float scale_log2e;
    int keep_first;                                // with a window: the first so many keys of a sequence stay visible
    const float* slopes; float inv_scale;          // [nh] or null: slopes[h] * (query position - key position) is taken off the scaled score
    int pool_rows;                                 // rows of the key (and value) pool seen as a matrix [rows][head size]
    const float* sinks;                            // [nh] or null: one more place of this (scaled) score joins a row's denominator and carries no value
};

// tiles[i] = (batch row, first packed token, number of tokens (<= AT_QTILE), position of the first token)
__global__ void __launch_bounds__(AT_THREADS, 1) attention_prefill_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q,
                                                                                  const __grid_constant__ CUtensorMap map_k,
                                                                                  const __grid_constant__ CUtensorMap map_v,
                                                                                  const AtArgs p, int* status) {
    // Q | stages of (K, V of two pages) | barriers | what the warpgroups tell each other.  The tiles need 1024-byte
    // alignment for the swizzle, which the declaration asks for and the kernel checks.
    extern __shared__ __align__(1024) unsigned char at_mem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned q_s = at_smem(at_mem), kv_s = q_s + AT_Q_BYTES;
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(at_mem + AT_TILE_BYTES);
    unsigned long long& q_full = bars[0];
    unsigned& tmem_base_s = *reinterpret_cast<unsigned*>(bars + 1);
    unsigned long long *s_full = bars + 2, *p_full = s_full + AT_BUFFERS, *pv_done = p_full + AT_BUFFERS;
    unsigned long long *k_full = pv_done + AT_BUFFERS, *v_full = k_full + AT_STAGES, *k_empty = v_full + AT_STAGES, *v_empty = k_empty + AT_STAGES;
    unsigned long long* told = v_empty + AT_STAGES;                 // [warpgroup][32 rows]: a step's reference points are there
    unsigned long long* met = told + 8;                             // [32 rows]: both warpgroups have come to the end
    float* refs = reinterpret_cast<float*>(bars + AT_BAR_WORDS);    // [warpgroup][row]: reference point of the group's last step
    float* sums = refs + 2 * AT_QTILE;                              // [warpgroup][row]: at the end, the group's share of the row's sum
    if (q_s & 1023u) {                                              // every thread alike: nothing is allocated yet
        if (threadIdx.x == 0) atomicExch(status, 6);
        return;
    }

    // (the step's description and the page table are inputs like any other: the kernel in front may have written them)
    pdl_wait();
    const int4 info = p.tiles[blockIdx.y];                          // heads vary fastest: the runs that see the most keys start first
    const int brow = info.x, tok0 = info.y, n = info.z, pos0 = info.w;
    const int h = blockIdx.x, kvh = h / (p.nh / p.nkv);
    // the pages the run can see: from the first row's window start to the last row's position, two to a step
    const int first_key = (p.window > 0 && pos0 - p.window + 1 > 0) ? pos0 - p.window + 1 : 0;
    // (with kept first keys: their pages first, then the window's; where the two meet, all pages from the sequence's start)
    int page_lo = first_key / AT_KTILE, kept = 0;
    const int page_hi = (pos0 + n - 1) / AT_KTILE;
    if (p.window > 0 && p.keep_first > 0) {
        const int keep_pages = (p.keep_first + AT_KTILE - 1) / AT_KTILE;
        if (page_lo <= keep_pages) page_lo = 0; else kept = keep_pages;
    }
    const int n_pages = kept + page_hi - page_lo + 1, n_steps = (n_pages + 1) / 2;
    auto page_at = [&](int j) { return j < kept ? j : page_lo + j - kept; };     // the j-th page the run reads, j < n_pages

    const int* table = p.block_table + (size_t)brow * p.table_stride;
    auto bring = [&](const CUtensorMap* map, unsigned dst, const int (&y)[2], unsigned bar) {      // two pages' keys or values of a head
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((unsigned)AT_STAGE_BYTES / 2) : "memory");
#pragma unroll
        for (int g = 0; g < 2; ++g)
#pragma unroll
            for (int c = 0; c < AT_PANELS; ++c) at_tma_2d(dst + c * (2 * AT_KTILE * 128) + g * (AT_KTILE * 128), map, 64 * c, y[g], bar);
    };
    // a page that is not there (beyond the run's last page, or left behind by the window) is read from
    // beyond the pool's end, which gives zeros: its scores are masked and its values add nothing
    auto rows_of = [&](int page) { return page >= 0 ? (page * p.nkv + kvh) * AT_KTILE : p.pool_rows; };
    if (threadIdx.x == 0) {
        auto init = [](unsigned long long* bar, unsigned count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(at_smem(bar)), "r"(count) : "memory"); };
        init(&q_full, 1);
        for (int s = 0; s < AT_STAGES; ++s) { init(&k_full[s], 1); init(&v_full[s], 1); init(&k_empty[s], 1); init(&v_empty[s], 1); }
        for (int b = 0; b < AT_BUFFERS; ++b) { init(&s_full[b], 1); init(&p_full[b], 4); init(&pv_done[b], 1); }     // p_full: a warpgroup's four warps
        for (int w = 0; w < 8; ++w) init(&told[w], 1);
        for (int q = 0; q < 4; ++q) init(&met[q], 2);
        asm volatile("fence.mbarrier_init.release.cluster;\n\tfence.proxy.async.shared::cta;" ::: "memory");
        // the queries and the first step are asked for before the block meets
        const int y[2] = {rows_of(table[page_at(0)]), rows_of(1 < n_pages ? table[page_at(1)] : -1)};
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(at_smem(&q_full)), "r"((unsigned)AT_Q_BYTES) : "memory");
#pragma unroll
        for (int c = 0; c < AT_PANELS; ++c) at_tma_2d(q_s + c * (AT_QTILE * 128), &map_q, h * AT_HD + 64 * c, tok0, at_smem(&q_full));
        bring(&map_k, kv_s, y, at_smem(&k_full[0]));
        bring(&map_v, kv_s + AT_STAGE_BYTES / 2, y, at_smem(&v_full[0]));
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(at_smem(&tmem_base_s)), "r"((unsigned)AT_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = tmem_base_s;
    // Only now may the next kernel of the stream be scheduled: if it came earlier, took tensor memory on this SM
    // and then waited for this grid to end, a CTA of this grid that still had to allocate would wait for it in turn.
    pdl_launch_dependents();

    if (warp == 0) {
        if (lane == 0) {                                            // ---------------- loader
            int page[2] = {2 < n_pages ? table[page_at(2)] : -1, 3 < n_pages ? table[page_at(3)] : -1};
            for (int it = 1; it < n_steps; ++it) {
                const int s = it % AT_STAGES;
                int next[2] = {-1, -1};                             // the step after this one: its entries travel during the wait
                if (2 * it + 2 < n_pages) next[0] = table[page_at(2 * it + 2)];
                if (2 * it + 3 < n_pages) next[1] = table[page_at(2 * it + 3)];
                const unsigned k_dst = kv_s + s * AT_STAGE_BYTES, v_dst = k_dst + AT_STAGE_BYTES / 2, round = (unsigned)((it / AT_STAGES) - 1) & 1u;
                const int y[2] = {rows_of(page[0]), rows_of(page[1])};
                if (it >= AT_STAGES && !at_wait(at_smem(&k_empty[s]), round)) { atomicExch(status, 5); break; }
                bring(&map_k, k_dst, y, at_smem(&k_full[s]));
                if (it >= AT_STAGES && !at_wait(at_smem(&v_empty[s]), round)) { atomicExch(status, 5); break; }
                bring(&map_v, v_dst, y, at_smem(&v_full[s]));
                page[0] = next[0]; page[1] = next[1];
            }
        }
    } else if (warp == 1) {
        {                                                           // ---------------- MMA issuer: the warp waits, one thread issues
            const unsigned elected = pe_elect();
            // instruction descriptors: float32 accumulator, bfloat16 operands, M = 128;
            // S: A and B K-major, N = 128 keys;  O: B MN-major (bit 16), N = head size
            const unsigned idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)((2 * AT_KTILE) >> 3) << 17) | ((unsigned)(AT_QTILE >> 4) << 24);
            const unsigned idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((unsigned)(AT_HD >> 3) << 17) | ((unsigned)(AT_QTILE >> 4) << 24);
            // operand descriptors of stage 0; a stage further on adds its offset in 16-byte units
            const unsigned long long dq = at_desc(q_s, 0, 1024), dk = at_desc(kv_s, 0, 1024);
            const unsigned long long dv = at_desc(kv_s + AT_STAGE_BYTES / 2, 2 * AT_KTILE * 128, 1024);
            bool ok = at_wait_warp(at_smem(&q_full), 0u);
            auto issue_s = [&](int it) -> bool {                    // S = Q . K^T of step `it`, when P.V has read the P that lay in its buffer
                const int s = it % AT_STAGES, b = it % AT_BUFFERS;
                if (it >= AT_BUFFERS && !at_wait_warp(at_smem(&pv_done[b]), (unsigned)(it / AT_BUFFERS - 1) & 1u)) return false;
                if (!at_wait_warp(at_smem(&k_full[s]), (unsigned)(it / AT_STAGES) & 1u)) return false;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned long long dks = dk + (unsigned long long)(s * (AT_STAGE_BYTES >> 4));
#pragma unroll
                for (int kk = 0; kk < AT_HD / 16; ++kk) {           // 16 columns = 32 bytes inside the swizzle atom; 64 columns = one panel
                    const unsigned off_q = ((kk / 4) * (AT_QTILE * 128) + (kk % 4) * 32) >> 4, off_k = ((kk / 4) * (2 * AT_KTILE * 128) + (kk % 4) * 32) >> 4;
                    at_mma(elected, tmem + b * (2 * AT_KTILE), dq + off_q, dks + off_k, idesc_s, kk > 0 ? 1u : 0u);
                }
                at_commit_by(elected, at_smem(&k_empty[s]));   // the stage's keys have been read
                at_commit_by(elected, at_smem(&s_full[b]));
                return true;
            };
            for (int it = 0; it < min(AT_AHEAD, n_steps) && ok; ++it) ok = issue_s(it);
            for (int it = 0; it < n_steps && ok; ++it) {
                const int s = it % AT_STAGES, b = it % AT_BUFFERS;
                if (!at_wait_warp(at_smem(&v_full[s]), (unsigned)(it / AT_STAGES) & 1u)) { ok = false; break; }
                if (!at_wait_warp(at_smem(&p_full[b]), (unsigned)(it / AT_BUFFERS) & 1u)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned long long dvs = dv + (unsigned long long)(s * (AT_STAGE_BYTES >> 4));
#pragma unroll
                for (int kk = 0; kk < 2 * AT_KTILE / 16; ++kk)      // 16 keys: 8 columns further in P, 16 rows further in V
                    at_mma_ts(elected, tmem + AT_O_COL, tmem + b * (2 * AT_KTILE) + kk * 8, dvs + ((kk * 16 * 128) >> 4), idesc_o, (it > 0 || kk > 0) ? 1u : 0u);
                at_commit_by(elected, at_smem(&v_empty[s]));   // the stage's values have been read
                at_commit_by(elected, at_smem(&pv_done[b]));   // and O holds this step's share
                if (it + AT_AHEAD < n_steps && !issue_s(it + AT_AHEAD)) ok = false;
            }
            if (!ok) atomicExch(status, 5);
        }
    } else {                                                        // ---------------- softmax, warps 2..9
        const int quarter = warp & 3;                               // the 32 lanes of tensor memory this warp may touch
        const int g = (warp - 2) >> 2;                              // the warpgroup: steps g, g + 2, ..
        const int r = quarter * 32 + lane;                          // this thread's query row
        const int p_r = pos0 + r;
        const unsigned lane_addr = tmem + ((unsigned)(quarter * 32) << 16);
        const float slope = p.slopes ? p.slopes[h] * p.inv_scale : 0.f;     // in units of the unscaled score
        const unsigned long long scale2 = at_two(p.scale_log2e, p.scale_log2e);
        float m_mine = -INFINITY, l_mine = 0.f;                     // the reference point of this group's last step; its share of the row's sum
        bool ok = true;
        int entry[2];                                               // the page table's entries of the next step of this group
#pragma unroll
        for (int x = 0; x < 2; ++x) entry[x] = 2 * g + x < n_pages ? table[page_at(2 * g + x)] : -1;
        for (int it = g; it < n_steps; it += 2) {
            const int b = it % AT_BUFFERS;
            const unsigned s_addr = lane_addr + b * (2 * AT_KTILE);
            const bool there[2] = {entry[0] >= 0, entry[1] >= 0};   // (a page that is not there was read as zeros and is masked)
#pragma unroll
            for (int x = 0; x < 2; ++x) entry[x] = 2 * it + 4 + x < n_pages ? table[page_at(2 * it + 4 + x)] : -1;
            if (!at_wait_warp(at_smem(&s_full[b]), (unsigned)(it / AT_BUFFERS) & 1u)) { ok = false; break; }
            if (it + 1 == n_steps && (pos0 + n) % AT_KTILE) {       // values behind the run's last token, in the second or the first of the step's pages
                if (!at_wait_warp(at_smem(&v_full[it % AT_STAGES]), (unsigned)(it / AT_STAGES) & 1u)) { ok = false; break; }
                at_clear_rows(kv_s + it % AT_STAGES * AT_STAGE_BYTES + AT_STAGE_BYTES / 2, AT_PANELS, 2 * AT_KTILE * 128,
                              (n_pages - 1 - 2 * it) * AT_KTILE + (pos0 + n) % AT_KTILE, (threadIdx.x - 64) & 127, 128);
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            unsigned raw[2 * AT_KTILE];
#pragma unroll
            for (int c = 0; c < 4; ++c) at_ld32_start(s_addr + 32 * c, raw + 32 * c);
            at_ld_wait();
#pragma unroll
            for (int c = 0; c < 4; ++c) at_pin32(raw + 32 * c);
            // the row sees the keys up to its own position and inside its window
            float s[2 * AT_KTILE], base[2] = {0.f, 0.f}, mx[8];
#pragma unroll
            for (int c = 0; c < 2 * AT_KTILE; ++c) s[c] = __uint_as_float(raw[c]);
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const int key0 = page_at(2 * it + x) * AT_KTILE;
                float* sx = s + x * AT_KTILE;
                const int hi = there[x] ? p_r - key0 : -1;          // the last of the page's keys that the row sees
                if (p.window <= 0) {
                    if (hi < AT_KTILE - 1) at_mask_behind<AT_KTILE>(sx, hi);
                } else if (hi < AT_KTILE - 1 || (key0 <= p_r - p.window && key0 + AT_KTILE - 1 >= p.keep_first)) {
                    const int lo = p_r - p.window + 1 - key0, kept_here = p.keep_first - key0;      // the window's first one, and how many are kept
#pragma unroll
                    for (int c = 0; c < AT_KTILE; ++c)
                        if (c > hi || (c < lo && c >= kept_here)) sx[c] = -INFINITY;
                }
                // the distance's share of the score, slope * (key - row): the part that grows along the page is added here, the
                // page's own part (`base`, one number a page) joins the maximum and the exponent's offset
                if (p.slopes) {
                    base[x] = slope * (float)(key0 - p_r);
#pragma unroll
                    for (int c = 0; c < AT_KTILE; ++c) sx[c] = fmaf(slope, (float)c, sx[c]);
                }
                // four chains a page: a warp has little else to hide their latency
#pragma unroll
                for (int c = 0; c < 4; ++c) mx[4 * x + c] = fmaxf(fmaxf(sx[c], sx[c + 4]), sx[c + 8]);
#pragma unroll
                for (int c = 12; c < AT_KTILE - 4; c += 8) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) mx[4 * x + i] = fmaxf(fmaxf(mx[4 * x + i], sx[c + i]), sx[c + 4 + i]);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) mx[4 * x + i] = fmaxf(mx[4 * x + i], sx[AT_KTILE - 4 + i]);
            }
            const float m_step = fmaxf(fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) + base[0], fmaxf(fmaxf(mx[4], mx[5]), fmaxf(mx[6], mx[7])) + base[1]);
            // the row's reference point up to the step before, from the other warpgroup
            float m_run = -INFINITY;
            if (it > 0) {
                if (!at_wait_warp(at_smem(&told[4 * (g ^ 1) + quarter]), (unsigned)((it - 1) >> 1) & 1u)) { ok = false; break; }
                m_run = refs[(g ^ 1) * AT_QTILE + r];
            }
            // The reference point of the exponentials follows the row's maximum only when that has grown by more than
            // AT_LAZY (in powers of two): P then holds values up to 2^AT_LAZY, which bfloat16 and the float32 sums take
            // as well as values up to 1, and O is rescaled on few steps instead of on nearly all.
            const float m_tile = m_step * p.scale_log2e;
            const float m_new = (m_run != -INFINITY && m_tile <= m_run + AT_LAZY) ? m_run : fmaxf(m_run, m_tile);
            refs[g * AT_QTILE + r] = m_new;
            __syncwarp();
            if (lane == 0) at_arrive(at_smem(&told[4 * g + quarter]));
            const float m_use = m_new == -INFINITY ? 0.f : m_new;
            const float alpha = m_run == -INFINITY ? 1.0f : at_exp2(m_run - m_use);          // for O
            l_mine *= m_mine == -INFINITY ? 1.0f : at_exp2(m_mine - m_use);                  // (no sum yet: it is zero)
            m_mine = m_new;
            unsigned long long sum[2] = {0ull, 0ull};
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                float packed[AT_KTILE / 2];
                const float off = fmaf(base[x], p.scale_log2e, -m_use);
#pragma unroll
                for (int c = 0; c < AT_KTILE; c += 2) packed[c >> 1] = __uint_as_float(at_exp2_pair(s[x * AT_KTILE + c], s[x * AT_KTILE + c + 1], scale2, at_two(off, off), sum[(c >> 1) & 1]));
                at_st32(s_addr + x * (AT_KTILE / 2), packed);       // P over the scores, two keys a column
            }
            l_mine += at_sum_four(sum[0], sum[1]);
            if (it > 0 && __any_sync(0xffffffffu, alpha != 1.0f)) { // a row's reference point moved: rescale the warp's rows of O
                if (!at_wait_warp(at_smem(&pv_done[(it - 1) % AT_BUFFERS]), (unsigned)((it - 1) / AT_BUFFERS) & 1u)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
                for (int c = 0; c < AT_HD; c += 32) {
                    float o[32];
                    at_ld32(lane_addr + AT_O_COL + c, o);
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] *= alpha;
                    at_st32(lane_addr + AT_O_COL + c, o);
                }
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) at_arrive(at_smem(&p_full[b]));
        }
        // the row's sum, in powers of two of the last step's reference point, and the last P.V (products complete in the order they were issued)
        refs[g * AT_QTILE + r] = m_mine;                            // (what stands there already, or, for a group without a step, nothing)
        sums[g * AT_QTILE + r] = l_mine;
        __syncwarp();
        if (lane == 0) at_arrive(at_smem(&met[quarter]));
        const int last = n_steps - 1;
        if (ok && !at_wait_warp(at_smem(&met[quarter]), 0u)) ok = false;
        if (ok && !at_wait_warp(at_smem(&pv_done[last % AT_BUFFERS]), (unsigned)(last / AT_BUFFERS) & 1u)) ok = false;
        if (ok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const float m_run = refs[(last & 1) * AT_QTILE + r];
            float l = 0.f;                                          // the same sum in both threads
#pragma unroll
            for (int w = 0; w < 2; ++w) {
                const float m = refs[w * AT_QTILE + r];
                if (m != -INFINITY) l = fmaf(sums[w * AT_QTILE + r], at_exp2(m - m_run), l);
            }
            if (p.sinks) l += at_exp2(fmaf(p.sinks[h], 1.4426950408889634f, -m_run));   // (a row that saw no key: 2^inf, and 1 / l = 0)
            const float inv = l > 0.f ? 1.0f / l : 0.f;
            // through the queries' place: the last products have read them
            const unsigned o_addr = lane_addr + AT_O_COL + g * (AT_HD / 2);
            constexpr int GROUPS = AT_HD / 16;                      // 16-byte groups of a warpgroup's half of a row
#pragma unroll
            for (int c = 0; c < AT_HD / 2; c += 32) {
                float o[32];
                unsigned packed[16];
                at_ld32(o_addr + c, o);
#pragma unroll
                for (int i = 0; i < 16; ++i) packed[i] = at_pack(o[2 * i] * inv, o[2 * i + 1] * inv);
                at_put_row<32>(q_s, AT_HD * 2, r, g * GROUPS + c / 8, packed);
            }
            at_store_rows<AT_HD / 2>(q_s, AT_HD * 2, quarter * 32, g * GROUPS, n, p.out + ((size_t)tok0 * p.nh + h) * AT_HD + g * (AT_HD / 2), (size_t)p.nh * AT_HD, lane);
        }
        if (!ok) atomicExch(status, 5);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((unsigned)AT_TMEM_COLS) : "memory");
    }
}

extern "C" int pe_attention_prefill_tcgen05_tile() { return AT_QTILE; }

// how many of the kernel's CTAs an SM holds at once (one: it takes all of tensor memory), or a negative CUDA error
extern "C" int pe_attention_prefill_tcgen05_ctas_per_sm() {
    int n = 0;
    if (cudaFuncSetAttribute(attention_prefill_tcgen05_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)AT_SMEM_BYTES) != cudaSuccess) return -1;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, attention_prefill_tcgen05_kernel, AT_THREADS, AT_SMEM_BYTES);
    return e == cudaSuccess ? n : -(int)e;
}

// q: [n_tokens][q_stride] with head h at columns h * hd; pools: [pool_pages][nkv][64][hd]
extern "C" int pe_attention_prefill_tcgen05(const void* q, int q_stride, void* out, const void* k_pool, const void* v_pool,
                                            long long pool_pages, const int* block_table, int table_stride, const void* tiles,
                                            int n_tiles, int n_tokens, int nh, int nkv, int hd, int window, float scale,
                                            int keep_first, const float* slopes, int* status, void* stream, const float* sinks) {
    if (n_tiles <= 0) return 0;
    if (hd != AT_HD || nkv <= 0 || nh % nkv || n_tiles > 65535 || q_stride % 8 || !(scale > 0.f) || !status) return PE_ERR_UNSUPPORTED;
    if (((uintptr_t)q | (uintptr_t)k_pool | (uintptr_t)v_pool | (uintptr_t)out | (uintptr_t)tiles) & 15) return PE_ERR_UNSUPPORTED;
    if (pool_pages * nkv * AT_KTILE > 0x7fffff00ll) return PE_ERR_UNSUPPORTED;       // TMA coordinates are 32-bit
    CUtensorMap mq, mk, mv;
    int rc = at_make_map(&mq, q, n_tokens, (long long)nh * hd, q_stride, AT_QTILE);
    if (rc) return rc;
    rc = at_make_map(&mk, k_pool, pool_pages * nkv * AT_KTILE, hd, hd, AT_KTILE);
    if (rc) return rc;
    rc = at_make_map(&mv, v_pool, pool_pages * nkv * AT_KTILE, hd, hd, AT_KTILE);
    if (rc) return rc;
    AtArgs p = {};
    p.out = (bf16*)out; p.block_table = block_table; p.table_stride = table_stride; p.tiles = (const int4*)tiles;
    p.nh = nh; p.nkv = nkv; p.window = window; p.scale_log2e = scale * 1.4426950408889634f;
    p.keep_first = window > 0 && keep_first > 0 ? keep_first : 0; p.slopes = slopes; p.inv_scale = 1.0f / scale;
    p.pool_rows = (int)(pool_pages * nkv * AT_KTILE);
    p.sinks = sinks;
    const size_t smem = AT_SMEM_BYTES;
    static bool attr_set = false;
    if (!attr_set) {
        PE_TRY(cudaFuncSetAttribute(attention_prefill_tcgen05_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr_set = true;
    }
    PE_TRY(pe_launch(attention_prefill_tcgen05_kernel, dim3(nh, n_tiles), AT_THREADS, smem, (cudaStream_t)stream, mq, mk, mv, p, status));
    return 0;
}

#else   // other head sizes: the mma.sync kernel of attention_prefill.cu takes them

extern "C" int pe_attention_prefill_tcgen05_tile() { return 0; }
extern "C" int pe_attention_prefill_tcgen05_ctas_per_sm() { return 0; }
extern "C" int pe_attention_prefill_tcgen05(const void*, int, void*, const void*, const void*, long long, const int*, int, const void*,
                                            int, int, int, int, int, int, float, int, const float*, int*, void*, const float*) {
    return PE_ERR_UNSUPPORTED;
}

#endif
