// out[M, N] = A[M, K] . W[N, K]^T (+ bias[N]) for float32 operands on the 5th-generation tensor cores, at float32 accuracy.
//
// Every operand is cut in three bfloat16 numbers, x = hi + mid + lo, which together hold its 24 bits.  Six of the nine products of parts are
// multiplied on tcgen05.mma (kind::f16, products exact in float32); mid lo, lo mid and lo lo are left out, of either sign and together at
// most 2^-24 of a product (2^-28 as a root mean square).  The tensor core's sums are not rounded to nearest: addends lose what lies 2^-25
// below the largest, results are cut to 24 bits.  So hi hi, 16 bits a product, is summed over 32 entries of K at a time into an accumulator that
// starts at zero, and these sums are added in registers, in float32 to nearest; the small products, a 256th of it, have an accumulator of
// their own for all of a CTA's K.  The product with a power of two is exact.
// Error against float64, here / a chain of multiply-adds (linear_simt.cu), relative 2-norm, 60 rows of A:
//               3,200 x 256      896 x 896        9,728 x 896      896 x 4,864      3,584 x 3,584    3,584 x 18,944
//   normal      7.3e-8 / 2.0e-7  8.1e-8 / 2.7e-7  1.1e-7 / 3.8e-7  1.1e-7 / 4.4e-7  1.1e-7 / 7.6e-7  2.2e-7 / 1.7e-6
//   positive    6.4e-8 / 1.2e-7  5.2e-8 / 1.1e-7  8.5e-8 / 2.1e-7  6.6e-8 / 1.4e-7  6.2e-8 / 4.2e-7  8.4e-8 / 1.0e-6
//   one term    2.6e-8 / 2.5e-8  2.6e-8 / 2.5e-8  2.6e-8 / 2.5e-8  2.6e-8 / 2.6e-8  2.6e-8 / 2.5e-8  2.6e-8 / 2.5e-8   (largest 1.7 / 1.0 x 2^-24)
//   four terms  2.7e-8 / 4.1e-8  4.2e-8 / 4.5e-8  2.7e-8 / 4.2e-8  4.5e-8 / 4.6e-8  4.4e-8 / 4.2e-8  4.3e-8 / 4.2e-8
// An entry below 2^-110 (7.7e-34) that is not the sum of three bfloat16 numbers is marked by a part that is no number.
//
// K is cut into ranges whose number depends on N and K only, a CTA each; the ranges of a tile are a cluster that adds its sums up in
// their order (up to 64 rows of A each CTA sends the others their rows' sums, and none waits for another to read them: 0.7 to 1.1 us less
// than reading them between two cluster barriers).  How many rows of A a tile has depends on M but changes no sum: a row's result does not depend on the rows beside it.
//
// A CTA: 128 rows of W (the accumulator's lanes) x up to 128 rows of A (its columns).
//   cutting    two groups of four warps, or four, that take the chunks in turn: a thread reads its row of W from the ring in shared memory, cuts it
//              and stores the parts to tensor memory, where the products read them (an operand in shared memory would be read twelve times a
//              chunk); up to 64 rows of A are cut here too and go to shared memory
//   products   a warp issues a chunk's twelve
//   loads      a warp brings W (float32) by TMA, into L2 as far as the ring goes before the kernel waits for its predecessor; more than 64 rows of
//              A have been cut by a kernel before this one and come by TMA as well
//   sums       4 or 16 warps take the sums of hi hi out of tensor memory
// Bound by the hand-overs between them: 508 rows, 9,728 x 896, a chunk of 112 rows of A takes 1,600 cycles, the tensor pipe is busy for a third
// of it, the issue slots for half.  Leaving out two thirds of the products, the cutting or the reading of sums saves 3 to 7 % each.
//
// One B200, W read from memory, us, here / in linear_simt.cu (the only way before): rows of A 1 12 60 130 508
//   1,152 x 896   5.4 / 5.5     5.6 / 7.7    7.9 / 12.2   11.1 / 21.7   24.0 / 34.8
//     896 x 896   5.4 / 5.8     5.6 / 7.6    7.9 / 13.1   10.8 / 25.5   15.4 / 28.0
//   9,728 x 896  13.8 / 12.8   14.1 / 27.2  19.0 / 51.0   44.5 / 84.3   70.5 / 208
//     896 x 4864 10.0 / 11.4   10.2 / 20.4  13.5 / 29.9   20.4 / 64.5   49.6 / 111
//   3,584 x 3584 24.6 / 28.7   25.0 / 50.3  32.3 / 77.3   65.1 / 176.8  133 / 316
//
// Infinities, values that are no number, marked entries and sums beyond float32 leave results that are not finite; those are worked out again with
// plain multiply-adds, a warp a result (one thread a result, down the columns of W, took 812 us where 60 rows meet an infinity in a weight of 9,728 x
// 896, and 30 ms where 508 rows hold no number; 36 us and 2.8 ms so).
//
// Every wait is bounded by the clock; one that runs out sets *status to 9 and a flag that lets every other role leave its loop.  The CTA
// then waits (with a limit again) for the copies and products it has under way, stores nothing, and takes the same steps with its cluster as
// every other CTA: none leaves before all have sent their sums, and the wait for these does not look at the flag, since
// every CTA sends them whatever became of its loops.
//
// pico-engine leaves these products to cuBLAS (src/pico_engine/model.py:177, 213, 223, 235, 164).
#include "tcgen05_attention.cuh"

#define SP_KC 32                                           // entries of K of a chunk: as float32 a row of the 128-byte swizzle, as bfloat16 one of the 64-byte one
#define SP_PARTS 3
#define SP_W_COLS (SP_PARTS * SP_KC / 2)                   // columns of tensor memory of a chunk's parts of W
#define SP_ROWS 128                                        // rows of W of a tile
#define SP_BOX (SP_ROWS * SP_KC * 4)
#define SP_SLOTS 4                                         // chunks at most whose parts are in tensor memory and, of A, in shared memory
#define SP_MANY 128                                        // NT of the form for many rows of A
#define SP_TMEM 512

// W in shared memory, chunks; sums in tensor memory, chunks; warps that take them
template <int NT> constexpr int sp_ring() { return 8; }
template <int NT> constexpr int sp_sums() { return NT == SP_MANY ? 2 : 4; }
template <int NT> constexpr int sp_takers() { return NT == SP_MANY ? 16 : 4; }
// Warps that cut, four a chunk, in turns of two groups or four (few rows of A wait for W to be cut: 12 rows, 3,584 x 3584 27.0 us with two groups, 24.4;
// 60 rows, whose sums take more registers, 31.5 and with three groups 35.2).
template <int NT> constexpr int sp_cutters() { return NT <= 32 ? 16 : 8; }
template <int NT> constexpr int sp_threads() { return 32 * (sp_cutters<NT>() + 2 + sp_takers<NT>()); }
// (few rows of A: a place of its own for the sums that the other CTAs of a cluster send, up to 8 x ceil(NT / 8) rows)
template <int NT> constexpr int sp_sent_bytes() { return NT == SP_MANY ? 0 : (NT + 8) * SP_ROWS * 4; }
// Parts of W, two accumulators of the large products and one of the small ones share 512 columns.
__host__ __device__ constexpr int sp_slots(int nt) { return nt > 112 ? 2 : nt > 96 ? 3 : SP_SLOTS; }
template <int NT> constexpr int sp_smem_bytes() { return sp_ring<NT>() * SP_BOX + (NT == SP_MANY ? SP_SLOTS * 96 : SP_SLOTS * NT) * SP_PARTS * SP_KC * 2 + sp_sent_bytes<NT>() + 1024; }
static_assert(sp_slots(128) * SP_W_COLS + 3 * 128 <= SP_TMEM && sp_slots(112) * SP_W_COLS + 3 * 112 <= SP_TMEM && SP_SLOTS * SP_W_COLS + 3 * 96 <= SP_TMEM &&
              SP_SLOTS * SP_W_COLS + 5 * 64 <= SP_TMEM && sp_slots(128) * 128 <= SP_SLOTS * 96 && sp_slots(112) * 112 <= SP_SLOTS * 96, "room for the parts and the sums");
// A group that waits for a slot's n-th products knows that those before them have ended (or the parity would not tell them apart) from its own
// turn before: groups must not outnumber slots.
static_assert(sp_cutters<SP_MANY>() / 4 <= sp_slots(128) && sp_cutters<64>() / 4 <= SP_SLOTS && sp_cutters<16>() / 4 <= SP_SLOTS, "a slot for every group");

// The status word of products captured into a graph before their device had one (pe_linear_split_gave_up reads it).
static __device__ int sp_gave_up;

// A CTA an SM where few rows of A stream the weights, and ranges of seven chunks at least: what a CTA does once (its first loads, the sum
// over the cluster) takes as long as about six chunks.
static int sp_ranges(int N, int K) {
    const int tiles = (N + SP_ROWS - 1) / SP_ROWS, chunks = (K + SP_KC - 1) / SP_KC;
    int r = 148 / tiles;
    if (r > chunks / 7) r = chunks / 7;
    r = r > 8 ? 8 : r < 1 ? 1 : r;
    const int each = (chunks + r - 1) / r;
    return (chunks + each - 1) / each;                     // (no range without a chunk)
}

__device__ __forceinline__ void sp_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ float4 sp_peer_four(unsigned at, int rank) {
    unsigned peer;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(at), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(peer) : "memory");
    return v;
}
__device__ __forceinline__ float4 sp_shared_four(unsigned at) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ void sp_put_four(unsigned at, const unsigned* v) {
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(at), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
__device__ __forceinline__ void sp_load8(float (&v)[8], const float* p) {
    asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "l"(p) : "memory");
}
__device__ __forceinline__ unsigned long long sp_pair(unsigned a, unsigned b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b));
    return r;
}
// Two neighbouring entries as their parts (of an infinity or no number, parts that are no numbers are left).
__device__ __forceinline__ void sp_cut(float x, float y, unsigned& hi, unsigned& mid, unsigned& lo) {
    unsigned long long rest = at_two(x, y);
    const unsigned long long minus = at_two(-1.f, -1.f);
    hi = at_pack(x, y);
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(rest) : "l"(sp_pair(hi << 16, hi & 0xffff0000u)), "l"(minus));      // (exact)
    float2 r = at_both(rest);
    mid = at_pack(r.x, r.y);
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(rest) : "l"(sp_pair(mid << 16, mid & 0xffff0000u)), "l"(minus));
    r = at_both(rest);
    lo = at_pack(r.x, r.y);
}
// Entries below this may not be the sum of three bfloat16 numbers (the last would lie below 2^-133).
#define SP_SMALL 0x1p-110f
// The first parts of a pair in which an entry that its parts are not the sum of is marked by one that is no number, so that its results are
// not finite and are worked out again with multiply-adds.
__device__ __noinline__ unsigned sp_marked(float x, float y) {
    unsigned hi, mid, lo;
    sp_cut(x, y, hi, mid, lo);
    const float a = (__uint_as_float(hi << 16) + __uint_as_float(mid << 16)) + __uint_as_float(lo << 16);
    const float b = (__uint_as_float(hi & 0xffff0000u) + __uint_as_float(mid & 0xffff0000u)) + __uint_as_float(lo & 0xffff0000u);
    return (a == x ? hi & 0xffffu : 0x7fffu) | (b == y ? hi & 0xffff0000u : 0x7fff0000u);
}
__device__ __forceinline__ void sp_least(float& least, float x, float y) { asm("min.abs.f32 %0, %0, %1, %2;" : "+f"(least) : "f"(x), "f"(y)); }
// operand descriptor of the 64-byte swizzle: rows of 64 bytes, eight of them every 512
__device__ __forceinline__ unsigned long long sp_desc(unsigned at) {
    return (unsigned long long)((at >> 4) & 0x3FFFu) | (1ull << 16) | ((unsigned long long)(512 >> 4) << 32) | (1ull << 46) | (4ull << 61);
}

// The twelve products of a chunk, two steps of sixteen entries each.  hi hi go to `large`, an accumulator that starts at zero with every chunk, the
// small ones to `small`, which starts with the first chunk (`more`: this is a later one).
// w: columns of tensor memory, 16 of hi, of mid and of lo; a, a_mid, a_lo: descriptors.  The whole warp calls; the elected thread issues.
__device__ __forceinline__ void sp_products(unsigned elected, unsigned large, unsigned small, unsigned w, unsigned long long a, unsigned long long a_mid, unsigned long long a_lo,
                                            unsigned idesc, unsigned more) {
#define SP_MMA(d, wt, ad, p) " @e tcgen05.mma.cta_group::1.kind::f16 [" d "], [" wt "], " ad ", %10, " p ";\n"
    asm volatile("{\n .reg .pred yes, no, e, f;\n .reg .b32 h1, m0, m1, l0, l1;\n"
                 " setp.eq.u32 yes, 0, 0;\n setp.ne.u32 no, 0, 0;\n setp.ne.u32 e, %0, 0;\n setp.ne.u32 f, %11, 0;\n"
                 " add.u32 h1, %3, 8;\n add.u32 m0, %3, 16;\n add.u32 m1, %3, 24;\n add.u32 l0, %3, 32;\n add.u32 l1, %3, 40;\n"
                 SP_MMA("%2", "l0", "%4", "f") SP_MMA("%2", "l1", "%5", "yes") SP_MMA("%2", "%3", "%8", "yes") SP_MMA("%2", "h1", "%9", "yes")
                 SP_MMA("%2", "m0", "%6", "yes") SP_MMA("%2", "m1", "%7", "yes") SP_MMA("%2", "m0", "%4", "yes") SP_MMA("%2", "m1", "%5", "yes")
                 SP_MMA("%2", "%3", "%6", "yes") SP_MMA("%2", "h1", "%7", "yes") SP_MMA("%1", "%3", "%4", "no") SP_MMA("%1", "h1", "%5", "yes")
                 "}"
                 ::"r"(elected), "r"(large), "r"(small), "r"(w), "l"(a), "l"(a + 2), "l"(a_mid), "l"(a_mid + 2), "l"(a_lo), "l"(a_lo + 2), "r"(idesc), "r"(more) : "memory");
#undef SP_MMA
}
__device__ __forceinline__ void sp_st8(unsigned taddr, const unsigned (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
// acc (pairs of columns) += the first `columns` columns (a multiple of eight) of this thread's lane
template <int COLS>
__device__ __forceinline__ void sp_add_columns(unsigned long long (&acc)[COLS / 2], unsigned taddr, int columns) {
    constexpr int STEP = COLS < 32 ? COLS : 32;
#pragma unroll
    for (int c0 = 0; c0 < COLS; c0 += STEP) {
        unsigned r[STEP];
#pragma unroll
        for (int c = 0; c < STEP; c += 8)
            if (c0 + c < columns)
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(r[c]), "=r"(r[c + 1]), "=r"(r[c + 2]), "=r"(r[c + 3]), "=r"(r[c + 4]), "=r"(r[c + 5]), "=r"(r[c + 6]), "=r"(r[c + 7]) : "r"(taddr + c0 + c) : "memory");
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int c = 0; c < STEP; c += 8)                  // (not before the wait)
            asm volatile("" : "+r"(r[c]), "+r"(r[c + 1]), "+r"(r[c + 2]), "+r"(r[c + 3]), "+r"(r[c + 4]), "+r"(r[c + 5]), "+r"(r[c + 6]), "+r"(r[c + 7]) :: "memory");
#pragma unroll
        for (int c = 0; c < STEP; c += 2) asm("add.rn.f32x2 %0, %0, %1;" : "+l"(acc[(c0 + c) / 2]) : "l"(sp_pair(r[c], r[c + 1])));
    }
}
// epilogue: 0 store float32, 1 store bfloat16, 2 add into float32 (the residual stream)
__device__ __forceinline__ void sp_finish(float v, void* out, size_t at, const void* bias, int bias_dtype, int n, int epilogue) {
    if (bias) v += load_as_f(bias, bias_dtype, n);
    if (epilogue == 0) ((float*)out)[at] = v;
    else if (epilogue == 1) ((bf16*)out)[at] = __float2bfloat16_rn(v);
    else ((float*)out)[at] += v;
}
// true when the phase with this parity has completed; false when the wait ran out or another role gave up
__device__ __forceinline__ bool sp_wait(unsigned bar, unsigned parity, volatile int* abort_flag, int* status) {
    unsigned done;
    asm volatile("{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    if (done) return true;
    const long long deadline = clock64() + AT_WAIT_CYCLES;
    for (;;) {
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
        if (*abort_flag) return false;
        if (clock64() > deadline) {
            *abort_flag = 1;
            atomicExch(status, 9);
            return false;
        }
    }
}
// The wait for what the cluster's other CTAs send: whatever happened here they send it, at the latest when their own waits have run out.
__device__ __forceinline__ bool sp_wait_sent(unsigned bar) { return at_wait(bar, 0) || at_wait(bar, 0) || at_wait(bar, 0); }
__device__ __forceinline__ bool sp_wait_warp(unsigned bar, unsigned parity, volatile int* abort_flag, int* status) {
    return __all_sync(0xffffffffu, sp_wait(bar, parity, abort_flag, status));
}

// Rows of A as their parts, [3][M][K], for tiles of many rows.
__global__ void __launch_bounds__(256) split_rows_kernel(const float* A, bf16* parts, long long entries, int vec_a) {
    pdl_launch_dependents();
    pdl_wait();
    const long long at = ((long long)blockIdx.x * 256 + threadIdx.x) * 8;
    if (at >= entries) return;
    float v[8];
    if (vec_a) {
        const float4 lo = *reinterpret_cast<const float4*>(A + at), hi = *reinterpret_cast<const float4*>(A + at + 4);
        v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w; v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = A[at + i];
    }
    unsigned part[SP_PARTS][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        sp_cut(v[2 * i], v[2 * i + 1], part[0][i], part[1][i], part[2][i]);
        if (fminf(fabsf(v[2 * i]), fabsf(v[2 * i + 1])) < SP_SMALL) part[0][i] = sp_marked(v[2 * i], v[2 * i + 1]);
    }
#pragma unroll
    for (int q = 0; q < SP_PARTS; ++q) *reinterpret_cast<uint4*>(parts + q * entries + at) = make_uint4(part[q][0], part[q][1], part[q][2], part[q][3]);
}

// NT rows of A a tile: 16, 32 or 64; or (SP_MANY) up to 128, `nt` of them, whose parts come by TMA.
template <int NT>
__global__ void __launch_bounds__(sp_threads<NT>(), 1) linear_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const float* A,
                                                                           const float* W, const void* bias, int bias_dtype, void* out, int epilogue, int M, int N, int K,
                                                                           int ranges, int nt, int vec_a, int* status) {
    constexpr bool MANY = NT == SP_MANY;
    constexpr int RING = sp_ring<NT>(), SUMS = sp_sums<NT>(), CUTTERS = sp_cutters<NT>(), TAKER = CUTTERS + 2, COLS = NT * 4 / sp_takers<NT>();
    constexpr int TPT = NT >= 32 ? NT / 32 : 1, GROUPS = CUTTERS / 4;      // TPT: runs of eight entries of A a thread cuts
    if (!MANY) nt = NT;
    const int part_bytes = nt * SP_KC * 2, slots = MANY ? sp_slots(nt) : SP_SLOTS;
    extern __shared__ unsigned char sp_raw[];
    __shared__ __align__(8) unsigned long long bars[2 * RING + 3 * SP_SLOTS + 2 * SUMS + 1];
    __shared__ unsigned tmem_base_s;
    __shared__ int abort_s, odd_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (!status) status = &sp_gave_up;
    const unsigned smem = (at_smem(sp_raw) + 1023u) & ~1023u, a_parts = smem + RING * SP_BOX;
    const int rank = blockIdx.x % ranges, n0 = blockIdx.x / ranges * SP_ROWS, m0 = blockIdx.y * nt;
    const int all = (K + SP_KC - 1) / SP_KC, each = (all + ranges - 1) / ranges;
    const int k_begin = rank * each * SP_KC, k_end = min(K, k_begin + each * SP_KC), chunks = (k_end - k_begin + SP_KC - 1) / SP_KC;
    const unsigned w_full = at_smem(bars), w_empty = w_full + 8 * RING, full = w_empty + 8 * RING, empty = full + 8 * SP_SLOTS, sum_full = empty + 8 * SP_SLOTS,
                   sum_empty = sum_full + 8 * SUMS, sent = sum_empty + 8 * SUMS, a_full = sent + 8;
    // the rows of A whose sums over the cluster this CTA finishes
    const int slice = (nt + ranges - 1) / ranges, first_row = rank * slice, rows = max(0, min(min(nt, first_row + slice), M - m0) - first_row);

    if (warp == CUTTERS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(at_smem(&tmem_base_s)), "r"((unsigned)SP_TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 32 * (CUTTERS + 1)) {
        const auto init = [](unsigned bar, int count, unsigned arrivals) {
            for (int i = 0; i < count; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar + 8 * i), "r"(arrivals) : "memory");
        };
        init(w_full, RING, 1); init(w_empty, RING, 4); init(full, SP_SLOTS, 4); init(a_full, SP_SLOTS, 1); init(empty, SP_SLOTS, 1); init(sum_full, SUMS, 1); init(sum_empty, SUMS, sp_takers<NT>());
        if (!MANY) {
            init(sent, 1, 1);
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sent), "r"((unsigned)((ranges - 1) * rows * SP_ROWS * 4)) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n\tfence.proxy.async.shared::cta;" ::: "memory");
        abort_s = odd_s = 0;
    }
    const auto bring_w = [&](int c) {                      // rows and entries behind the last are zeros
        const int s = c % RING;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(w_full + 8 * s), "r"((unsigned)SP_BOX) : "memory");
        at_tma_2d(smem + s * SP_BOX, &map_w, k_begin + c * SP_KC, n0, w_full + 8 * s);
    };
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (!MANY && ranges > 1) asm volatile("barrier.cluster.arrive.release;" ::: "memory");      // this CTA can be sent to
    const unsigned tmem = tmem_base_s, sums = tmem + slots * SP_W_COLS, small = sums + SUMS * nt;
    pdl_launch_dependents();                               // (behind the allocation of tensor memory: a later kernel must not take it first)
    // W may be what the kernel in front writes: until that has ended it is only brought as far as L2, where its writes arrive too
    if (tid == 32 * (CUTTERS + 1))
        for (int c = 0; c < min(RING, chunks); ++c)
            asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(&map_w), "r"(k_begin + c * SP_KC), "r"(n0) : "memory");
    pdl_wait();
    if (tid == 32 * (CUTTERS + 1))
        for (int c = 0; c < min(RING, chunks); ++c) bring_w(c);

    unsigned long long acc[COLS / 2];                      // pairs of columns
    const int column0 = MANY ? ((warp - TAKER) >> 2) * COLS : 0, columns = MANY ? max(0, min(COLS, nt - column0)) : NT;
    if (warp < CUTTERS) {
        const int row = tid & 127, lr = row >> 2, lk = (tid & 3) * 8;
        const unsigned lanes = (unsigned)((warp & 3) * 32) << 16;
        // entries k .. k + 7 of a row are 16 bytes; the four groups of a row are exchanged by half its place in a run of eight
        const unsigned group = lr * 64 + ((((unsigned)lk >> 3) ^ ((lr >> 1) & 3)) << 4);
        float ra[TPT][8];
        auto fetch_a = [&](int c) {                        // rows behind the last are read as the last and not stored (K is a multiple of eight)
            const int k = k_begin + c * SP_KC + lk;
#pragma unroll
            for (int e = 0; e < TPT; ++e) {
                const float* p = A + (size_t)min(m0 + lr + 32 * e, M - 1) * K + k;
                if (k < k_end && vec_a) sp_load8(ra[e], p);
                else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) ra[e][i] = k < k_end ? p[i] : 0.f;
                }
            }
        };
        if (!MANY && (warp >> 2) < chunks) fetch_a(warp >> 2);
        int s = warp >> 2, turn = 0;                       // the chunk's slot, and how often it was taken before (parity): stepped, not divided out of c
        for (int c = warp >> 2; c < chunks; c += GROUPS) {
            const int r = c % RING;
            if (!sp_wait_warp(w_full + 8 * r, (c / RING) & 1, &abort_s, status)) break;
            bool ok = true;
            float least = INFINITY;                        // the smallest of the entries cut here
            const auto four = [&](int j) { return sp_shared_four(smem + r * SP_BOX + row * 128 + ((j ^ (row & 7)) << 4)); };
            const unsigned to = tmem + lanes + s * SP_W_COLS, a_to = a_parts + s * SP_PARTS * part_bytes + group;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                unsigned hi[SP_KC / 4], mid[SP_KC / 4], lo[SP_KC / 4];
#pragma unroll
                for (int j = 0; j < SP_KC / 8; ++j) {
                    const float4 v = four(4 * half + j);
                    sp_least(least, v.x, v.y); sp_least(least, v.z, v.w);
                    sp_cut(v.x, v.y, hi[2 * j], mid[2 * j], lo[2 * j]);
                    sp_cut(v.z, v.w, hi[2 * j + 1], mid[2 * j + 1], lo[2 * j + 1]);
                }
                if (half == 0) {                           // (the first half is cut while the slot's last products end)
                    if (c >= slots && !(ok = sp_wait_warp(empty + 8 * s, turn ^ 1, &abort_s, status))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                }
                sp_st8(to + 8 * half, hi); sp_st8(to + 8 * half + SP_KC / 2, mid); sp_st8(to + 8 * half + SP_KC, lo);
            }
            if (!ok) break;
            if (!MANY) {
#pragma unroll
                for (int e = 0; e < TPT; ++e)
                    if (NT >= 32 || lr < NT) {
                        unsigned part[SP_PARTS][4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            sp_least(least, ra[e][2 * i], ra[e][2 * i + 1]);
                            sp_cut(ra[e][2 * i], ra[e][2 * i + 1], part[0][i], part[1][i], part[2][i]);
                        }
#pragma unroll
                        for (int q = 0; q < SP_PARTS; ++q) sp_put_four(a_to + e * 32 * 64 + q * part_bytes, part[q]);
                    }
            }
            if (__any_sync(0xffffffffu, least < SP_SMALL)) {      // (zeros, as a rule)
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
#pragma unroll 1
                for (int half = 0; half < 2; ++half) {
                    unsigned hi[SP_KC / 4];
#pragma unroll
                    for (int j = 0; j < SP_KC / 8; ++j) {
                        const float4 v = four(4 * half + j);
                        hi[2 * j] = sp_marked(v.x, v.y); hi[2 * j + 1] = sp_marked(v.z, v.w);
                    }
                    __syncwarp();
                    sp_st8(to + 8 * half, hi);
                }
                if (!MANY) {
#pragma unroll
                    for (int e = 0; e < TPT; ++e)
                        if (NT >= 32 || lr < NT) {
                            unsigned part[4];
#pragma unroll
                            for (int i = 0; i < 4; ++i) part[i] = sp_marked(ra[e][2 * i], ra[e][2 * i + 1]);
                            sp_put_four(a_to + e * 32 * 64, part);
                        }
                }
            }
            __syncwarp();
            if (lane == 0) at_arrive(w_empty + 8 * r);
            if (!MANY) {
                if (c + GROUPS < chunks) fetch_a(c + GROUPS);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            } else if ((warp & 3) == 0 && !sp_wait_warp(a_full + 8 * s, turn, &abort_s, status)) break;
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) at_arrive(full + 8 * s);
            s += GROUPS;                                   // (no more groups than slots)
            if (s >= slots) { s -= slots; turn ^= 1; }
        }
    } else if (warp == CUTTERS) {
        const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(nt / 8) << 17) | ((unsigned)(SP_ROWS / 16) << 24);
        const unsigned elected = pe_elect();
        int issued = 0, s = 0, turn = 0;
        for (int c = 0; c < chunks; ++c) {
            const int b = c % SUMS;
            if (c >= SUMS && !sp_wait_warp(sum_empty + 8 * b, (c / SUMS - 1) & 1, &abort_s, status)) break;
            if (!sp_wait_warp(full + 8 * s, turn, &abort_s, status)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned long long a = sp_desc(a_parts + s * SP_PARTS * part_bytes), part = part_bytes >> 4;
            sp_products(elected, sums + b * nt, small, tmem + s * SP_W_COLS, a, a + part, a + 2 * part, idesc, c > 0);
            if (elected) {
                at_commit(empty + 8 * s);
                at_commit(sum_full + 8 * b);
            }
            __syncwarp();
            issued = c + 1;
            if (++s == slots) { s = 0; turn ^= 1; }
        }
        if (issued > 0) at_wait_warp(sum_full + 8 * ((issued - 1) % SUMS), ((issued - 1) / SUMS) & 1);      // nothing stays under way
    } else if (warp == CUTTERS + 1) {
        if (lane == 0) {
            int brought = min(RING, chunks), brought_a = 0, s = 0, turn = 0;
            for (int c = 0; c < chunks; ++c) {
                const int r = c % RING;
                if (MANY) {
                    if (c >= slots && !sp_wait(empty + 8 * s, turn ^ 1, &abort_s, status)) break;
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a_full + 8 * s), "r"((unsigned)(SP_PARTS * part_bytes)) : "memory");
                    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                                 ::"r"(a_parts + s * SP_PARTS * part_bytes), "l"(&map_a), "r"(a_full + 8 * s), "r"(k_begin + c * SP_KC), "r"(m0), "r"(0) : "memory");
                    brought_a = c + 1;
                    if (++s == slots) { s = 0; turn ^= 1; }
                }
                if (c + RING < chunks) {
                    if (!sp_wait(w_empty + 8 * r, (c / RING) & 1, &abort_s, status)) break;
                    bring_w(c + RING);
                    brought = c + RING + 1;
                }
            }
            // (each of them has landed long ago unless a role gave up)
            for (int c = max(0, brought - RING); c < brought; ++c) at_wait(w_full + 8 * (c % RING), (c / RING) & 1);
            for (int c = max(0, brought_a - slots); c < brought_a; ++c) at_wait(a_full + 8 * (c % slots), (c / slots) & 1);
        }
        __syncwarp();
    } else {
        const unsigned mine = sums + ((unsigned)((warp & 3) * 32) << 16) + column0;
#pragma unroll
        for (int i = 0; i < COLS / 2; ++i) acc[i] = 0ull;
        for (int c = 0; c < chunks; ++c) {
            const int b = c % SUMS;
            if (!sp_wait_warp(sum_full + 8 * b, (c / SUMS) & 1, &abort_s, status)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            sp_add_columns<COLS>(acc, mine + b * nt, columns);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) at_arrive(sum_empty + 8 * b);
        }
        if (chunks > 0) sp_add_columns<COLS>(acc, mine + SUMS * nt, columns);      // (the last chunk's products were these accumulators' last)
    }
    __syncthreads();                                       // all products have ended, all copies have landed
    bool whole = *(volatile int*)&abort_s == 0;
    if (warp >= TAKER) {                                   // [nt][128] sums where the operands were
        const int row = (warp & 3) * 32 + lane, n = n0 + row;
        float zero = 0.f;                                  // no number if one of the sums is not finite
#pragma unroll
        for (int i = 0; i < COLS; ++i)
            if (i < columns) {
                const float v = __uint_as_float((unsigned)(acc[i / 2] >> (32 * (i & 1))));
                zero = fmaf(v, 0.f, zero);
                asm volatile("st.shared.f32 [%0], %1;" ::"r"(smem + ((column0 + i) * SP_ROWS + row) * 4), "f"(v) : "memory");
            }
        if (zero != 0.f && n < N) odd_s = 1;
    }
    __syncthreads();
    if (odd_s) {                                           // sums that are not finite, a warp each, all warps a share
#pragma unroll 1
        for (int i = warp; i < 4 * min(nt, M - m0); i += sp_threads<NT>() / 32) {
            const unsigned at = smem + ((i >> 2) * SP_ROWS + (i & 3) * 32 + lane) * 4;
            const float* a = A + (size_t)(m0 + (i >> 2)) * K;
            float v;
            asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
            unsigned odd = __ballot_sync(0xffffffffu, !isfinite(v) && n0 + (i & 3) * 32 + lane < N);
#pragma unroll 1
            for (; odd; odd &= odd - 1) {
                const float* w = W + (size_t)(n0 + (i & 3) * 32 + __ffs(odd) - 1) * K;
                float sum = 0.f;
#pragma unroll 4
                for (int k = k_begin + lane; k < k_end; k += 32) sum = fmaf(a[k], w[k], sum);
                sum = warp_sum(sum);
                if (lane == __ffs(odd) - 1) asm volatile("st.shared.f32 [%0], %1;" ::"r"(at), "f"(sum) : "memory");
            }
        }
    }
    const unsigned sums_sent = a_parts + SP_SLOTS * SP_PARTS * part_bytes;       // [rank][slice][128]
    if (MANY) {
        if (ranges > 1) sp_cluster_sync(); else __syncthreads();
    } else {
        __syncthreads();
        if (ranges > 1) {
            asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
            for (int i = tid; i < min(nt, M - m0) * (SP_ROWS / 4); i += sp_threads<NT>()) {
                const int t = i / (SP_ROWS / 4), col = i % (SP_ROWS / 4) * 4, to = t / slice;
                if (to == rank) continue;
                const float4 v = sp_shared_four(smem + (t * SP_ROWS + col) * 4);
                asm volatile("{\n .reg .b32 at, bar;\n mapa.shared::cluster.u32 at, %0, %2;\n mapa.shared::cluster.u32 bar, %1, %2;\n"
                             " st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [at], {%3, %4, %5, %6}, [bar];\n}"
                             ::"r"(sums_sent + ((rank * slice + t - to * slice) * SP_ROWS + col) * 4), "r"(sent), "r"(to), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
            }
            asm volatile("barrier.cluster.arrive.release;" ::: "memory");      // this CTA has sent
            if (rows > 0 && !sp_wait_sent(sent)) {
                whole = false;
                atomicExch(status, 9);
            }
        }
    }
#pragma unroll 1
    for (int i = tid; i < (whole ? rows * (SP_ROWS / 4) : 0); i += sp_threads<NT>()) {
        const int t = i / (SP_ROWS / 4), col = i % (SP_ROWS / 4) * 4, n = n0 + col;
        if (n >= N) continue;
        const unsigned at = smem + ((first_row + t) * SP_ROWS + col) * 4;
        float4 part[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            if (c >= ranges) part[c] = make_float4(0.f, 0.f, 0.f, 0.f);
            else if (MANY) part[c] = sp_peer_four(at, c);
            else part[c] = sp_shared_four(c == rank ? at : sums_sent + ((c * slice + t) * SP_ROWS + col) * 4);
        }
        float4 v = part[0];
#pragma unroll
        for (int c = 1; c < 8; ++c)
            if (c < ranges) { v.x += part[c].x; v.y += part[c].y; v.z += part[c].z; v.w += part[c].w; }
        const float four[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (n + e < N) sp_finish(four[e], out, (size_t)(m0 + first_row + t) * N + n + e, bias, bias_dtype, n + e, epilogue);
    }
    if (MANY && ranges > 1) sp_cluster_sync();             // nobody leaves while its sums are being read
    if (!MANY && ranges > 1) {
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");           // or before all have sent
        if (!whole && rows > 0) sp_wait_sent(sent);
    }
    if (warp == CUTTERS) {
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((unsigned)SP_TMEM) : "memory");
    }
}

// Boxes of 32 entries x `rows` rows of float32 [R][K], or of all parts in bfloat16 [SP_PARTS][R][K]; what lies outside reads as zero.
static int sp_map(CUtensorMap* map, const void* base, int K, int R, int rows, bool parts) {
    at_encode_fn enc = at_encoder();
    if (!enc) return PE_ERR_UNSUPPORTED;
    const unsigned size = parts ? 2 : 4;
    const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)R, SP_PARTS}, strides[2] = {(cuuint64_t)K * size, (cuuint64_t)K * R * size};
    const cuuint32_t box[3] = {SP_KC, (cuuint32_t)rows, SP_PARTS}, elem[3] = {1, 1, 1};
    const CUresult r = enc(map, parts ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, parts ? 3 : 2, const_cast<void*>(base), dims, strides, box, elem,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, parts ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : 20000 + (int)r;
}

template <int NT>
static int sp_go(const CUtensorMap& map_w, const CUtensorMap& map_a, int nt, const float* A, const float* W, const void* bias, int bias_dtype, void* out, int epilogue,
                 int M, int N, int K, int* status, cudaStream_t s) {
    auto kernel = linear_split_kernel<NT>;
    const int mt = (M + nt - 1) / nt, ranges = sp_ranges(N, K);
    if (mt > 65535) return PE_ERR_UNSUPPORTED;
    PE_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sp_smem_bytes<NT>()));
    PE_TRY(pe_launch_cluster(kernel, dim3((N + SP_ROWS - 1) / SP_ROWS * ranges, mt), sp_threads<NT>(), sp_smem_bytes<NT>(), s, ranges, map_w, map_a, A, W, bias, bias_dtype,
                             out, epilogue, M, N, K, ranges, nt, (int)((uintptr_t)A % 32 == 0), status));
    PE_LAUNCH_CHECK();
    return 0;
}

// How many clusters of `ranges` CTAs of the form for many rows run at once on this device.
static int sp_resident_clusters(int ranges, int& n) {
    static int known[64][9];                               // (the same number whoever writes it)
    int device = 0;
    PE_TRY(cudaGetDevice(&device));
    if (device < 64 && known[device][ranges] > 0) { n = known[device][ranges]; return 0; }
    auto kernel = linear_split_kernel<SP_MANY>;
    PE_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sp_smem_bytes<SP_MANY>()));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ranges); cfg.blockDim = dim3(sp_threads<SP_MANY>()); cfg.dynamicSmemBytes = sp_smem_bytes<SP_MANY>();
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ranges; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    PE_TRY(cudaOccupancyMaxActiveClusters(&n, kernel, &cfg));
    if (n < 1) return PE_ERR_UNSUPPORTED;
    if (device < 64) known[device][ranges] = n;
    return 0;
}

// Whether a product of float32 operands comes here: by N, K and the place of W alone, so that a row's result is the same in every step.
// 800,000 entries is where one row takes as long either way: 1, 12, 60 and 508 rows, here / as multiply-adds, 512 x 512 5.3 5.5 8.4 11.5 / 3.2 4.2 8.4 16.8,
// 768 x 768 5.7 5.9 8.7 13.8 / 4.5 5.8 11.2 24.8, 1024 x 768 5.6 5.7 8.6 14.3 / 5.3 7.6 12.1 25.0, 832 x 960 5.5 5.7 8.3 15.7 / 5.5 7.9 13.6 31.5, 1024 x 1024 5.6 5.7 8.4
// 16.3 / 6.3 9.4 14.9 31.4; narrow ones lose a little at one row: 3200 x 256 5.1 / 4.8, 256 x 3200 7.1 / 6.9, 1280 x 640 6.3 / 5.8.
extern "C" int pe_linear_split_takes(const void* W, int N, int K) { return N >= 256 && K >= 256 && (long long)N * K >= 800000 && K % 8 == 0 && (uintptr_t)W % 16 == 0; }

// Rows of A that are cut at a time, so that their parts take 256 MB at most; and the bytes of scratch a product of M rows needs.
static int sp_slab(int K) { return (int)((256ll << 20) / (2ll * SP_PARTS * K) > SP_MANY ? (256ll << 20) / (2ll * SP_PARTS * K) / SP_MANY * SP_MANY : SP_MANY); }
extern "C" long long pe_linear_split_scratch(int M, int K) { return M <= 64 ? 0 : 2ll * SP_PARTS * K * (M < sp_slab(K) ? M : sp_slab(K)); }
// The kernels that a product of M rows launches.
extern "C" int pe_linear_split_launches(int M, int K) { return M <= 0 ? 0 : M <= 64 ? 1 : 2 * ((M + sp_slab(K) - 1) / sp_slab(K)); }

// What the word of products without one holds on the current device; it is zero again behind this.  Synchronises.
extern "C" int pe_linear_split_gave_up(int* code) {
    const int zero = 0;
    PE_TRY(cudaMemcpyFromSymbol(code, sp_gave_up, sizeof(int)));
    if (*code) PE_TRY(cudaMemcpyToSymbol(sp_gave_up, &zero, sizeof(int)));
    return 0;
}

extern "C" int pe_linear_split(const void* A, const void* W, const void* bias, int bias_dtype, void* out, int epilogue, int M, int N, int K, void* scratch, void* status, void* stream) {
    if (M <= 0) return 0;
    if (!pe_linear_split_takes(W, N, K) || epilogue < 0 || epilogue > 2) return PE_ERR_UNSUPPORTED;
    CUtensorMap map_w = {}, map_a = {};
    const cudaStream_t s = (cudaStream_t)stream;
    if (const int e = sp_map(&map_w, W, K, N, SP_ROWS, false)) return e;
#define SP_GO(NT, nt, A, out, M) sp_go<NT>(map_w, map_a, nt, (const float*)(A), (const float*)W, bias, bias_dtype, out, epilogue, M, N, K, (int*)status, s)
    if (M <= 16) return SP_GO(16, 16, A, out, M);
    if (M <= 32) return SP_GO(32, 32, A, out, M);
    if (M <= 64) return SP_GO(64, 64, A, out, M);
    int clusters = 0;
    if (const int e = sp_resident_clusters(sp_ranges(N, K), clusters)) return e;
    const long long tiles = (N + SP_ROWS - 1) / SP_ROWS;
    for (int first = 0; first < M; first += sp_slab(K)) {
        const int rows = M - first < sp_slab(K) ? M - first : sp_slab(K);
        // Rows of A a tile: the fewest turns of clusters, each as long as its rows and as what it does whatever their number (508 rows, 9,728 x
        // 896, three turns of 112 rows 66 us; 896 x 896, one of 128 13 us, two of 112 22).
        int nt = SP_MANY;
        long long least = -1;
        for (int t = SP_MANY; t >= 64; t -= 16) {
            const long long cost = ((rows + t - 1) / t * tiles + clusters - 1) / clusters * (t + 96);
            if (least < 0 || cost < least) { least = cost; nt = t; }
        }
        const float* a = (const float*)A + (size_t)first * K;
        void* o = (char*)out + (size_t)first * N * (epilogue == 1 ? 2 : 4);
        const long long entries = (long long)rows * K;
        PE_TRY(pe_launch(split_rows_kernel, dim3((unsigned)((entries / 8 + 255) / 256)), 256, 0, s, a, (bf16*)scratch, entries, (int)((uintptr_t)a % 16 == 0)));
        PE_LAUNCH_CHECK();
        if (const int e = sp_map(&map_a, scratch, K, rows, nt, true)) return e;
        if (const int e = SP_GO(SP_MANY, nt, a, o, rows)) return e;
    }
#undef SP_GO
    return 0;
}
