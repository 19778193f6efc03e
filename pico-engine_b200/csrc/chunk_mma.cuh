// Float32 products over chunks of 64 tokens on the tensor cores, every float32 number in three bfloat16 parts that hold all of its bits:
// hi = round(v), mid = round(v - hi), lo = round(v - hi - mid).  Of the nine products of two numbers six are made (the other three are
// below 2^-25 of theirs).  The tensor cores cut their sums to 24 bits, so hi hi is summed over 32 entries at a time and these sums are
// added as float32 numbers are; the small products, 2^-8 of it at most, are summed first.
//
// Numbers are cut times 2^24, so that the lowest part of the smallest of them is still a bfloat16 number, and results are brought back: a power of two
// changes no bits.  What parts are not made of is numbers of 2^35 and more (sums of products of smaller ones stay inside float32), infinities and numbers that are
// none: cm_watch finds them on the way, and the results that they reach are worked out with multiply-adds.  (A token with such a number reaches none in
// front of it: cm_mend puts zeros in its place, and those keep their bits.)
//
// A plane is 64 rows (tokens) of 64 bfloat16 numbers, a part each: rows of 128 bytes whose eight 16-byte groups are exchanged by the row's
// place in a run of eight, which is what the 128-byte swizzle of an operand in shared memory is, along a row (K-major) or across rows.
#pragma once
#include "tcgen05_attention.cuh"

#define CM_CHUNK 64                                       // tokens of a chunk
#define CM_PLANE (CM_CHUNK * 128)                         // bytes
#define CM_PARTS 3
#define CM_UP 0x1p24f
#define CM_DOWN 0x1p-24f                                  // for each operand that was cut
#define CM_MOST 0x5d00u                                   // 2^59 as bfloat16: 2^35 times 2^24
#define CM_MOST_PLAIN 0x5100u                             // 2^35, of numbers that are bfloat16 already

__device__ __forceinline__ unsigned cm_at(int row, int group) { return row * 128 + ((group ^ (row & 7)) << 4); }      // eight numbers of a row in a plane

// Two neighbouring numbers' parts, packed.
__device__ __forceinline__ unsigned long long cm_pair(unsigned a, unsigned b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ float2 cm_scaled(float a, float b, float by) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(at_two(a, b)), "l"(at_two(by, by)));
    return at_both(r);
}
template <int N>
__device__ __forceinline__ void cm_scale(float (&v)[N], float by) {
#pragma unroll
    for (int i = 0; i < N; i += 2) { const float2 r = cm_scaled(v[i], v[i + 1], by); v[i] = r.x; v[i + 1] = r.y; }
}
// Two numbers at a time, each half as a plain multiply or multiply-add.
__device__ __forceinline__ unsigned long long cm_mul2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long cm_fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// A walk over a chunk's tokens with multiply-adds, for what parts are not made of: 256 threads, 128 columns.  Eight neighbouring lanes share four columns; a
// lane has their rows 32 j + 4 (lane % 8) .. + 3 of a state that lies [ND / 8][64 columns][8] (with a column a lane a token's reads of shared memory took 1,500 cycles).
template <int ND>
struct CMWalk {
    static constexpr int RUNS = ND / 32;
    unsigned long long s[4][2 * RUNS];
    static __device__ __forceinline__ int column() { return (threadIdx.x >> 3) * 4; }                        // the first of the thread's four
    static __device__ __forceinline__ int row() { return (threadIdx.x & 7) * 4; }
    static __device__ __forceinline__ size_t place() { return (size_t)(column() >> 6) * ND * 64 + ((row() >> 3) * 64 + (column() & 63)) * 8 + (row() & 7); }
    static __device__ __forceinline__ int written() { return column() + (threadIdx.x >> 1 & 2) + (threadIdx.x >> 1 & 1); }      // the column whose output `output` leaves
    // (no state: zeros); whether each of the thread's columns has a row that is no number, here or in a neighbour: no output of theirs is one then
    __device__ __forceinline__ bool begin(const float* state) {
        unsigned lost = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int j = 0; j < RUNS; ++j) {
                const float4 f = state ? *reinterpret_cast<const float4*>(state + place() + c * 8 + j * 2048) : make_float4(0.f, 0.f, 0.f, 0.f);
                s[c][2 * j] = at_two(f.x, f.y); s[c][2 * j + 1] = at_two(f.z, f.w);
                if (f.x != f.x || f.y != f.y || f.z != f.z || f.w != f.w) lost |= 1u << c;
            }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) lost |= __shfl_xor_sync(0xffffffffu, lost, o);
        return lost == 15u;
    }
    __device__ __forceinline__ void end(float* state) const {
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int j = 0; j < RUNS; ++j) *reinterpret_cast<ulonglong2*>(state + place() + c * 8 + j * 2048) = make_ulonglong2(s[c][2 * j], s[c][2 * j + 1]);
    }
    // s = decay s + k u: k (and decays, if there are any) a token's ND numbers in shared memory
    __device__ __forceinline__ void step(const float* k, const float* decays, float decay, const float (&u)[4]) {
        unsigned long long uu[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) uu[c] = at_two(u[c], u[c]);
#pragma unroll
        for (int j = 0; j < RUNS; ++j) {
            const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(k + row() + 32 * j);
            ulonglong2 d = make_ulonglong2(at_two(decay, decay), at_two(decay, decay));
            if (decays) d = *reinterpret_cast<const ulonglong2*>(decays + row() + 32 * j);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                s[c][2 * j] = cm_fma2(d.x, s[c][2 * j], cm_mul2(x.x, uu[c]));
                s[c][2 * j + 1] = cm_fma2(d.y, s[c][2 * j + 1], cm_mul2(x.y, uu[c]));
            }
        }
    }
    // q . s of column written(), in both lanes that have it
    __device__ __forceinline__ float output(const float* q) const {
        unsigned long long sum[4] = {0, 0, 0, 0};
#pragma unroll
        for (int j = 0; j < RUNS; ++j) {
            const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(q + row() + 32 * j);
#pragma unroll
            for (int c = 0; c < 4; ++c) sum[c] = cm_fma2(x.y, s[c][2 * j + 1], cm_fma2(x.x, s[c][2 * j], sum[c]));
        }
        float o[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) { const float2 v = at_both(sum[c]); o[c] = v.x + v.y; }
        const bool upper = threadIdx.x & 4, odd = threadIdx.x & 2;
        const float a = (upper ? o[2] : o[0]) + __shfl_xor_sync(0xffffffffu, upper ? o[0] : o[2], 4), b = (upper ? o[3] : o[1]) + __shfl_xor_sync(0xffffffffu, upper ? o[1] : o[3], 4);
        const float r = (odd ? b : a) + __shfl_xor_sync(0xffffffffu, odd ? a : b, 2);
        return r + __shfl_xor_sync(0xffffffffu, r, 1);
    }
};
// (numbers times CM_UP)
__device__ __forceinline__ void cm_cut(float a, float b, unsigned& hi, unsigned& mid, unsigned& lo) {
    unsigned long long rest = at_two(a, b);
    const unsigned long long minus = at_two(-1.f, -1.f);
    float2 r;
    hi = at_pack(a, b);
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(rest) : "l"(cm_pair(hi << 16, hi & 0xffff0000u)), "l"(minus));      // (exact)
    r = at_both(rest);
    mid = at_pack(r.x, r.y);
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(rest) : "l"(cm_pair(mid << 16, mid & 0xffff0000u)), "l"(minus));
    r = at_both(rest);
    lo = at_pack(r.x, r.y);
}
// The largest upper part that was seen (no number beats every number); whether it is more than parts are made of, as a tile's bit of a word.
__device__ __forceinline__ void cm_watch(unsigned& most, unsigned hi) {
    asm("{\n\t.reg .b32 t;\n\tabs.bf16x2 t, %1;\n\tmax.NaN.bf16x2 %0, %0, t;\n\t}" : "+r"(most) : "r"(hi));
}
// The same of numbers alone.  Where an entry joins every sum of its row (or column) of a product, one that is no number makes them all none, here as with
// multiply-adds, and reaches no other: nothing is left to be worked out.
__device__ __forceinline__ void cm_watch_numbers(unsigned& most, unsigned hi) {
    asm("{\n\t.reg .b32 t;\n\tabs.bf16x2 t, %1;\n\tmax.bf16x2 %0, %0, t;\n\t}" : "+r"(most) : "r"(hi));
}
__device__ __forceinline__ bool cm_odd(unsigned most, unsigned limit = CM_MOST) { return (most & 0x7fffu) >= limit || ((most >> 16) & 0x7fffu) >= limit; }
__device__ __forceinline__ unsigned cm_seen(unsigned most, int tile, unsigned limit = CM_MOST) { return (cm_odd(most, limit) ? 1u : 0u) << tile; }
__device__ __forceinline__ void cm_report(unsigned* seen, unsigned mine) {         // (a block's word in shared memory)
    const unsigned all = __reduce_or_sync(0xffffffffu, mine);
    if ((threadIdx.x & 31) == 0 && all) atomicOr(seen, all);
}
// Eight numbers' parts into planes that lie `stride` bytes apart, at `to` in the first (numbers times CM_UP).
template <bool NUMBERS = false>
__device__ __forceinline__ void cm_put(unsigned char* to, int stride, const float4& a, const float4& b, unsigned& most) {
    unsigned part[CM_PARTS][4];
    cm_cut(a.x, a.y, part[0][0], part[1][0], part[2][0]); cm_cut(a.z, a.w, part[0][1], part[1][1], part[2][1]);
    cm_cut(b.x, b.y, part[0][2], part[1][2], part[2][2]); cm_cut(b.z, b.w, part[0][3], part[1][3], part[2][3]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if constexpr (NUMBERS) cm_watch_numbers(most, part[0][i]);
        else cm_watch(most, part[0][i]);
    }
#pragma unroll
    for (int p = 0; p < CM_PARTS; ++p) *reinterpret_cast<uint4*>(to + p * stride) = make_uint4(part[p][0], part[p][1], part[p][2], part[p][3]);
}
// A plane of upper parts of which some are more than parts are made of: zeros for such entries in all of its `parts`, `stride` bytes apart; `first` becomes
// the first row that has one.  All threads.
__device__ __forceinline__ void cm_mend(unsigned char* plane, int stride, int parts, unsigned* first, unsigned limit = CM_MOST) {
#pragma unroll 1
    for (int i = threadIdx.x; i < CM_PLANE / 4; i += blockDim.x) {
        unsigned* at = reinterpret_cast<unsigned*>(plane) + i;
        const unsigned v = *at, keep = ((v & 0x7fffu) >= limit ? 0u : 0xffffu) | (((v >> 16) & 0x7fffu) >= limit ? 0u : 0xffff0000u);
        if (keep == 0xffffffffu) continue;
        for (int p = 0; p < parts; ++p) at[p * stride / 4] &= keep;
        atomicMin(first, (unsigned)(i / 32));
    }
}
// `bytes` (a multiple of 16, both addresses too) into shared memory, all threads of the block; cm_landed waits for all that were asked for.
__device__ __forceinline__ void cm_bring(unsigned char* dst, const void* src, int bytes) {
    for (int i = threadIdx.x * 16; i < bytes; i += blockDim.x * 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(at_smem(dst + i)), "l"((const char*)src + i) : "memory");
}
__device__ __forceinline__ void cm_landed() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void cm_load8(float4& a, float4& b, const float* p) {
    asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];" : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w) : "l"(p) : "memory");
}
__device__ __forceinline__ void cm_store8(float* p, const float (&v)[8]) {
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
}
// ---------------------------------------------------------------- products by tcgen05 (one warp calls, its elected thread issues)
// An operand of 64 entries of K: descriptors of its parts (`stride` bytes apart), and how far 16 entries of K are in 16-byte units.
struct CMOperand { unsigned long long hi, mid, lo; unsigned step; };
__device__ __forceinline__ CMOperand cm_along(unsigned at, int stride) {                     // K along the rows of the planes
    const unsigned long long d = at_desc(at, 0, 1024);
    return {d, d + (stride >> 4), d + 2 * (stride >> 4), 2u};
}
// K across the rows; the operand's second 64 columns are the plane `second` bytes behind
__device__ __forceinline__ CMOperand cm_across(unsigned at, int stride, int second) {
    const unsigned long long d = at_desc(at, second, 1024);
    return {d, d + (stride >> 4), d + 2 * (stride >> 4), 128u};
}
__device__ __forceinline__ void cm_issue(unsigned elected, unsigned sums, unsigned long long a, unsigned long long b, unsigned idesc, bool add) {
    asm volatile("{\n .reg .pred e, p;\n setp.ne.u32 e, %0, 0;\n setp.ne.u32 p, %5, 0;\n"
                 " @e tcgen05.mma.cta_group::1.kind::f16 [%1], %2, %3, %4, p;\n}"
                 ::"r"(elected), "r"(sums), "l"(a), "l"(b), "r"(idesc), "r"((unsigned)add) : "memory");
}
// [128 x N] products over 64 entries: hi hi of the first 32 in `first`; the small ones and then hi hi of the other 32 in `rest` (so that either sum is
// cut twice at its full size).  The whole warp goes through it, with the same operands (in a branch of one thread each instruction waits for
// its operands to be moved: 150 cycles apiece).
__device__ __forceinline__ void cm_products(unsigned elected, unsigned first, unsigned rest, const CMOperand& a, const CMOperand& b, unsigned idesc) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const unsigned ka = k * a.step, kb = k * b.step;
        cm_issue(elected, rest, a.lo + ka, b.hi + kb, idesc, k);
        cm_issue(elected, rest, a.hi + ka, b.lo + kb, idesc, true);
        cm_issue(elected, rest, a.mid + ka, b.mid + kb, idesc, true);
        cm_issue(elected, rest, a.mid + ka, b.hi + kb, idesc, true);
        cm_issue(elected, rest, a.hi + ka, b.mid + kb, idesc, true);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) cm_issue(elected, k < 2 ? first : rest, a.hi + k * a.step, b.hi + k * b.step, idesc, k != 0);
}
// The same for an A of one part (numbers that are bfloat16 already): three products.
__device__ __forceinline__ void cm_products_one(unsigned elected, unsigned first, unsigned rest, unsigned long long a, unsigned step, const CMOperand& b, unsigned idesc) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        cm_issue(elected, rest, a + k * step, b.lo + k * b.step, idesc, k);
        cm_issue(elected, rest, a + k * step, b.mid + k * b.step, idesc, true);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) cm_issue(elected, k < 2 ? first : rest, a + k * step, b.hi + k * b.step, idesc, k != 0);
}
// idesc: float32 sums of bfloat16 products, 128 rows, n columns, either operand across the rows of its planes or along them
__device__ __forceinline__ constexpr unsigned cm_idesc(int n, bool a_across, bool b_across) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((a_across ? 1u : 0u) << 15) | ((b_across ? 1u : 0u) << 16) | ((unsigned)(n >> 3) << 17) | ((unsigned)(128 >> 4) << 24);
}
// 16 or 32 columns of this thread's row, and acc += them
__device__ __forceinline__ void cm_read(float (&v)[16], unsigned taddr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\ttcgen05.wait::ld.sync.aligned;"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]),
                   "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void cm_read(float (&v)[32], unsigned taddr) { at_ld32(taddr, v); }
template <int N>
__device__ __forceinline__ void cm_take(float (&acc)[N], unsigned taddr) {
    float v[N];
    cm_read(v, taddr);
#pragma unroll
    for (int i = 0; i < N; ++i) acc[i] += v[i];
}

#define CM_TMEM 256                                       // columns of tensor memory a block: the two sums of 128 columns, or of two times 64
// A block's tensor memory and the barrier that its products arrive at.
__device__ __forceinline__ unsigned cm_begin(unsigned* tmem, unsigned long long* bar) {
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(at_smem(bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(at_smem(tmem)), "r"((unsigned)CM_TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    pdl_launch_dependents();                               // (behind the allocation: a later kernel must not take tensor memory first)
    return *tmem;
}
__device__ __forceinline__ void cm_end(unsigned tmem) {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (threadIdx.x < 32) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((unsigned)CM_TMEM) : "memory");
}
// What the block wrote to shared memory is there for the tensor core, and what it read of tensor memory has been read.
__device__ __forceinline__ void cm_ready() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// The block's next products have ended: one warp waits for them, the others for it (eight warps that ask the barrier again and again take the
// other block's issue slots).  A wait that runs out leaves a status, and every later one is bounded too.
__device__ __forceinline__ void cm_done(unsigned long long* bar, unsigned& phase, int* status) {
    if (threadIdx.x < 32 && !at_wait_warp(at_smem(bar), phase) && threadIdx.x == 0) atomicExch(status, 11);
    phase ^= 1;
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// ---------------------------------------------------------------- products by mma.sync (scores of a chunk's tokens over its keys)
__device__ __forceinline__ void cm_ldmatrix(unsigned& a, unsigned& b, unsigned& c, unsigned& d, unsigned at) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(a), "=r"(b), "=r"(c), "=r"(d) : "r"(at) : "memory");
}
__device__ __forceinline__ void cm_mma(float (&c)[4], const unsigned (&a)[4], const unsigned (&b)[2]) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// A warp's 16 tokens x 32 keys of [t][s], over 64 entries of queries and keys: planes of parts, `stride` bytes apart.  A thread holds tokens
// lane / 4 and lane / 4 + 8, keys 2 (lane % 4) and the one behind it of each run of eight.
struct CMScores {
    float sum[4][4], small[4][4];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) sum[j][e] = small[j][e] = 0.f;
    }
    __device__ __forceinline__ void add(unsigned q, unsigned k, int stride, int t0, int s0) {
        const int lane = threadIdx.x & 31;
#pragma unroll 1
        for (int ks = 0; ks < 4; ++ks) {
            unsigned a[CM_PARTS][4];
#pragma unroll
            for (int p = 0; p < CM_PARTS; ++p) cm_ldmatrix(a[p][0], a[p][1], a[p][2], a[p][3], q + p * stride + cm_at(t0 + (lane & 15), 2 * ks + (lane >> 4)));
#pragma unroll
            for (int y = CM_PARTS - 1; y >= 0; --y) {
                unsigned b[4][2];
#pragma unroll
                for (int j = 0; j < 4; j += 2)
                    cm_ldmatrix(b[j][0], b[j][1], b[j + 1][0], b[j + 1][1], k + y * stride + cm_at(s0 + 8 * j + (lane & 7) + (lane >> 4) * 8, 2 * ks + ((lane >> 3) & 1)));
#pragma unroll
                for (int x = CM_PARTS - 1 - y; x >= 0; --x)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (x + y) { cm_mma(small[j], a[x], b[j]); continue; }
                        float t[4] = {0.f, 0.f, 0.f, 0.f};
                        cm_mma(t, a[0], b[j]);
#pragma unroll
                        for (int e = 0; e < 4; ++e) sum[j][e] += t[e];
                    }
            }
        }
    }
    __device__ __forceinline__ float get(int j, int e) const { return sum[j][e] + small[j][e]; }      // (times CM_UP twice)
};
