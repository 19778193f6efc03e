// What the attention kernels on the 5th-generation tensor cores share: bounded mbarrier waits, TMA tiled loads, operand descriptors of the
// 128-byte swizzle, tcgen05.mma and its commits, loads and stores of tensor memory, and the tensor maps of the host side.
#pragma once
#include "common.cuh"
#include <cuda.h>

#define AT_WAIT_CYCLES 1000000000ll

__device__ __forceinline__ unsigned at_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool at_wait(unsigned bar, unsigned parity) {
    unsigned done;
    asm volatile("{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    if (done) return true;                                          // the usual case costs neither a clock read nor a suspended wait
    const long long deadline = clock64() + AT_WAIT_CYCLES;
    for (;;) {
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
        if (clock64() > deadline) return false;
    }
}
// the same for a whole warp: every lane gets the same answer, so the warp stays together on its way out
__device__ __forceinline__ bool at_wait_warp(unsigned bar, unsigned parity) {
    return __all_sync(0xffffffffu, at_wait(bar, parity));
}
__device__ __forceinline__ void at_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void at_tma_2d(unsigned dst, const CUtensorMap* map, int x, int y, unsigned bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y) : "memory");
}
// shared-memory operand descriptor, 128-byte swizzle: start address, leading and stride byte offsets
__device__ __forceinline__ unsigned long long at_desc(unsigned smem_addr, unsigned lbo, unsigned sbo) {
    return (unsigned long long)((smem_addr >> 4) & 0x3FFFu) | ((unsigned long long)((lbo >> 4) & 0x3FFFu) << 16) |
           ((unsigned long long)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46) | (2ull << 61);
}
// Products and commits are issued by a warp's elected thread (pe_elect).  The warp goes through the loop that issues them as one, waits included: in a branch
// of one lane's own a product took about 90 cycles to issue.  The kernels themselves gain little (2,048 tokens, 14 heads of 64: 21.9 -> 21.6 us; differential attention 47.9 -> 47.1;
// latent rows and mixed heads the same), in a chain of kernels the mixer with latent rows 98.2 -> 95.9 us, with mixed heads 71.5 -> 69.9.
__device__ __forceinline__ void at_mma(unsigned elected, unsigned tmem_d, unsigned long long a, unsigned long long b, unsigned idesc, unsigned accumulate) {
    asm volatile("{\n .reg .pred p, e;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 e, %5, 0;\n"
                 " @e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
                 ::"r"(tmem_d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(elected) : "memory");
}
// the same with A from tensor memory: row i on lane i, two neighbouring entries of a row in a column
__device__ __forceinline__ void at_mma_ts(unsigned elected, unsigned tmem_d, unsigned tmem_a, unsigned long long b, unsigned idesc, unsigned accumulate) {
    asm volatile("{\n .reg .pred p, e;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 e, %5, 0;\n"
                 " @e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
                 ::"r"(tmem_d), "r"(tmem_a), "l"(b), "r"(idesc), "r"(accumulate), "r"(elected) : "memory");
}
__device__ __forceinline__ void at_commit(unsigned bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void at_commit_by(unsigned elected, unsigned bar) {
    asm volatile("{\n .reg .pred e;\n setp.ne.b32 e, %1, 0;\n"
                 " @e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(bar), "r"(elected) : "memory");
}
// The value rows of a step (128 rows of 128 bytes in each of `panels` panels) from `used` on to the end of their page become zero.  They
// lie behind the run's last token, and a page is taken as its last owner left it: a weight of zero would not keep a value that is no
// number out of the outputs.  `threads` threads call it when the copies have landed and nothing but P V still reads the rows; each of
// them arrives (behind a __syncwarp of its warp) at the barrier that P V waits for.
__device__ __forceinline__ void at_clear_rows(unsigned values, int panels, int panel_bytes, int used, int thread, int threads) {
    const int bytes = (-used & (PE_PAGE - 1)) * 128;
    if (bytes == 0) return;
    for (int c = 0; c < panels; ++c)
        for (int i = thread * 16; i < bytes; i += threads * 16)
            asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(values + c * panel_bytes + used * 128 + i), "r"(0u) : "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // P V reads them through the tensor core's proxy
}
// 32 columns of this thread's lane.  at_ld32_start only issues the load: the values are there after at_ld_wait, and
// at_pin32 after that keeps the compiler from using the registers any earlier.
__device__ __forceinline__ void at_ld32_start(unsigned taddr, unsigned* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void at_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void at_pin32(unsigned* r) {
    asm volatile("" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                      "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]),
                      "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
                      "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
                 :: "memory");
}
__device__ __forceinline__ void at_ld32(unsigned taddr, float* v) {     // load and wait
    unsigned r[32];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void at_st32(unsigned taddr, const float* v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
                 "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
                 ::"r"(taddr),
                   "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])),
                   "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])),
                   "r"(__float_as_uint(v[8])), "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])), "r"(__float_as_uint(v[11])),
                   "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])), "r"(__float_as_uint(v[15])),
                   "r"(__float_as_uint(v[16])), "r"(__float_as_uint(v[17])), "r"(__float_as_uint(v[18])), "r"(__float_as_uint(v[19])),
                   "r"(__float_as_uint(v[20])), "r"(__float_as_uint(v[21])), "r"(__float_as_uint(v[22])), "r"(__float_as_uint(v[23])),
                   "r"(__float_as_uint(v[24])), "r"(__float_as_uint(v[25])), "r"(__float_as_uint(v[26])), "r"(__float_as_uint(v[27])),
                   "r"(__float_as_uint(v[28])), "r"(__float_as_uint(v[29])), "r"(__float_as_uint(v[30])), "r"(__float_as_uint(v[31]))
                 : "memory");
}
__device__ __forceinline__ float at_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ unsigned at_pack(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<unsigned*>(&v);
}

// Two numbers for the multiply-adds that take two at a time (each half rounds as a plain one does).
__device__ __forceinline__ unsigned long long at_two(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 at_both(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
// 2^(a * scale + off) and 2^(b * scale + off) as two bfloat16 numbers, and both (unrounded) into `sum`
__device__ __forceinline__ unsigned at_exp2_pair(float a, float b, unsigned long long scale, unsigned long long off, unsigned long long& sum) {
    unsigned long long x = at_two(a, b);
    asm("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(x) : "l"(scale), "l"(off));
    const float2 v = at_both(x);
    const float e0 = at_exp2(v.x), e1 = at_exp2(v.y);
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(sum) : "l"(at_two(e0, e1)));
    return at_pack(e0, e1);
}
__device__ __forceinline__ float at_sum_four(unsigned long long a, unsigned long long b) {
    const float2 x = at_both(a), y = at_both(b);
    return (x.x + x.y) + (y.x + y.y);
}
// COLS bfloat16 columns of 32 rows (a row a lane, `packed` pairs) to global memory through shared memory: `tile` holds rows of `row_bytes` (128 or
// more), this warp's from `row0` on, its columns from 16-byte group `group0` on; groups are exchanged by the row inside a run of eight.  A lane
// storing its own row touched 32 lines an instruction: 3,700 cycles for 128 columns of eight warps, 700 here.
template <int COLS>
__device__ __forceinline__ void at_put_row(unsigned tile, int row_bytes, int row, int group0, const unsigned* packed) {
#pragma unroll
    for (int j = 0; j < COLS / 8; ++j)
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(tile + row * row_bytes + (((group0 + j) ^ (row & 7)) << 4)), "r"(packed[4 * j]), "r"(packed[4 * j + 1]),
                     "r"(packed[4 * j + 2]), "r"(packed[4 * j + 3]) : "memory");
}
template <int COLS>
__device__ __forceinline__ void at_store_rows(unsigned tile, int row_bytes, int row0, int group0, int rows, bf16* out, size_t stride, int lane, int cols = COLS) {
    constexpr int LANES = COLS / 8, ROWS = 32 / LANES;     // lanes a row, rows at a time
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 32; i += ROWS) {
        const int row = row0 + i + lane / LANES, j = lane % LANES;
        uint4 v;
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(tile + row * row_bytes + (((group0 + j) ^ (row & 7)) << 4)) : "memory");
        if (row < rows && j * 8 < cols) *reinterpret_cast<uint4*>(out + (size_t)row * stride + j * 8) = v;
    }
}
// scores behind the last one a row sees do not count
template <int N>
__device__ __forceinline__ void at_mask_behind(float* s, int last) {
#pragma unroll
    for (int c = 0; c < N; ++c) s[c] = c <= last ? s[c] : -INFINITY;
}

// ---------------------------------------------------------------- host side
namespace {

typedef CUresult (*at_encode_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                 const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

at_encode_fn at_encoder() {
    static at_encode_fn fn = nullptr;
    if (!fn) {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = (at_encode_fn)sym;
    }
    return fn;
}

// a bfloat16 matrix of `rows` rows of `cols` columns, `stride` elements apart, read in boxes of 64 columns x box_rows rows
int at_make_map(CUtensorMap* map, const void* base, long long rows, long long cols, long long stride, int box_rows) {
    at_encode_fn enc = at_encoder();
    if (!enc) return PE_ERR_UNSUPPORTED;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)stride * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : 20000 + (int)r;
}

}  // namespace
