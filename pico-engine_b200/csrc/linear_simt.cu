// out[M, N] = A[M, K] . W[N, K]^T (+ bias[N]) on the CUDA cores: float32 multiply-add for
// every product, whatever the storage dtype of A and W.  This is the matrix product of operands
// that are not stored alike, of small float32 matrices and of a K that is no multiple of eight;
// other float32 products are linear_split.cu's.
//
// K is cut into ranges whose number depends on N and K only.  The sum over k of one output element
// runs in increasing k inside a range, one fused multiply-add per k, and the ranges' sums are added in
// their order, in either kernel and whatever M is: a row's result does not depend on the rows beside it.
//
// pico-engine leaves these products to cuBLAS (src/pico_engine/model.py:177, 213, 223, 235, 164).
#include "common.cuh"

// How many ranges K is cut into.  A product with few columns has few tiles (896 columns and 508 rows: 56 of 64 x 128 for
// 148 SMs), a wide one fills the GPU without; a range of less than 64 entries would cost more in its sum than it saves.
#define LS_MOST_RANGES 8
static int ls_ranges(int N, int K) {
    int s = N <= 2048 ? (K >= 2048 ? 8 : 4) : N <= 12288 ? 2 : 1;
    while (s > 1 && K / s < 64) s /= 2;
    return s;
}
__host__ __device__ __forceinline__ int ls_range_len(int K, int ranges) { return ((K + ranges - 1) / ranges + 15) / 16 * 16; }

// (not .aligned: the lanes of a warp come here from loops that they leave apart)
__device__ __forceinline__ void ls_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ float ls_peer_value(const float* mine, int rank) {          // the same place in the shared memory of CTA `rank`
    unsigned at = (unsigned)__cvta_generic_to_shared(mine), peer;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(at), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(peer) : "memory");
    return v;
}

// the ranges' sums of one place, added in their order (all of them asked for before any is used)
__device__ __forceinline__ float ls_sum(const float* mine, int ranges) {
    float part[LS_MOST_RANGES];
#pragma unroll
    for (int c = 0; c < LS_MOST_RANGES; ++c) part[c] = c < ranges ? ls_peer_value(mine, c) : 0.f;
    float v = part[0] + part[1];
#pragma unroll
    for (int c = 2; c < LS_MOST_RANGES; c += 2)
        if (c < ranges) v = (v + part[c]) + part[c + 1];
    return v;
}

// epilogue: 0 store float32, 1 store bfloat16, 2 add into float32 (the residual stream)
__device__ __forceinline__ void ls_finish(float v, void* out, size_t at, const void* bias, int bias_dtype, int n, int epilogue) {
    if (bias) v += load_as_f(bias, bias_dtype, n);
    if (epilogue == 0) ((float*)out)[at] = v;
    else if (epilogue == 1) ((bf16*)out)[at] = __float2bfloat16_rn(v);
    else ((float*)out)[at] += v;
}

template <typename T>
__device__ __forceinline__ float4 ls_load4(const T* p, int left, bool vec) {           // up to four entries, zeros behind `left`
    if (vec && left >= 4) {
        if constexpr (sizeof(T) == 4) return *reinterpret_cast<const float4*>(p);
        else {
            const uint2 r = *reinterpret_cast<const uint2*>(p);
            const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.y));
            return make_float4(a.x, a.y, b.x, b.y);
        }
    }
    return make_float4(left > 0 ? to_f(p[0]) : 0.f, left > 1 ? to_f(p[1]) : 0.f, left > 2 ? to_f(p[2]) : 0.f, left > 3 ? to_f(p[3]) : 0.f);
}

// ---------------------------------------------------------------------------- many rows
// A CTA of 128 threads: a tile of 64 rows and BN columns over one range of K; a thread 8 x 8 (BN = 128) or 8 x 4 (64) of it, as
// multiply-adds in pairs (fma.rn.f32x2: each half rounds as a plain one does).  Bound by the multiply-adds: a thread reads 16 entries from shared memory
// for 64 of them, a warp's reads of either operand are one broadcast wavefront, and the next 16 (BN = 64: 32) entries of K are on their
// way in registers meanwhile.  The ranges of a tile are a cluster; its CTAs add up a slice of the tile each from the others' shared memory.
// The products of two layers of the Qwen2.5-0.5B widths at 508 rows on a B200: 0.79 ms (38 TFLOP/s); the two layers whole took 3.47 ms
// with tiles of 64 x 64, 4 x 4 a thread and nothing in flight, and 1.53 ms with nothing else changed.
#define LS_BM 64
#define LS_THREADS 128

template <typename TA, typename TW, int LS_BN>
__global__ void __launch_bounds__(LS_THREADS, LS_BN == 128 ? 3 : 4) linear_simt_kernel(const TA* A, const TW* W, const void* bias, int bias_dtype,
                                                                    void* out, int epilogue, int M, int N, int K, int ranges, int vec_a, int vec_w) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int LS_SW = LS_BN + 4, NP = LS_BN / 32;      // NP: pairs of columns a thread
    constexpr int LS_BK = LS_BN == 64 ? 32 : 16, STAGE = LS_BK * (LS_BM + LS_BN);      // entries of K on their way while as many are used
    constexpr int KQ = LS_BK / 4, LR = LS_THREADS / KQ;    // threads that share a row's entries; rows brought at a time
    __shared__ __align__(16) float smem[LS_BM * LS_SW > 2 * STAGE ? LS_BM * LS_SW : 2 * STAGE];
    // row r at entry k: groups of four rows exchanged by k, so that neither a thread's four stores nor four neighbours' reads meet in a bank
    const auto place = [](int k, int r, int width) { return k * width + (r ^ (((k >> 2) & 7) << 2)); };
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ty = (warp >> 1) * 4 + (lane >> 3), tx = (warp & 1) * 8 + (lane & 7);     // rows ty * 4 + 32 i, columns tx * 4 + 64 j
    const int rank = blockIdx.x % ranges, n0 = blockIdx.x / ranges * LS_BN, m0 = blockIdx.y * LS_BM;
    const int len = ls_range_len(K, ranges), k_begin = rank * len, k_end = min(K, k_begin + len);

    unsigned long long acc[8][NP];                         // row i, column pairs
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < NP; ++j) acc[i][j] = 0ull;

    const int lr = tid / KQ, lk = tid % KQ * 4;            // a thread brings four entries of K of rows lr + LR e
    float4 ra[LS_BM / LR], rw[LS_BN / LR];
    auto fetch = [&](int k0) {
        const int left = k_end - k0 - lk;
#pragma unroll
        for (int e = 0; e < LS_BM / LR; ++e) {
            const int m = m0 + lr + LR * e;
            ra[e] = ls_load4(A + (size_t)min(m, M - 1) * K + k0 + lk, m < M ? left : 0, vec_a);
        }
#pragma unroll
        for (int e = 0; e < LS_BN / LR; ++e) {
            const int n = n0 + lr + LR * e;
            rw[e] = ls_load4(W + (size_t)min(n, N - 1) * K + k0 + lk, n < N ? left : 0, vec_w);
        }
    };
    auto put = [&](float* as) {
        float* ws = as + LS_BK * LS_BM;
#pragma unroll
        for (int e = 0; e < LS_BM / LR; ++e) {
            float* p = as + place(lk, lr + LR * e, LS_BM);
            p[0] = ra[e].x; p[LS_BM] = ra[e].y; p[2 * LS_BM] = ra[e].z; p[3 * LS_BM] = ra[e].w;
        }
#pragma unroll
        for (int e = 0; e < LS_BN / LR; ++e) {
            float* p = ws + place(lk, lr + LR * e, LS_BN);
            p[0] = rw[e].x; p[LS_BN] = rw[e].y; p[2 * LS_BN] = rw[e].z; p[3 * LS_BN] = rw[e].w;
        }
    };
    if (k_begin < k_end) {
        fetch(k_begin);
        put(smem);
    }
    __syncthreads();
    for (int k0 = k_begin, b = 0; k0 < k_end; k0 += LS_BK, b ^= 1) {
        const bool more = k0 + LS_BK < k_end;
        if (more) fetch(k0 + LS_BK);
        const float* as = smem + b * STAGE;
        const float* ws = as + LS_BK * LS_BM;
#pragma unroll
        for (int k = 0; k < LS_BK; ++k) {                  // (entries behind the range are zeros: they add nothing)
            float a[8];
            unsigned long long w[NP];
            *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(as + place(k, ty * 4, LS_BM));
            *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(as + place(k, ty * 4, LS_BM) + 32);
#pragma unroll
            for (int j = 0; j < NP; j += 2) *reinterpret_cast<ulonglong2*>(w + j) = *reinterpret_cast<const ulonglong2*>(ws + place(k, tx * 4, LS_BN) + 32 * j);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                unsigned long long aa;
                asm("mov.b64 %0, {%1, %1};" : "=l"(aa) : "f"(a[i]));
#pragma unroll
                for (int j = 0; j < NP; ++j) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(aa), "l"(w[j]));
            }
        }
        if (more) put(smem + (b ^ 1) * STAGE);
        __syncthreads();
    }
    // the tile through shared memory: rows of neighbouring columns go out together, and the other ranges' CTAs can read it
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        float* row = smem + (ty * 4 + 32 * (i / 4) + i % 4) * LS_SW + tx * 4;
#pragma unroll
        for (int j = 0; j < NP; j += 2) *reinterpret_cast<ulonglong2*>(row + 32 * j) = make_ulonglong2(acc[i][j], acc[i][j + 1]);
    }
    if (ranges > 1) ls_cluster_sync(); else __syncthreads();
    const int col = tid % LS_BN, n = n0 + col, rows = LS_BM / ranges;
#pragma unroll 4
    for (int i = tid / LS_BN; i < rows; i += LS_THREADS / LS_BN) {
        const int r = rank * rows + i, m = m0 + r;
        if (m >= M || n >= N) break;
        const float v = ranges == 1 ? smem[r * LS_SW + col] : ls_sum(smem + r * LS_SW + col, ranges);
        ls_finish(v, out, (size_t)m * N + n, bias, bias_dtype, n, epilogue);
    }
    if (ranges > 1) ls_cluster_sync();                     // nobody leaves while its tile is being read
}

// ---------------------------------------------------------------------------- few rows
// Up to 16 rows stream the weights: a CTA takes 32 rows of W over one range of K, its four warps share them and take RT rows of A
// each; a lane has one column.  Float32 operands come by cp.async through a ring of four stages of 64 entries (32 KB a CTA, 3 to 4
// CTAs an SM: what the memory's latency needs in flight), others through registers.
#define LR_BN 32
#define LR_BK 64
#define LR_S (LR_BK + 4)
#define LR_STAGES 4
#define LR_THREADS 128

template <typename TA, typename TW, int RT, bool ASYNC>
__global__ void __launch_bounds__(LR_THREADS) linear_simt_rows_kernel(const TA* A, const TW* W, const void* bias, int bias_dtype,
                                                                      void* out, int epilogue, int M, int N, int K, int ranges) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int MT = 4 * RT, STAGES = ASYNC ? LR_STAGES : 1, STAGE = (LR_BN + MT) * LR_S;
    extern __shared__ __align__(16) float lr_smem[];       // [stage][32 rows of W, MT rows of A][64 + 4]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = blockIdx.x % ranges, n0 = blockIdx.x / ranges * LR_BN;
    const int len = ls_range_len(K, ranges), k_begin = rank * len, k_end = min(K, k_begin + len);
    const int chunks = k_begin < k_end ? (k_end - k_begin + LR_BK - 1) / LR_BK : 0;
    float acc[RT];
#pragma unroll
    for (int i = 0; i < RT; ++i) acc[i] = 0.f;

    auto bring = [&](int c) {
        if (c < chunks) {
            float* dst = lr_smem + (c % STAGES) * STAGE;
            const int k0 = k_begin + c * LR_BK;
            for (int i = tid; i < (LR_BN + MT) * (LR_BK / 4); i += LR_THREADS) {
                const int r = i / (LR_BK / 4), k = i % (LR_BK / 4) * 4, left = k_end - k0 - k;
                const bool is_w = r < LR_BN;
                const int row = is_w ? n0 + r : r - LR_BN;
                float* to = dst + r * LR_S + k;
                const bool there = left > 0 && row < (is_w ? N : M);
                const size_t at = (size_t)row * K + k0 + k;
                if constexpr (ASYNC) {                     // left is a multiple of 4 here
                    const float* src = there ? (is_w ? (const float*)W : (const float*)A) + at : (const float*)W;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"((unsigned)__cvta_generic_to_shared(to)), "l"(src), "r"(there ? 16 : 0) : "memory");
                } else *reinterpret_cast<float4*>(to) = !there ? make_float4(0.f, 0.f, 0.f, 0.f) : is_w ? ls_load4(W + at, left, false) : ls_load4(A + at, left, false);
            }
        }
        if constexpr (ASYNC) asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if constexpr (ASYNC)
        for (int c = 0; c < STAGES - 1; ++c) bring(c);
    for (int c = 0; c < chunks; ++c) {
        if constexpr (ASYNC) asm volatile("cp.async.wait_group %0;" :: "n"(LR_STAGES - 2) : "memory");
        __syncthreads();                                   // chunk c is there for all; the stage of chunk c - 1 is free
        if constexpr (ASYNC) bring(c + STAGES - 1);
        else { bring(c); __syncthreads(); }
        const float* w_row = lr_smem + (c % STAGES) * STAGE + lane * LR_S;
        const float* a_row = lr_smem + (c % STAGES) * STAGE + (LR_BN + warp * RT) * LR_S;
#pragma unroll
        for (int k = 0; k < LR_BK; k += 4) {
            const float4 w = *reinterpret_cast<const float4*>(w_row + k);
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(a_row + i * LR_S + k);
                acc[i] = fmaf(a.x, w.x, acc[i]); acc[i] = fmaf(a.y, w.y, acc[i]);
                acc[i] = fmaf(a.z, w.z, acc[i]); acc[i] = fmaf(a.w, w.w, acc[i]);
            }
        }
    }
    const int n = n0 + lane;
    if (ranges == 1) {
#pragma unroll
        for (int i = 0; i < RT; ++i) {
            const int m = warp * RT + i;
            if (m < M && n < N) ls_finish(acc[i], out, (size_t)m * N + n, bias, bias_dtype, n, epilogue);
        }
        return;
    }
    __syncthreads();                                       // (the last chunk has been read: its place takes the sums)
    if constexpr (ASYNC) asm volatile("cp.async.wait_group 0;" ::: "memory");
    float* sums = lr_smem;                                 // [MT][32]
    __syncthreads();
#pragma unroll
    for (int i = 0; i < RT; ++i) sums[(warp * RT + i) * LR_BN + lane] = acc[i];
    ls_cluster_sync();
    for (int m = warp * ranges + rank; m < MT; m += 4 * ranges) {      // the rows dealt out to the cluster's warps
        if (m >= M || n >= N) break;
        ls_finish(ls_sum(sums + m * LR_BN + lane, ranges), out, (size_t)m * N + n, bias, bias_dtype, n, epilogue);
    }
    ls_cluster_sync();
}

// ---------------------------------------------------------------------------- a short K
// Up to 16 entries of K, or 32 and few results: the product is its operands' way in and the result's way out, and the kernels above, made to keep 8 x 8 sums and the
// next entries of K a thread, only start later.  A block of 256 threads: 64 x 64 results, 4 x 4 a thread.  16 entries of K, 2,048
// columns on a B200, tiles above / here: 17 rows 3.5 / 2.7 us, 64 rows 5.0 / 2.9, 300 rows 6.5 / 4.1, 1,000 rows 8.1 / 7.1; 32 entries:
// 64 rows 4.8 / 4.3 us, 300 rows 6.4 / 6.5, 1,000 rows 8.1 / 12.5.
#define LK_SHORT 16
#define LK_LONG 32
#define LK_B 64
#define LK_K 16

template <typename TA, typename TW>
__global__ void __launch_bounds__(256) linear_simt_short_kernel(const TA* A, const TW* W,
                                                          const void* bias, int bias_dtype,
                                                          void* out, int epilogue, int M, int N, int K) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float As[LK_K][LK_B + 4];
    __shared__ float Ws[LK_K][LK_B + 4];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * LK_B, n0 = blockIdx.x * LK_B;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

    const int lrow = tid >> 2, lk = (tid & 3) * 4;      // each thread loads 4 consecutive k of one row
    for (int k0 = 0; k0 < K; k0 += LK_K) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int k = k0 + lk + e;
            const int am = m0 + lrow, wn = n0 + lrow;
            As[lk + e][lrow] = (am < M && k < K) ? to_f(A[(size_t)am * K + k]) : 0.f;
            Ws[lk + e][lrow] = (wn < N && k < K) ? to_f(W[(size_t)wn * K + k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < LK_K; ++k) {
            const float4 a = *reinterpret_cast<const float4*>(&As[k][ty * 4]);
            const float4 w = *reinterpret_cast<const float4*>(&Ws[k][tx * 4]);
            const float av[4] = {a.x, a.y, a.z, a.w}, wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n >= N) continue;
            ls_finish(acc[i][j], out, (size_t)m * N + n, bias, bias_dtype, n, epilogue);
        }
    }
}

template <typename TA, typename TW, int RT, bool ASYNC>
static int ls_rows(const void* A, const void* W, const void* bias, int bias_dtype, void* out, int epilogue, int M, int N, int K, int ranges, cudaStream_t s) {
    const size_t smem = (size_t)(ASYNC ? LR_STAGES : 1) * (LR_BN + 4 * RT) * LR_S * 4;
    auto kernel = linear_simt_rows_kernel<TA, TW, RT, ASYNC>;
    if (smem > 48 * 1024) PE_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    PE_TRY(pe_launch_cluster(kernel, dim3((N + LR_BN - 1) / LR_BN * ranges), LR_THREADS, smem, s, ranges, (const TA*)A, (const TW*)W, bias, bias_dtype,
                             out, epilogue, M, N, K, ranges));
    PE_LAUNCH_CHECK();
    return 0;
}

template <typename TA, typename TW>
static int ls_go(const void* A, const void* W, const void* bias, int bias_dtype, void* out, int epilogue, int M, int N, int K, cudaStream_t s) {
    const int ranges = ls_ranges(N, K);
    const auto vec = [K](const void* p, size_t size) { return (int)(K % 4 == 0 && (uintptr_t)p % (4 * size) == 0); };
    const int vec_a = vec(A, sizeof(TA)), vec_w = vec(W, sizeof(TW));
    if (K <= LK_LONG && (K <= LK_SHORT || (long long)M * N <= 500000)) {       // (one range: the same sums as in the other kernels)
        const int mt = (M + LK_B - 1) / LK_B;
        if (mt > 65535) return PE_ERR_UNSUPPORTED;
        PE_TRY(pe_launch(linear_simt_short_kernel<TA, TW>, dim3((N + LK_B - 1) / LK_B, mt), 256, 0, s, (const TA*)A, (const TW*)W, bias, bias_dtype, out, epilogue, M, N, K));
        PE_LAUNCH_CHECK();
        return 0;
    }
    // The line between the kernels: a tile of 64 rows costs the same however few of them there are.
    if (M <= 16) {
        if constexpr (sizeof(TA) == 4 && sizeof(TW) == 4)
            if (vec_a && vec_w) return M <= 4 ? ls_rows<TA, TW, 1, true>(A, W, bias, bias_dtype, out, epilogue, M, N, K, ranges, s)
                                     : M <= 8 ? ls_rows<TA, TW, 2, true>(A, W, bias, bias_dtype, out, epilogue, M, N, K, ranges, s)
                                              : ls_rows<TA, TW, 4, true>(A, W, bias, bias_dtype, out, epilogue, M, N, K, ranges, s);
        return ls_rows<TA, TW, 4, false>(A, W, bias, bias_dtype, out, epilogue, M, N, K, ranges, s);
    }
    const int mt = (M + LS_BM - 1) / LS_BM;
    if (mt > 65535) return PE_ERR_UNSUPPORTED;
#define LS_TILES(BN) PE_TRY(pe_launch_cluster(linear_simt_kernel<TA, TW, BN>, dim3((N + BN - 1) / BN * ranges, mt), LS_THREADS, 0, s, ranges, (const TA*)A, \
                                              (const TW*)W, bias, bias_dtype, out, epilogue, M, N, K, ranges, vec_a, vec_w))
    // Tiles of 64 columns where those of 128 would leave an SM with fewer than four CTAs: with so few, one more or less is what a product
    // waits for.  Measured on a B200, columns x K, 64 wide / 128 wide: 60 rows 1152 x 896 13 / 20 us, 896 x 4864 30 / 42 us; 508 rows
    // 1152 x 896 35 / 40, 896 x 896 30 / 39, 896 x 4864 113 / 127 (all below the line); 9728 x 896 215 / 205 (above it).
    if ((long long)((N + 127) / 128) * ranges * mt < 4 * 148) LS_TILES(64);
    else LS_TILES(128);
#undef LS_TILES
    PE_LAUNCH_CHECK();
    return 0;
}

extern "C" int pe_linear_simt(const void* A, int a_dtype, const void* W, int w_dtype, const void* bias, int bias_dtype,
                              void* out, int epilogue, int M, int N, int K, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || epilogue < 0 || epilogue > 2) return PE_ERR_UNSUPPORTED;
    cudaStream_t s = (cudaStream_t)stream;
#define LS_GO(TA, TW) return ls_go<TA, TW>(A, W, bias, bias_dtype, out, epilogue, M, N, K, s)
    if (a_dtype == PE_F32 && w_dtype == PE_F32) LS_GO(float, float);
    if (a_dtype == PE_BF16 && w_dtype == PE_BF16) LS_GO(bf16, bf16);
    if (a_dtype == PE_BF16 && w_dtype == PE_F32) LS_GO(bf16, float);
    if (a_dtype == PE_F32 && w_dtype == PE_BF16) LS_GO(float, bf16);
#undef LS_GO
    return PE_ERR_UNSUPPORTED;
}
