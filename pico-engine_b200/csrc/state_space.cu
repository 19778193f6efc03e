// A selective state-space mixer with a scalar decay a head and token: the short causal convolution with silu on its inputs,
// the recurrence, and the gate followed by a norm over groups of channels.  Decays, step sizes, the state, its outputs, the
// gate and the norm are float32 in either engine dtype; only the loads of projections and the store of the result convert.
//
//   dt_t = softplus(dt_raw_t + dt_bias_h)        a_t = exp(-exp(A_log_h) * dt_t)
//   S_t = a_t S_(t-1) + dt_t B_t x_t^T           (S [N, P] a head, B and C shared by the heads of a group)
//   y_t = S_t^T C_t + D_h x_t
//
// The recurrence runs token after token: a block owns (sequence, head, a tile of the P columns); thread (p, ns) keeps rows
// n = ns NR + r (r < NR) of column p in registers (B and C are read from shared memory four rows at a time), the NS threads of a
// column are neighbours in a warp and add their parts of y by shuffles.  Prompts run as products of tiles (state_space_tiles.cu).
// A sequence's state lies in its row of the cache's state area in exactly the order the threads hold it,
// element ((h * NR + r) * P + p) * NS + ns, so it is read and written in whole lines; rows n >= N are padding and stay zero.
// NS depends on N alone (the smallest power of two that leaves a thread at most 16 rows), so a model's layout never changes.
#include "state_space.cuh"

extern "C" void pe_set_pdl(int on) { pe_pdl_enabled() = on ? 1 : 0; }     // (this library's own copy of the switch)

#define SS_TOKENS 8          // tokens whose B, C, x, dt are staged in shared memory at a time

// ---------------------------------------------------------------- convolution + silu
// in: columns c_off .. c_off + C - 1 of proj [T, ld] (the step's dtype).  out [T, C] float32:
// silu(bias[c] + sum_j w[c, j] * u_(t - taps + 1 + j)[c]); inputs before the step's first token come from the sequence's state
// (entry k: the input k + 1 places before the next step's first token), inputs before the sequence's start are zero (the state of a
// new sequence is zero).
template <typename T>
__global__ void conv_silu_kernel(const T* proj, int ld, int c_off, int C, int taps, const void* w, int w_dtype, const void* bias,
                                 int b_dtype, const float* state, long long state_stride, const int* tok_row, const int* row_first,
                                 const int* slots, float* out, size_t total) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= total) return;
    const int t = (int)(e / C), c = (int)(e % C);
    const int b = tok_row[t], i = t - row_first[b];              // the token's place within its row's tokens of this step
    const float* st = state + (size_t)slots[b] * state_stride;
    float acc = bias ? load_as_f(bias, b_dtype, c) : 0.f;
    for (int j = 0; j < taps; ++j) {
        const int back = taps - 1 - j;                           // 0: the token itself
        const float v = back <= i ? to_f(proj[(size_t)(t - back) * ld + c_off + c]) : st[(size_t)(back - i - 1) * C + c];
        acc = fmaf(load_as_f(w, w_dtype, (size_t)c * taps + j), v, acc);
    }
    out[e] = ss_silu(acc);
}

// Runs of four channels: a thread takes CONV_TOKENS neighbouring tokens of them, all asked for at once, and hands each token's inputs on
// to the next ones, so that an input is read once (and `taps` - 1 times more at the front of a run) where the kernel above reads it
// `taps` times, with a division an element to find its place.  The sums run in the same order.  Where the run and the inputs in front of
// it lie in one row, those are asked for together with the run's own: places and states, three reads one behind the other, are
// looked up only where a row begins.  Weights come four at a time, as far as L2 before the wait for the kernel in front (which may be writing them).  2,047 tokens of
// 4,608 channels, bfloat16, on a B200: 79 us by the kernel above, 23.3 with the look-up for each run and single weights, 20.1 here.
#define CONV_TOKENS 8
__device__ __forceinline__ float4 ss_read4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 ss_read4(const bf16* p) {
    const uint2 r = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ float4 ss_weights4(const void* p, int dtype, size_t i) {       // entries i .. i + 3, i a multiple of four
    if (dtype == PE_BF16 && ((uintptr_t)p & 7) == 0) return ss_read4((const bf16*)p + i);
    if (dtype == PE_F32 && ((uintptr_t)p & 15) == 0) return ss_read4((const float*)p + i);
    return make_float4(load_as_f(p, dtype, i), load_as_f(p, dtype, i + 1), load_as_f(p, dtype, i + 2), load_as_f(p, dtype, i + 3));
}
template <typename T, int TAPS>
__global__ void __launch_bounds__(128) conv_silu_vec_kernel(const T* proj, int ld, int c_off, int C, const void* w, int w_dtype, const void* bias,
                                                            int b_dtype, const float* state, long long state_stride, const int* tok_row,
                                                            const int* row_first, const int* slots, float* out, int n_tok) {
    pdl_launch_dependents();
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 4, t0 = blockIdx.y * CONV_TOKENS, m = min(CONV_TOKENS, n_tok - t0);
    if (c >= C) return;
    const unsigned w_size = w_dtype == PE_BF16 ? 2 : 4, b_size = b_dtype == PE_BF16 ? 2 : 4;
    asm volatile("prefetch.global.L2 [%0];" ::"l"((const char*)w + (size_t)c * TAPS * w_size) : "memory");
    if (bias) asm volatile("prefetch.global.L2 [%0];" ::"l"((const char*)bias + (size_t)c * b_size) : "memory");
    pdl_wait();
    __align__(16) float flat[4 * TAPS], b4[4];                   // channel c + e, weight j: flat[e * TAPS + j]
#pragma unroll
    for (int q = 0; q < TAPS; ++q) *reinterpret_cast<float4*>(flat + 4 * q) = ss_weights4(w, w_dtype, (size_t)c * TAPS + 4 * q);
    *reinterpret_cast<float4*>(b4) = bias ? ss_weights4(bias, b_dtype, c) : make_float4(0.f, 0.f, 0.f, 0.f);
    const T* src = proj + (size_t)t0 * ld + c_off + c;
    float4 in[CONV_TOKENS], past[TAPS];                          // past[k]: the input k + 1 places back
    const int front = t0 - (TAPS - 1), last = tok_row[t0 + m - 1];
    const bool inside = front >= 0 && tok_row[max(front, 0)] == last;      // (a row's tokens stand together)
#pragma unroll
    for (int u = 0; u < CONV_TOKENS; ++u)
        if (u < m) in[u] = ss_read4(src + (size_t)u * ld);
    if (front >= 0) {
#pragma unroll
        for (int k = 0; k < TAPS - 1; ++k) past[k] = ss_read4(proj + (size_t)(t0 - k - 1) * ld + c_off + c);
    }
    int row = inside ? last : -1;
#pragma unroll
    for (int u = 0; u < CONV_TOKENS; ++u) {
        if (u >= m) break;
        const int t = t0 + u, b = inside ? last : tok_row[t];
        if (b != row) {
            const int i = t - row_first[b];                      // the token's place within its row's tokens of this step
            const float* st = state + (size_t)slots[b] * state_stride + c;
#pragma unroll
            for (int k = 0; k < TAPS - 1; ++k) {
                if (k + 1 <= i) past[k] = ss_read4(proj + (size_t)(t - k - 1) * ld + c_off + c);
                else past[k] = make_float4(st[(size_t)(k - i) * C], st[(size_t)(k - i) * C + 1], st[(size_t)(k - i) * C + 2], st[(size_t)(k - i) * C + 3]);
            }
            row = b;
        }
        float4 acc = make_float4(b4[0], b4[1], b4[2], b4[3]);
#pragma unroll
        for (int j = 0; j < TAPS; ++j) {
            const float4 v = j == TAPS - 1 ? in[u] : past[TAPS - 2 - j];
            acc.x = fmaf(flat[j], v.x, acc.x); acc.y = fmaf(flat[1 * TAPS + j], v.y, acc.y);
            acc.z = fmaf(flat[2 * TAPS + j], v.z, acc.z); acc.w = fmaf(flat[3 * TAPS + j], v.w, acc.w);
        }
        *reinterpret_cast<float4*>(out + (size_t)t * C + c) = make_float4(ss_silu(acc.x), ss_silu(acc.y), ss_silu(acc.z), ss_silu(acc.w));
#pragma unroll
        for (int k = TAPS - 2; k > 0; --k) past[k] = past[k - 1];
        past[0] = in[u];
    }
}
template <typename T>
static int conv_silu_vec(const T* proj, int ld, int c_off, int C, int taps, const void* w, int w_dtype, const void* bias, int b_dtype,
                         const float* state, long long state_stride, const int* tok_row, const int* row_first, const int* slots, float* out,
                         int n_tok, cudaStream_t s) {
    const dim3 grid((C / 4 + 127) / 128, (n_tok + CONV_TOKENS - 1) / CONV_TOKENS);
#define CONV_GO(TAPS) PE_TRY(pe_launch(conv_silu_vec_kernel<T, TAPS>, grid, 128, 0, s, proj, ld, c_off, C, w, w_dtype, bias, b_dtype, state, state_stride, tok_row, row_first, slots, out, n_tok))
    if (taps == 2) CONV_GO(2);
    else if (taps == 3) CONV_GO(3);
    else CONV_GO(4);
#undef CONV_GO
    PE_LAUNCH_CHECK();
    return 0;
}

// New state from the step's inputs: entry k <- the input of the step's token n - 1 - k, or, where the step brought fewer tokens,
// the old entry k - n.  Entries are rewritten from the oldest to the newest, so an old entry is read before it is overwritten.
template <typename T>
__global__ void conv_state_kernel(const T* proj, int ld, int c_off, int C, int taps, float* state, long long state_stride,
                                  const int* row_first, const int* row_lens, const int* slots) {
    pdl_launch_dependents();
    pdl_wait();
    const int b = blockIdx.x;
    const int n = row_lens[b], first = row_first[b];
    float* st = state + (size_t)slots[b] * state_stride;
    for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < C; c += gridDim.y * blockDim.x)
        for (int k = taps - 2; k >= 0; --k)
            st[(size_t)k * C + c] = k < n ? to_f(proj[(size_t)(first + n - 1 - k) * ld + c_off + c]) : st[(size_t)(k - n) * C + c];
}

extern "C" int pe_conv_silu(const void* proj, int dtype, int ld, int c_off, int C, int taps, const void* w, int w_dtype, const void* bias,
                            int b_dtype, float* state, long long state_stride, const int* tok_row, const int* row_first,
                            const int* row_lens, const int* slots, float* out, int T, int B, void* stream) {
    if (T <= 0) return 0;
    if (taps < 1 || C <= 0 || c_off < 0 || c_off + C > ld) return PE_ERR_UNSUPPORTED;
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype != PE_F32 && dtype != PE_BF16) return PE_ERR_UNSUPPORTED;
    const size_t total = (size_t)T * C, size = dtype == PE_F32 ? 4 : 2;
    const unsigned blocks = (unsigned)((total + 255) / 256);
    // Runs of four channels where they can be read and written at once (grid.y holds up to 65,535 runs of tokens) and where there are enough
    // of them: a thread's eight tokens wait for one another's rows, which the kernel above takes side by side.  Measured on a B200, above /
    // runs: 1 row of 17 tokens x 4,608 channels 4.3 / 6.7 us, of 100 7.0 / 6.8, of 128 7.9 / 6.8, of 400 17.4 / 8.1; 8 x 1 4.4 / 10.0, 64 x 1
    // 6.8 / 12.5, 64 x 2 9.1 / 10.5, 64 x 4 13.4 / 9.6; 128 x 1 of 10,000 19.4 / 17.3.
    const bool vec = taps >= 2 && taps <= 4 && C % 4 == 0 && c_off % 4 == 0 && ld % 4 == 0 && (uintptr_t)proj % (4 * size) == 0 &&
                     (uintptr_t)out % 16 == 0 && (T + CONV_TOKENS - 1) / CONV_TOKENS <= 65535 && total >= (T >= 8 * B ? 500000u : 1000000u);
    if (vec) {
        const int rc = dtype == PE_F32 ? conv_silu_vec((const float*)proj, ld, c_off, C, taps, w, w_dtype, bias, b_dtype, state, state_stride, tok_row, row_first, slots, out, T, s)
                                       : conv_silu_vec((const bf16*)proj, ld, c_off, C, taps, w, w_dtype, bias, b_dtype, state, state_stride, tok_row, row_first, slots, out, T, s);
        if (rc) return rc;
    } else if (dtype == PE_F32) PE_TRY(pe_launch(conv_silu_kernel<float>, blocks, 256, 0, s, (const float*)proj, ld, c_off, C, taps, w, w_dtype, bias, b_dtype, (const float*)state, state_stride, tok_row, row_first, slots, out, total));
    else PE_TRY(pe_launch(conv_silu_kernel<bf16>, blocks, 256, 0, s, (const bf16*)proj, ld, c_off, C, taps, w, w_dtype, bias, b_dtype, (const float*)state, state_stride, tok_row, row_first, slots, out, total));
    PE_LAUNCH_CHECK();
    if (taps > 1) {
        if (dtype == PE_F32) PE_TRY(pe_launch(conv_state_kernel<float>, dim3(B, (C + 255) / 256), 256, 0, s, (const float*)proj, ld, c_off, C, taps, state, state_stride, row_first, row_lens, slots));
        else PE_TRY(pe_launch(conv_state_kernel<bf16>, dim3(B, (C + 255) / 256), 256, 0, s, (const bf16*)proj, ld, c_off, C, taps, state, state_stride, row_first, row_lens, slots));
        PE_LAUNCH_CHECK();
    }
    return 0;
}

// ---------------------------------------------------------------- the recurrence
extern "C" int pe_state_space_split(int N) {
    int ns = 1;
    while ((N + ns - 1) / ns > 16 && ns < 32) ns *= 2;
    return ns;
}
// float32 numbers of a sequence's state for these sizes (with the padding rows)
extern "C" long long pe_state_space_elems(int H, int P, int N) {
    const int ns = pe_state_space_split(N);
    return (long long)H * ((N + ns - 1) / ns) * ns * P;
}
// Chunks a step of T tokens in B sequences can have at most; those that are worked on at a time, as many as SS_SCRATCH_FLOATS of scratch
// hold (one at least), in slabs of equal size; and the floats of scratch that a slab needs.  A slab of the sizes that fill it keeps the GPU
// full (64 heads of 64 columns, 128 state rows: 101 chunks on the tensor cores, 3,232 units of two heads a launch), and batches of prompts need no more scratch than it.
#define SS_SCRATCH_FLOATS (64ll << 20)
extern "C" int pe_state_space_chunks(int T, int B) { return (T + SS_CHUNK - 1) / SS_CHUNK + B; }
static int ss_step_floats(int H, int P, int N, int G) { return ss_on_tensor_cores(H, P, N, G) ? SS_MATRIX_STEP_FLOATS : SS_STEP_FLOATS; }
static long long ss_chunk_floats(int H, int P, int N, int G) {
    const long long parts = ss_on_tensor_cores(H, P, N, G) ? (long long)G * (2 * ss_plane_bytes(N) / 4 + 1) + H / 2 : 0;
    return (long long)G * SS_CHUNK * SS_CHUNK + (long long)H * (P * N + ss_step_floats(H, P, N, G) + 1) + 8 + parts;
}
static int ss_slab(int chunks, int H, int P, int N, int G) {
    const long long floats = ss_chunk_floats(H, P, N, G), most = floats >= SS_SCRATCH_FLOATS ? 1 : SS_SCRATCH_FLOATS / floats;
    const long long slabs = (chunks + most - 1) / most;
    return (int)((chunks + slabs - 1) / slabs);
}
extern "C" int pe_state_space_slabs(int T, int B, int H, int P, int N, int G) {
    const int chunks = pe_state_space_chunks(T, B), slab = ss_slab(chunks, H, P, N, G);
    return (chunks + slab - 1) / slab;
}
extern "C" long long pe_state_space_scratch_floats(int T, int B, int H, int P, int N, int G) {
    return ss_slab(pe_state_space_chunks(T, B), H, P, N, G) * ss_chunk_floats(H, P, N, G);
}

// A sequence's tokens one after the other, from its stored state.
template <typename T, int NRMAX>
__global__ void __launch_bounds__(256) scan_kernel(ScanArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float ss_smem[];
    const int h = blockIdx.y, p0 = blockIdx.z * a.PT;
    const int N = a.N, P = a.P, NS = a.NS, NR = a.NR, NRP = a.NRP, PT = a.PT, ROW = NS * NRP;
    const int tid = threadIdx.x, ns = tid % NS, pl = tid / NS, p = p0 + pl;
    const bool on = pl < PT && p < P;
    const int g = h / (a.H / a.G), inner = a.H * P;
    float* Bs = ss_smem;                      // [SS_TOKENS][ROW]: row n = s NR + r at s NRP + r (a thread's rows side by side, padded)
    float* Cs = Bs + SS_TOKENS * ROW;         // [SS_TOKENS][ROW]
    float* xs = Cs + SS_TOKENS * ROW;         // [SS_TOKENS][PT]
    float* dts = xs + SS_TOKENS * PT;         // [SS_TOKENS]: step sizes
    float* das = dts + SS_TOKENS;             // [SS_TOKENS]: decays
    const int b = blockIdx.x, first = a.row_first[b], n_tok = a.row_lens[b];
    if (n_tok <= 0) return;
    float* st = a.state + (size_t)a.slots[b] * a.state_stride + (size_t)h * NR * P * NS;
    float S[NRMAX];
#pragma unroll
    for (int r = 0; r < NRMAX; ++r) S[r] = (on && r < NR) ? st[((size_t)r * P + p) * NS + ns] : 0.f;
    const float A = expf(load_as_f(a.a_log, a.al_dtype, h)), Dh = load_as_f(a.d_skip, a.d_dtype, h), dtb = load_as_f(a.dt_bias, a.dtb_dtype, h);
    const T* proj = (const T*)a.proj;
    for (int c0 = 0; c0 < n_tok; c0 += SS_TOKENS) {
        const int nc = min(SS_TOKENS, n_tok - c0);
        __syncthreads();                                       // the group before has been walked
        for (int e = tid; e < nc * ROW; e += blockDim.x) {
            const int i = e / ROW, w = e % ROW, s = w / NRP, r = w % NRP, n = s * NR + r;
            const bool there = r < NR && n < N;
            const float* row = a.xbc + (size_t)(first + c0 + i) * a.xbc_ld;
            Bs[e] = there ? row[inner + g * N + n] : 0.f;
            Cs[e] = there ? row[inner + a.G * N + g * N + n] : 0.f;
        }
        for (int e = tid; e < nc * PT; e += blockDim.x) {
            const int i = e / PT, q = e % PT;
            xs[i * PT + q] = p0 + q < P ? a.xbc[(size_t)(first + c0 + i) * a.xbc_ld + h * P + p0 + q] : 0.f;
        }
        if (tid < nc) {
            const float dt = ss_softplus(to_f(proj[(size_t)(first + c0 + tid) * a.proj_ld + a.dt_off + h]) + dtb);
            dts[tid] = dt;
            das[tid] = expf(-A * dt);
        }
        __syncthreads();
        for (int i = 0; i < nc; ++i) {
            const float x = xs[i * PT + (on ? pl : 0)];
            const float da = das[i], dtx = dts[i] * x;
            const float4* B4 = reinterpret_cast<const float4*>(Bs + i * ROW + ns * NRP);
            const float4* C4 = reinterpret_cast<const float4*>(Cs + i * ROW + ns * NRP);
            float acc0 = 0.f, acc1 = 0.f;
#pragma unroll
            for (int r = 0; r < NRMAX; r += 4) {
                if (r < NR) {                                  // rows NR .. of the last four meet zeros of B and C and stay zero
                    const float4 bv = B4[r / 4];
                    S[r + 0] = fmaf(da, S[r + 0], dtx * bv.x); S[r + 1] = fmaf(da, S[r + 1], dtx * bv.y);
                    S[r + 2] = fmaf(da, S[r + 2], dtx * bv.z); S[r + 3] = fmaf(da, S[r + 3], dtx * bv.w);
                    const float4 cv = C4[r / 4];
                    acc0 = fmaf(S[r + 0], cv.x, acc0); acc1 = fmaf(S[r + 1], cv.y, acc1);
                    acc0 = fmaf(S[r + 2], cv.z, acc0); acc1 = fmaf(S[r + 3], cv.w, acc1);
                }
            }
            float acc = acc0 + acc1;
            for (int o = 1; o < NS; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (on && ns == 0) a.y[(size_t)(first + c0 + i) * inner + h * P + p] = fmaf(Dh, x, acc);
        }
    }
    if (on) {
#pragma unroll
        for (int r = 0; r < NRMAX; ++r)
            if (r < NR) st[((size_t)r * P + p) * NS + ns] = S[r];
    }
}

template <typename T, int NRMAX>
static int scan_run(const ScanArgs& a, int threads, size_t smem, cudaStream_t s) {
    PE_TRY(pe_launch(scan_kernel<T, NRMAX>, dim3(a.B, a.H, (a.P + a.PT - 1) / a.PT), threads, smem, s, a));
    PE_LAUNCH_CHECK();
    return 0;
}

extern "C" int pe_state_space_scan(const float* xbc, int xbc_ld, const void* proj, int dtype, int proj_ld, int dt_off, const void* dt_bias,
                                   int dtb_dtype, const void* a_log, int al_dtype, const void* d_skip, int d_dtype, float* state,
                                   long long state_stride, const int* row_first, const int* row_lens, const int* slots, float* y,
                                   int T, int B, int H, int P, int N, int G, int chunked, float* scratch, int* status, void* stream) {
    if (B <= 0 || T <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G || P <= 0 || N <= 0 || N > 512) return PE_ERR_UNSUPPORTED;
    if (chunked && !scratch) return PE_ERR_UNSUPPORTED;
    const int NS = pe_state_space_split(N), NR = (N + NS - 1) / NS, NRP = (NR + 3) / 4 * 4 + 4;
    int PT = 256 / NS;
    if (PT > P) PT = P;
    int threads = ((PT * NS + 31) / 32) * 32;
    ScanArgs a = {xbc, xbc_ld, proj, proj_ld, dt_off, dt_bias, dtb_dtype, a_log, al_dtype, d_skip, d_dtype, state, state_stride,
                  row_first, row_lens, slots, y, B, H, P, N, G, NS, NR, NRP, PT, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, 0, 0, 0};
    if (dtype != PE_F32 && dtype != PE_BF16) return PE_ERR_UNSUPPORTED;
    if (chunked) {
        a.chunks = pe_state_space_chunks(T, B);
        a.slab = ss_slab(a.chunks, H, P, N, G);
        a.chunk_steps = scratch;                                  // (64-bit entries and vectors of eight first; eight floats for a chunk's place)
        const int step_floats = ss_step_floats(H, P, N, G);
        a.chunk_rows = reinterpret_cast<int2*>(scratch + (size_t)a.slab * H * step_floats);
        a.chunk_scores = scratch + (size_t)a.slab * (H * step_floats + 8);
        a.chunk_state = a.chunk_scores + (size_t)a.slab * G * SS_CHUNK * SS_CHUNK;
        a.chunk_decay = a.chunk_state + (size_t)a.slab * H * P * N;
        if (ss_on_tensor_cores(H, P, N, G)) {
            if (!status) return PE_ERR_UNSUPPORTED;
            a.chunk_planes = reinterpret_cast<unsigned char*>(a.chunk_decay);                                     // (vectors first)
            a.chunk_decay = reinterpret_cast<float*>(a.chunk_planes + (size_t)a.slab * G * 2 * ss_plane_bytes(N));
            a.chunk_seen = reinterpret_cast<unsigned*>(a.chunk_decay + (size_t)a.slab * H);
            a.unit_exact = reinterpret_cast<int*>(a.chunk_seen + (size_t)a.slab * G);
            return ss_tensor_tiles(a, dtype, status, (cudaStream_t)stream);
        }
        return ss_tiles(a, dtype, (cudaStream_t)stream);
    }
    const size_t smem = sizeof(float) * ((size_t)SS_TOKENS * (2 * NS * NRP + PT) + 2 * SS_TOKENS);
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == PE_F32) return NR <= 8 ? scan_run<float, 8>(a, threads, smem, s) : scan_run<float, 16>(a, threads, smem, s);
    return NR <= 8 ? scan_run<bf16, 8>(a, threads, smem, s) : scan_run<bf16, 16>(a, threads, smem, s);
}

// ---------------------------------------------------------------- gate, then a norm over groups of channels
// y [T, C] float32, the gate z at columns z_off .. of proj [T, ld] (the step's dtype): u = y * silu(z); every run of `group`
// channels of u is divided by sqrt(mean(run^2) + eps) and multiplied by weight[channel]; out [T, C] in the step's dtype.
// A block a (token, run).
template <typename T>
__global__ void __launch_bounds__(256) gate_norm_kernel(const float* y, int C, int group, const T* proj, int ld, int z_off, const void* weight,
                                                        int w_dtype, float eps, T* out) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float red[33];
    const int t = blockIdx.x, c0 = blockIdx.y * group;
    float ss = 0.f;
    for (int i = threadIdx.x; i < group; i += blockDim.x) {
        const float u = y[(size_t)t * C + c0 + i] * ss_silu(to_f(proj[(size_t)t * ld + z_off + c0 + i]));
        ss = fmaf(u, u, ss);
    }
    const float rstd = 1.0f / sqrtf(block_sum(ss, red) / (float)group + eps);
    for (int i = threadIdx.x; i < group; i += blockDim.x) {
        const float u = y[(size_t)t * C + c0 + i] * ss_silu(to_f(proj[(size_t)t * ld + z_off + c0 + i]));
        out[(size_t)t * C + c0 + i] = from_f<T>(u * rstd * load_as_f(weight, w_dtype, c0 + i));
    }
}

// Runs of up to 4,096 channels, four at a time, kept in registers between the two passes.  2,047 tokens, two runs of 2,048
// channels, bfloat16, on a B200: 15 us.
template <typename T, int NV>
__global__ void __launch_bounds__(256) gate_norm_vec_kernel(const float* y, int C, int group, const T* proj, int ld, int z_off, const void* weight,
                                                            int w_dtype, float eps, T* out) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float red[33];
    const int t = blockIdx.x, c0 = blockIdx.y * group;
    float4 u[NV], z[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int i = (k * blockDim.x + threadIdx.x) * 4;
        if (i < group) { u[k] = ss_read4(y + (size_t)t * C + c0 + i); z[k] = ss_read4(proj + (size_t)t * ld + z_off + c0 + i); }
    }
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        if ((k * blockDim.x + threadIdx.x) * 4 < group) {
            u[k] = make_float4(u[k].x * ss_silu(z[k].x), u[k].y * ss_silu(z[k].y), u[k].z * ss_silu(z[k].z), u[k].w * ss_silu(z[k].w));
            ss = fmaf(u[k].x, u[k].x, ss); ss = fmaf(u[k].y, u[k].y, ss); ss = fmaf(u[k].z, u[k].z, ss); ss = fmaf(u[k].w, u[k].w, ss);
        }
    }
    const float rstd = 1.0f / sqrtf(block_sum(ss, red) / (float)group + eps);
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int i = (k * blockDim.x + threadIdx.x) * 4;
        if (i >= group) continue;
        T* to = out + (size_t)t * C + c0 + i;
        const float4 v = make_float4(u[k].x * rstd * load_as_f(weight, w_dtype, c0 + i), u[k].y * rstd * load_as_f(weight, w_dtype, c0 + i + 1),
                                     u[k].z * rstd * load_as_f(weight, w_dtype, c0 + i + 2), u[k].w * rstd * load_as_f(weight, w_dtype, c0 + i + 3));
        if constexpr (sizeof(T) == 4) *reinterpret_cast<float4*>(to) = v;
        else {
            __nv_bfloat162 p[2] = {__floats2bfloat162_rn(v.x, v.y), __floats2bfloat162_rn(v.z, v.w)};
            *reinterpret_cast<uint2*>(to) = *reinterpret_cast<const uint2*>(p);
        }
    }
}
template <typename T>
static int gate_norm_vec(const float* y, int T_, int C, int group, const T* proj, int ld, int z_off, const void* weight, int w_dtype, float eps,
                         T* out, cudaStream_t s) {
    const dim3 grid(T_, C / group);
    const int threads = group >= 1024 ? 256 : ((group / 4 + 31) / 32) * 32;
#define GN_GO(NV) PE_TRY(pe_launch(gate_norm_vec_kernel<T, NV>, grid, threads, 0, s, y, C, group, proj, ld, z_off, weight, w_dtype, eps, out))
    if (group <= 1024) GN_GO(1);
    else if (group <= 2048) GN_GO(2);
    else GN_GO(4);
#undef GN_GO
    PE_LAUNCH_CHECK();
    return 0;
}

extern "C" int pe_gate_norm(const float* y, int T, int C, int group, const void* proj, int dtype, int ld, int z_off, const void* weight,
                            int w_dtype, float eps, void* out, void* stream) {
    if (T <= 0) return 0;
    if (group <= 0 || C % group || z_off < 0 || z_off + C > ld) return PE_ERR_UNSUPPORTED;
    const int threads = group >= 256 ? 256 : ((group + 31) / 32) * 32;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t size = dtype == PE_F32 ? 4 : 2;
    if ((dtype == PE_F32 || dtype == PE_BF16) && group % 4 == 0 && group <= 4096 && ld % 4 == 0 && z_off % 4 == 0 && (uintptr_t)y % 16 == 0 &&
        (uintptr_t)proj % (4 * size) == 0 && (uintptr_t)out % (4 * size) == 0)
        return dtype == PE_F32 ? gate_norm_vec(y, T, C, group, (const float*)proj, ld, z_off, weight, w_dtype, eps, (float*)out, s)
                               : gate_norm_vec(y, T, C, group, (const bf16*)proj, ld, z_off, weight, w_dtype, eps, (bf16*)out, s);
    if (dtype == PE_F32) PE_TRY(pe_launch(gate_norm_kernel<float>, dim3(T, C / group), threads, 0, s, y, C, group, (const float*)proj, ld, z_off, weight, w_dtype, eps, (float*)out));
    else if (dtype == PE_BF16) PE_TRY(pe_launch(gate_norm_kernel<bf16>, dim3(T, C / group), threads, 0, s, y, C, group, (const bf16*)proj, ld, z_off, weight, w_dtype, eps, (bf16*)out));
    else return PE_ERR_UNSUPPORTED;
    PE_LAUNCH_CHECK();
    return 0;
}
