// The state-space recurrence of prompts as products of tiles in float32 (state_space.cu has the recurrence itself).
//
// A sequence's tokens are cut into chunks of up to 64.  With t and s places in a chunk of n tokens and a(s, t) = a_(s+1) .. a_t:
//   contribution of a chunk to the state      L = sum_s a(s, n-1) dt_s B_s x_s^T                                        [N, P]
//   its outputs, from the incoming state S    y_t = a(-1, t) S^T C_t + sum_{s <= t} a(s, t) dt_s (C_t . B_s) x_s + D x_t
// The scores C_t . B_s are the same for all heads of a group and are worked out once a group and chunk.  Walking the tokens costs 2
// multiply-adds an element of the state and token and one product a token more; as tiles a token meets N + N / H' + 32 + N entries a
// column, with 8 x 8 or 8 x 4 results a thread in registers instead of a state that every token passes through.
//
// Bound by float32 multiply-adds (fma.rn.f32x2: two an instruction, each half rounds as a plain one does).  Decays between two tokens
// are exp of the difference of running sums of -exp(A_log) dt in float64, which costs no digits however long the chunk's sum.
// Measured on a B200, 64 heads of 64 columns, 128 state rows, rows of 1,400 and 647 tokens: 1,028 us as a walk, 190 us here (steps 3.5,
// contributions 61, 70 before the steps had a launch of their own, carry 32, outputs 94: 28 float32 TFLOP/s).  Heads of 64 columns, an even
// number of them a group, with 64 or 128 state rows go another way (state_space_tcgen05.cu: 132 us); these kernels have the other sizes.
#include "state_space.cuh"
#include "chunk_tiles.cuh"

// Four heads of a chunk: its place in the packed tokens, its steps' sizes dt and weights in the state's contribution dt_s a(s, n-1), and
// the running sums of -exp(A_log) dt (zero steps behind its tokens).  Once a chunk and head: worked out by every tile of contributions and
// again by every tile of outputs, in front of their products, they cost both kernels a chain of searches, logarithms and sums in float64.
template <typename T>
__global__ void __launch_bounds__(4 * SS_CHUNK) st_steps_kernel(ScanArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ double sums[4][2];
    int first, n;
    ss_find_chunk(a, a.first_chunk + blockIdx.x, first, n);
    if (threadIdx.x == 0 && blockIdx.y == 0) a.chunk_rows[blockIdx.x] = make_int2(first, n);
    if (n <= 0) return;
    const int hh = threadIdx.x / SS_CHUNK, t = threadIdx.x % SS_CHUNK, lane = t & 31, h = blockIdx.y * 4 + hh;
    const bool on = h < a.H;
    const float A = on ? expf(load_as_f(a.a_log, a.al_dtype, h)) : 0.f, bias = on ? load_as_f(a.dt_bias, a.dtb_dtype, h) : 0.f;
    const float dt = on && t < n ? ss_softplus(to_f(((const T*)a.proj)[(size_t)(first + t) * a.proj_ld + a.dt_off + h]) + bias) : 0.f;
    double la = fmax(-(double)A * (double)dt, -1e4);       // (exp of it is zero in float32 long before; a sum with an infinity has no differences)
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double below = __shfl_up_sync(0xffffffffu, la, o);
        if (lane >= o) la += below;
    }
    if (lane == 31) sums[hh][t >> 5] = la;
    __syncthreads();
    if (!on) return;
    const double end = sums[hh][1] + sums[hh][0];
    if (t >= 32) la += sums[hh][0];
    float* dst = a.chunk_steps + ((size_t)blockIdx.x * a.H + h) * SS_STEP_FLOATS;
    reinterpret_cast<float2*>(dst)[t] = make_float2(dt, dt * expf((float)(end - la)));
    reinterpret_cast<double*>(dst + 2 * SS_CHUNK)[t] = la;
    if (t == 0) a.chunk_decay[(size_t)blockIdx.x * a.H + h] = expf((float)end);
}

// blockIdx.y < H: chunk and head, 128 state rows x 64 columns of L (blockIdx.z: which).  From H on: the scores of a chunk and group.
__global__ void __launch_bounds__(ST_THREADS) st_contribution_kernel(ScanArgs a, int vec_bc, int vec_x, int tiles_n) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ __align__(16) float smem[SS_CHUNK * 128 / 2 + SS_CHUNK * 64 / 2];         // 32 tokens of B and of x; or two slices
    __shared__ float ws[SS_CHUNK];
    const int tid = threadIdx.x, H = a.H, N = a.N, P = a.P, inner = H * P;
    const int first = a.chunk_rows[blockIdx.x].x, n = a.chunk_rows[blockIdx.x].y;
    if (n <= 0) return;
    if ((int)blockIdx.y >= H) {
        if (blockIdx.z) return;
        const int g = blockIdx.y - H;
        float* bt = smem;
        float* ct = smem + ST_SLICE * SS_CHUNK;
        const float* src = a.xbc + (size_t)first * a.xbc_ld + inner + g * N;
        int ty, tx;
        st_place(ty, tx);
        st_pair acc[8][2];
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = 0ull;
        STSlice rb, rc;
        rb.load(src, a.xbc_ld, n, N, vec_bc);
        rc.load(src + a.G * N, a.xbc_ld, n, N, vec_bc);
        for (int k0 = 0; k0 < N; k0 += ST_SLICE) {
            __syncthreads();
            rb.store_turned(bt);
            rc.store_turned(ct);
            __syncthreads();
            if (k0 + ST_SLICE < N) {
                rb.load(src + k0 + ST_SLICE, a.xbc_ld, n, N - k0 - ST_SLICE, vec_bc);
                rc.load(src + a.G * N + k0 + ST_SLICE, a.xbc_ld, n, N - k0 - ST_SLICE, vec_bc);
            }
#pragma unroll 8
            for (int k = 0; k < ST_SLICE; ++k) {
                float s[8];
                *reinterpret_cast<float4*>(s) = *reinterpret_cast<const float4*>(bt + st_turned(k, ty * 4));
                *reinterpret_cast<float4*>(s + 4) = *reinterpret_cast<const float4*>(bt + st_turned(k, ty * 4 + 32));
                const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(ct + st_turned(k, tx * 4));
#pragma unroll
                for (int i = 0; i < 8; ++i) { st_fma(acc[i][0], s[i], t.x); st_fma(acc[i][1], s[i], t.y); }
            }
        }
        float* dst = a.chunk_scores + ((size_t)blockIdx.x * a.G + g) * SS_CHUNK * SS_CHUNK;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            *reinterpret_cast<float4*>(dst + (ty * 4 + 32 * (i / 4) + i % 4) * SS_CHUNK + tx * 4) = st_four(acc[i][0], acc[i][1]);
        return;
    }
    const int h = blockIdx.y, g = h / (H / a.G), n0 = blockIdx.z % tiles_n * 128, p0 = blockIdx.z / tiles_n * 64;
    const float* b_src = a.xbc + (size_t)first * a.xbc_ld + inner + g * N + n0;
    const float* x_src = a.xbc + (size_t)first * a.xbc_ld + h * P + p0;
    float* bs = smem;                                      // [32][128]
    float* xs = smem + 32 * 128;                           // [32][64]
    float4 rb[8], rx[4];                                   // 32 tokens of B (a token of 128 a warp) and x
    auto fetch = [&](int s0) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int i = tid + e * ST_THREADS, s = s0 + (i >> 5), c = (i & 31) * 4;
            rb[e] = s < n ? st_load4(b_src + (size_t)s * a.xbc_ld + c, N - n0 - c, vec_bc) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int i = tid + e * ST_THREADS, s = s0 + (i >> 4), c = (i & 15) * 4;
            rx[e] = s < n ? st_load4(x_src + (size_t)s * a.xbc_ld + c, P - p0 - c, vec_x) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    fetch(0);
    if (tid < SS_CHUNK) ws[tid] = reinterpret_cast<const float2*>(a.chunk_steps + ((size_t)blockIdx.x * H + h) * SS_STEP_FLOATS)[tid].y;
    const int lane = tid & 31, warp = tid >> 5, ty = warp * 4 + (lane >> 3), tx = lane & 7;       // 16 x 8 threads: rows ty * 4 + 64 i, columns tx * 4 + 32 j
    st_pair acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
    for (int s0 = 0; s0 < n; s0 += 32) {
        __syncthreads();
#pragma unroll
        for (int e = 0; e < 8; ++e) *reinterpret_cast<float4*>(bs + 4 * (tid + e * ST_THREADS)) = rb[e];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int i = tid + e * ST_THREADS, s = s0 + (i >> 4);
            const float w = ws[s];
            *reinterpret_cast<float4*>(xs + 4 * i) = make_float4(rx[e].x * w, rx[e].y * w, rx[e].z * w, rx[e].w * w);
        }
        if (s0 + 32 < n) fetch(s0 + 32);
        __syncthreads();
        const int m = min(32, n - s0);
#pragma unroll 4
        for (int s = 0; s < m; ++s) {
            float b[8];
            *reinterpret_cast<float4*>(b) = *reinterpret_cast<const float4*>(bs + s * 128 + ty * 4);
            *reinterpret_cast<float4*>(b + 4) = *reinterpret_cast<const float4*>(bs + s * 128 + ty * 4 + 64);
            const ulonglong2 x0 = *reinterpret_cast<const ulonglong2*>(xs + s * 64 + tx * 4), x1 = *reinterpret_cast<const ulonglong2*>(xs + s * 64 + tx * 4 + 32);
#pragma unroll
            for (int i = 0; i < 8; ++i) { st_fma(acc[i][0], b[i], x0.x); st_fma(acc[i][1], b[i], x0.y); st_fma(acc[i][2], b[i], x1.x); st_fma(acc[i][3], b[i], x1.y); }
        }
    }
    float* dst = a.chunk_state + ((size_t)blockIdx.x * H + h) * N * P;
    const bool vec = P % 4 == 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = n0 + ty * 4 + 64 * (i / 4) + i % 4;
        if (r >= N) continue;
        float* row = dst + (size_t)r * P + p0 + tx * 4;
        st_store4(row, P - p0 - tx * 4, vec, st_four(acc[i][0], acc[i][1]));
        st_store4(row + 32, P - p0 - tx * 4 - 32, vec, st_four(acc[i][2], acc[i][3]));
    }
}

// A thread an element of a sequence's state walks the sequence's chunks in order, leaves every chunk its incoming state where its own
// contribution was, and stores the sequence's new state (whose order is that of state_space.cu's threads).  ONE: the step is one slab, the
// usual case (with the slab's bounds in the loop's the compiler keeps fewer of the eight reads in flight: 65 us instead of 32).
template <bool ONE>
__global__ void __launch_bounds__(256) st_carry_kernel(ScanArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    const int b = blockIdx.y;
    const size_t per_head = (size_t)a.N * a.P, per = per_head * a.H;
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= per) return;
    int base = 0;
    for (int i = 0; i < b; ++i) base += (a.row_lens[i] + SS_CHUNK - 1) / SS_CHUNK;
    int nc = (a.row_lens[b] + SS_CHUNK - 1) / SS_CHUNK;
    if (!ONE) {                                           // the sequence's chunks of this slab, by their places in it
        const int end = min(base + nc - a.first_chunk, a.slab);
        base = max(base - a.first_chunk, 0);
        nc = max(end - base, 0);
    }
    if (nc == 0) return;
    const int h = (int)(e / per_head), r = (int)(e % per_head) / a.P, p = (int)(e % per_head) % a.P;
    float* sp = a.state + (size_t)a.slots[b] * a.state_stride + (((size_t)h * a.NR + r % a.NR) * a.P + p) * a.NS + r / a.NR;
    float carry = *sp;
    for (int c0 = base; c0 < base + nc; c0 += 8) {           // eight chunks' numbers in flight: they do not depend on the carry
        float own[8], dec[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const bool there = c0 + u < base + nc;
            own[u] = there ? a.chunk_state[(size_t)(c0 + u) * per + e] : 0.f;
            dec[u] = there ? a.chunk_decay[(size_t)(c0 + u) * a.H + h] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (c0 + u < base + nc) {
                a.chunk_state[(size_t)(c0 + u) * per + e] = carry;
                carry = fmaf(dec[u], carry, own[u]);
            }
        }
    }
    *sp = carry;
}

// Chunk, head and 64 columns of its outputs.
__global__ void __launch_bounds__(ST_THREADS) st_output_kernel(ScanArgs a, int vec_bc, int vec_x) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ __align__(16) float smem[2 * SS_CHUNK * SS_CHUNK];       // two buffers of a slice of C and of S; then weights and x
    __shared__ float dts[SS_CHUNK];
    __shared__ double las[SS_CHUNK];
    const int tid = threadIdx.x, H = a.H, N = a.N, P = a.P, inner = H * P, h = blockIdx.y, g = h / (H / a.G), p0 = blockIdx.z * 64;
    const int first = a.chunk_rows[blockIdx.x].x, n = a.chunk_rows[blockIdx.x].y;
    if (n <= 0) return;
    int ty, tx;
    st_place(ty, tx);
    const float* c_src = a.xbc + (size_t)first * a.xbc_ld + inner + a.G * N + g * N;
    const float* s_src = a.chunk_state + ((size_t)blockIdx.x * H + h) * N * P + p0;
    const bool vec_s = P % 4 == 0;
    STSlice rc;
    float4 rs[4];
    auto fetch = [&](int k0) {
        rc.load(c_src + k0, a.xbc_ld, n, N - k0, vec_bc);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int i = tid + e * ST_THREADS, k = k0 + (i >> 4), c = (i & 15) * 4;
            rs[e] = k < N ? st_load4(s_src + (size_t)k * P + c, P - p0 - c, vec_s) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    auto put = [&](float* to) {
        rc.store_turned(to);
#pragma unroll
        for (int e = 0; e < 4; ++e) *reinterpret_cast<float4*>(to + ST_SLICE * SS_CHUNK + 4 * (tid + e * ST_THREADS)) = rs[e];
    };
    fetch(0);
    if (tid < SS_CHUNK) {
        const float* steps = a.chunk_steps + ((size_t)blockIdx.x * H + h) * SS_STEP_FLOATS;
        dts[tid] = reinterpret_cast<const float2*>(steps)[tid].x;
        las[tid] = reinterpret_cast<const double*>(steps + 2 * SS_CHUNK)[tid];
    }
    put(smem);
    __syncthreads();
    st_pair acc[8][2];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = 0ull;
    for (int k0 = 0, b = 0; k0 < N; k0 += ST_SLICE, b ^= 1) {
        const bool more = k0 + ST_SLICE < N;
        if (more) fetch(k0 + ST_SLICE);
        const float* ct = smem + b * SS_CHUNK * SS_CHUNK;
        const float* ss = ct + ST_SLICE * SS_CHUNK;
#pragma unroll 8
        for (int k = 0; k < ST_SLICE; ++k) {
            float c[8];
            *reinterpret_cast<float4*>(c) = *reinterpret_cast<const float4*>(ct + st_turned(k, ty * 4));
            *reinterpret_cast<float4*>(c + 4) = *reinterpret_cast<const float4*>(ct + st_turned(k, ty * 4 + 32));
            const ulonglong2 s = *reinterpret_cast<const ulonglong2*>(ss + k * 64 + tx * 4);
#pragma unroll
            for (int i = 0; i < 8; ++i) { st_fma(acc[i][0], c[i], s.x); st_fma(acc[i][1], c[i], s.y); }
        }
        if (more) put(smem + (b ^ 1) * SS_CHUNK * SS_CHUNK);
        __syncthreads();
    }
    float* pt = smem;                                      // [64 s][64 t]
    float* xs = smem + SS_CHUNK * SS_CHUNK;                // [64 s][64 p]
    const float* scores = a.chunk_scores + ((size_t)blockIdx.x * a.G + g) * SS_CHUNK * SS_CHUNK;
    const float* x_src = a.xbc + (size_t)first * a.xbc_ld + h * P + p0;
    float zero = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int i = tid + e * ST_THREADS, s = i >> 4, t = (i & 15) * 4;
        float4 w = *reinterpret_cast<const float4*>(scores + 4 * i);
        const float4 x = s < n ? st_load4(x_src + (size_t)s * a.xbc_ld + t, P - p0 - t, vec_x) : make_float4(0.f, 0.f, 0.f, 0.f);
        const double ls = las[s];
        const float d = dts[s];
        w.x = s <= t ? w.x * (d * expf((float)(las[t] - ls))) : 0.f;
        w.y = s <= t + 1 ? w.y * (d * expf((float)(las[t + 1] - ls))) : 0.f;
        w.z = s <= t + 2 ? w.z * (d * expf((float)(las[t + 2] - ls))) : 0.f;
        w.w = s <= t + 3 ? w.w * (d * expf((float)(las[t + 3] - ls))) : 0.f;
        *reinterpret_cast<float4*>(pt + 4 * i) = w;
        st_zero(zero, x);
        *reinterpret_cast<float4*>(xs + 4 * i) = x;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float d = expf((float)las[ty * 4 + 32 * (i / 4) + i % 4]);
        float2 u = st_two(acc[i][0]), v = st_two(acc[i][1]);
        asm("mov.b64 %0, {%1, %2};" : "=l"(acc[i][0]) : "f"(u.x * d), "f"(u.y * d));
        asm("mov.b64 %0, {%1, %2};" : "=l"(acc[i][1]) : "f"(v.x * d), "f"(v.y * d));
    }
    const bool guarded = __syncthreads_or(zero != 0.f);
    const int last = min(n, 32 + 16 * (tid >> 6) + 16);    // a warp's tokens reach this far: later ones have no weight
    st_weighted(acc, pt, xs, last, ty, tx, guarded);
    const float Dh = load_as_f(a.d_skip, a.d_dtype, h);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int t = ty * 4 + 32 * (i / 4) + i % 4;
        if (t >= n) continue;
        const float4 x = *reinterpret_cast<const float4*>(xs + t * 64 + tx * 4), v = st_four(acc[i][0], acc[i][1]);
        st_store4(a.y + (size_t)(first + t) * inner + h * P + p0 + tx * 4, P - p0 - tx * 4, vec_s,
                  make_float4(fmaf(Dh, x.x, v.x), fmaf(Dh, x.y, v.y), fmaf(Dh, x.z, v.z), fmaf(Dh, x.w, v.w)));
    }
}

template <typename T>
static int st_run(ScanArgs a, cudaStream_t s) {
    const bool rows = a.xbc_ld % 4 == 0 && (uintptr_t)a.xbc % 16 == 0;
    const int vec_x = rows && a.P % 4 == 0, vec_bc = rows && (a.H * a.P) % 4 == 0 && a.N % 4 == 0;
    const int tn = (a.N + 127) / 128, tp = (a.P + 63) / 64;
    for (; a.first_chunk < a.chunks; a.first_chunk += a.slab) {      // (the carry between two slabs lies in the sequences' states)
        PE_TRY(pe_launch(st_steps_kernel<T>, dim3(a.slab, (a.H + 3) / 4), 4 * SS_CHUNK, 0, s, a));
        PE_LAUNCH_CHECK();
        PE_TRY(pe_launch(st_contribution_kernel, dim3(a.slab, a.H + a.G, tn * tp), ST_THREADS, 0, s, a, vec_bc, vec_x, tn));
        PE_LAUNCH_CHECK();
        PE_TRY(pe_launch(a.slab == a.chunks ? st_carry_kernel<true> : st_carry_kernel<false>, dim3((unsigned)(((size_t)a.H * a.N * a.P + 255) / 256), a.B), 256, 0, s, a));
        PE_LAUNCH_CHECK();
        PE_TRY(pe_launch(st_output_kernel, dim3(a.slab, a.H, tp), ST_THREADS, 0, s, a, vec_bc, vec_x));
        PE_LAUNCH_CHECK();
    }
    return 0;
}

int ss_tiles(const ScanArgs& a, int dtype, cudaStream_t s) {
    if (a.H + a.G > 65535) return PE_ERR_UNSUPPORTED;
    return dtype == PE_F32 ? st_run<float>(a, s) : st_run<bf16>(a, s);
}
