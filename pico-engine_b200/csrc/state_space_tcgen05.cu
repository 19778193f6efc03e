// The state-space recurrence of prompts as products of tiles on the 5th-generation tensor cores (state_space_tiles.cu has the same with
// multiply-adds, and the sums; chunk_mma.cuh how float32 numbers are multiplied).  Heads of 64 columns, an even number of them a group, 64 or 128 state rows.
//
// Two heads of a group are the 128 rows of a product: their columns p stand on the accumulator's lanes, and what all heads of a group
// share (B, C, cut into parts once a chunk and group) is the other operand:
//   contributions  L^T [(h, p)][n] = (x_s dt_s a(s, end))^T B          K: the chunk's tokens, 64 of the state's rows n at a time
//   outputs        y^T [(h, p)][t] = a(-1, t) S^T C^T + x^T W_h^T      K: the state's rows, 64 at a time; then the chunk's tokens
// W_h differs between the two heads: both heads' columns meet both heads' weights, and half of the results is left.
//
// A state in scratch is [N / 8][64 p][8 n], so that a thread writes and reads runs of 32 bytes and a warp whole lines.  Two CTAs of eight
// warps an SM, 256 columns of tensor memory each: the loads, cuts and stores of one cover the waits of the other.
//
// What bounds it: outputs the chain of a unit (loads, cuts, products, weights: 25,000 cycles of which the products are 5,000; two blocks
// an SM overlap), contributions and carry the state's way through L2 (5 to 10 TB/s).  Measured on a B200, 64 heads, 128 state rows,
// rows of 1,400 and 647 tokens: 134.5 us (steps with parts and scores 12, contributions 27, carry 25, outputs 63) where multiply-adds take 187 (3, 61, 32, 94);
// 28 heads, 2,500 tokens 76 (102), 8 heads, 65 tokens and one 28.7 (34.5): steps that go in chunks at all (StateSpace.chunks_pay) are sooner here whatever their size.
// Errors against 64 bits, means over eight inputs, outputs and states of their norms (multiply-adds): 64 heads, 128 state rows, rows of 1,400 and 647 tokens 7.9e-8
// and 9.1e-8 (1.09e-7 and 9.3e-8); 28 heads, 64 state rows, rows of 700 and 100 4.7e-8 and 1.00e-7 (6.3e-8 and 1.04e-7): most of it the decays' and the steps'.
// With mma.sync in place of tcgen05 contributions took 50 and outputs 99 us (the fragments' loads and cuts between the products); an exponential for
// each pair of tokens outputs 71 us; sixteen warps a block instead of eight contributions 35 and outputs 66 us.
#include "state_space.cuh"
#include "chunk_mma.cuh"

#define SM_THREADS 512
#define SM_FEW 256                                        // threads of a block of contributions and of outputs
#define SM_SLAB (CM_PARTS * CM_PLANE)                     // parts of 64 state rows (or columns of a head) of a chunk: 24 KB
// What outputs and contributions need of a chunk's steps, a head: 64 weights dt_s a(s, end) of its contribution; 64 decays a(-1, t); and a weight a(s, t) dt_s as a
// factor of s alone, dt_s a(s, last of its run of eight), and one of its run and t ([t][run]); inside a run of eight ([t][8]) as a whole.  A product of two
// exponentials instead of one for each pair: 19 exponentials a token where there were 35.
#define SM_WS 0
#define SM_ES 64
#define SM_FACTOR 128
#define SM_STEP 192                                       // and each token's own decay, for the walk
#define SM_RUNS 256
#define SM_INSIDE (256 + 8 * SS_CHUNK)
#define SM_CONTRIBUTION_SMEM (4 * SM_SLAB + 2048)         // (1,024 to begin on a boundary, 1,024 behind for the walk's decays and steps)
#define SM_OUTPUT_SMEM (4 * SM_SLAB + 2048)

__device__ __forceinline__ float4 sm_times(const float4& v, float w) {
    const float2 a = cm_scaled(v.x, v.y, w), b = cm_scaled(v.z, v.w, w);
    return make_float4(a.x, a.y, b.x, b.y);
}

// A chunk's place and where its numbers are read: those of two heads from h on, and their group's B and C.
struct SMChunk {
    int first, n, ld;
    const float* x; const float* b; const float* c;       // of the chunk's first token
    bool vec;
    __device__ __forceinline__ SMChunk(const ScanArgs& a, int first_, int n_, int h, int g, int vec_) : first(first_), n(n_), ld(a.xbc_ld), vec(vec_) {
        const float* row = a.xbc + (size_t)first * a.xbc_ld;
        x = row + h * 64; b = row + a.H * 64 + g * a.N; c = b + a.G * a.N;
    }
    __device__ __forceinline__ void eight(float4& u, float4& v, const float* p, int t, int col) const {       // (zeros behind the chunk's tokens)
        u = v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t >= n) return;
        p += (size_t)t * ld + col;
        if (vec) { u = *reinterpret_cast<const float4*>(p); v = *reinterpret_cast<const float4*>(p + 4); }
        else { u = make_float4(p[0], p[1], p[2], p[3]); v = make_float4(p[4], p[5], p[6], p[7]); }
    }
};

// blockIdx.y < G: a chunk's and group's B and C as their parts, which all heads of the group multiply with, and the scores C_t . B_s, [t][s].
// Behind: eight heads of a chunk: its place in the packed tokens and its steps (zero steps behind its tokens).
template <typename T>
__global__ void __launch_bounds__(SM_THREADS) sm_steps_kernel(ScanArgs a, int vec) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) unsigned char sm_mem[];
    __shared__ double sums[8], las[8][SS_CHUNK];
    __shared__ float dts[8][SS_CHUNK];
    __shared__ unsigned seen, from;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, row = tid >> 3, group = tid & 7;
    if (tid == 0) { seen = 0; from = SS_CHUNK; }
    pdl_wait();
    int first, n;
    ss_find_chunk(a, a.first_chunk + blockIdx.x, first, n);
    if (tid == 0 && (int)blockIdx.y == a.G) a.chunk_rows[blockIdx.x] = make_int2(first, n);
    if (n <= 0) return;
    if ((int)blockIdx.y < a.G) {
        const int g = blockIdx.y, N = a.N;
        const SMChunk chunk(a, first, n, 0, g, vec);
        unsigned char* planes = a.chunk_planes + ((size_t)blockIdx.x * a.G + g) * 2 * ss_plane_bytes(N);
        const int t0 = (warp & 3) * 16, s0 = warp < 8 ? (warp >> 2) * 32 : SS_CHUNK;
        CMScores acc;
        acc.clear();
        for (int k0 = 0; k0 < N; k0 += 64) {
            unsigned most[2] = {0, 0};
            float4 v[2][2];
#pragma unroll
            for (int e = 0; e < 2; ++e) chunk.eight(v[e][0], v[e][1], e ? chunk.c : chunk.b, row, k0 + 8 * group);
            __syncthreads();
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                cm_put(sm_mem + e * SM_SLAB + cm_at(row, group), CM_PLANE, sm_times(v[e][0], CM_UP), sm_times(v[e][1], CM_UP), most[e]);
                if (!cm_odd(most[e])) continue;
                atomicMin(&from, (unsigned)row);
                const float w[8] = {v[e][0].x, v[e][0].y, v[e][0].z, v[e][0].w, v[e][1].x, v[e][1].y, v[e][1].z, v[e][1].w};
                for (int i = 0; i < 8; ++i)
                    if (e == 0 && fabsf(w[i]) >= 0x1p34f) atomicOr(&seen, 1u);          // (2^34: what is rounded to 2^35 counts)
            }
            __syncthreads();
            unsigned char* to = planes + (size_t)(k0 / 64) * SM_SLAB;
            for (int i = tid * 16; i < SM_SLAB; i += SM_THREADS * 16) {
                *reinterpret_cast<uint4*>(to + i) = *reinterpret_cast<const uint4*>(sm_mem + i);
                *reinterpret_cast<uint4*>(to + ss_plane_bytes(N) + i) = *reinterpret_cast<const uint4*>(sm_mem + SM_SLAB + i);
            }
            if (s0 <= t0) acc.add(at_smem(sm_mem) + SM_SLAB, at_smem(sm_mem), CM_PLANE, t0, s0);
        }
        if (tid == 0) a.chunk_seen[(size_t)blockIdx.x * a.G + g] = seen | from << 16;
        float* dst = a.chunk_scores + ((size_t)blockIdx.x * a.G + g) * SS_CHUNK * SS_CHUNK;
        const int exact = from;                            // tokens in front of it have their scores from the parts
        if (exact < n) {                                   // the others with multiply-adds, B's rows in shared memory, 68 or 132 numbers apart
            float* rows = reinterpret_cast<float*>(sm_mem);
            __syncthreads();
#pragma unroll 1
            for (int i = tid; i < n * N; i += SM_THREADS) rows[i / N * (N + 4) + i % N] = chunk.b[(size_t)(i / N) * chunk.ld + i % N];
            __syncthreads();
#pragma unroll 1
            for (int i = exact * SS_CHUNK + tid; i < n * SS_CHUNK; i += SM_THREADS) {
                const int t = i / SS_CHUNK, s = i % SS_CHUNK;
                if (s > t) continue;
                const float *b = rows + s * (N + 4), *c = chunk.c + (size_t)t * chunk.ld;
                float v = 0.f;
#pragma unroll 4
                for (int k = 0; k < N; ++k) v = fmaf(b[k], c[k], v);
                dst[i] = v;
            }
        }
        if (s0 > t0) return;                               // (nobody reads the weights of later keys)
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
            const int t = t0 + lane / 4 + 4 * e;
            if (t >= exact) continue;
#pragma unroll
            for (int j = 0; j < 4; ++j) *reinterpret_cast<float2*>(dst + t * SS_CHUNK + s0 + 8 * j + lane % 4 * 2) = cm_scaled(acc.get(j, e), acc.get(j, e + 1), CM_DOWN * CM_DOWN);
        }
        return;
    }
    const int hh = tid / SS_CHUNK, t = tid % SS_CHUNK, h = (blockIdx.y - a.G) * 8 + hh;
    const bool on = h < a.H;
    const float A = on ? expf(load_as_f(a.a_log, a.al_dtype, h)) : 0.f, bias = on ? load_as_f(a.dt_bias, a.dtb_dtype, h) : 0.f;
    const float dt = on && t < n ? ss_softplus(to_f(((const T*)a.proj)[(size_t)(first + t) * a.proj_ld + a.dt_off + h]) + bias) : 0.f;
    double la = fmax(-(double)A * (double)dt, -1e4);       // (exp of it is zero in float32 long before; a sum with an infinity has no differences)
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double below = __shfl_up_sync(0xffffffffu, la, o);
        if (lane >= o) la += below;
    }
    if (t == 31) sums[hh] = la;
    __syncthreads();
    if (t >= 32) la += sums[hh];
    las[hh][t] = la;
    dts[hh][t] = dt;
    __syncthreads();
    if (!on) return;
    const double end = las[hh][SS_CHUNK - 1];
    float* dst = a.chunk_steps + ((size_t)blockIdx.x * a.H + h) * SS_MATRIX_STEP_FLOATS;
    dst[SM_WS + t] = dt * expf((float)(end - la));
    dst[SM_ES + t] = expf((float)la);
    dst[SM_STEP + t] = expf((float)(la - (t ? las[hh][t - 1] : 0.0)));
    dst[SM_FACTOR + t] = dt * expf((float)(las[hh][t | 7] - la));
    float runs[8], inside[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int s = (t & ~7) + i;
        runs[i] = i < t >> 3 ? expf((float)(la - las[hh][8 * i + 7])) : 0.f;
        inside[i] = s <= t ? dts[hh][s] * expf((float)(la - las[hh][s])) : 0.f;
    }
    cm_store8(dst + SM_RUNS + 8 * t, runs);
    cm_store8(dst + SM_INSIDE + 8 * t, inside);
    if (t == 0) a.chunk_decay[(size_t)blockIdx.x * a.H + h] = (float)exp(end);      // (a state hands its errors on from chunk to chunk)
}

// What parts are not made of: two heads' chunk token after token with multiply-adds, from its incoming state (none: zeros), all threads of a block.  Outputs from token
// `exact` on; the state behind the chunk to `to_state`, if that is asked for.  B, C and x lie in the block's shared memory (which nobody else uses then).  A state with
// infinities or huge numbers sends every unit behind it here, a token that is no number those of its chunk.  64 heads, 128 state rows, rows of 1,400 and 647 tokens with one
// number of x, one of B, all of a token, every token that is none: 178 / 203 / 203 / 262 us (139 without; multiply-add tiles 191; entry by entry from memory 640 to 1,637).
template <int N>
__device__ __noinline__ void sm_walk(const ScanArgs& a, int c, int first, int n, int h0, int g, const float* state, int exact, float* to_state) {
    extern __shared__ unsigned char sm_raw[];
    float* smem = reinterpret_cast<float*>(sm_raw + (-at_smem(sm_raw) & 1023u));
    using Walk = CMWalk<N>;
    const SMChunk chunk(a, first, n, h0, g, 0);
    const int tid = threadIdx.x, h = h0 + (Walk::column() >> 6), ld = chunk.ld, ld_y = a.H * 64;       // (loops that store read nothing of the arguments, which they would read again each time)
    float *bs = smem, *cs = smem + SS_CHUNK * N, *xs = cs + SS_CHUNK * N, *turns = xs + SS_CHUNK * 128;      // [64 t][N]; [64 t][128]; [head][64 t]: decays, then steps
    const bool writes = !(tid & 1);
    float* y = a.y + (size_t)first * ld_y + h0 * 64 + Walk::written();
    Walk walk;
    if (__syncthreads_and(walk.begin(state))) {            // no state that is a number: no output is one
        if (writes)
            for (int t = exact; t < n; ++t) y[(size_t)t * ld_y] = __int_as_float(0x7fffffff);
        return;
    }
    const auto fill = [&](float* dst, const float* src, int width) {       // eight reads in front of their stores
#pragma unroll 1
        for (int i = tid; i < SS_CHUNK * width; i += 8 * SM_FEW) {
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = src[(size_t)min((i + e * SM_FEW) / width, n - 1) * ld + (i + e * SM_FEW) % width];
#pragma unroll
            for (int e = 0; e < 8; ++e) dst[i + e * SM_FEW] = v[e];
        }
    };
    fill(bs, chunk.b, N);
    fill(cs, chunk.c, N);
    fill(xs, chunk.x, 128);
    if (tid < 2 * SS_CHUNK) {
        const float* steps = a.chunk_steps + ((size_t)c * a.H + h0 + (tid >> 6)) * SS_MATRIX_STEP_FLOATS;
        const int t = tid & 63;
        turns[tid] = steps[SM_STEP + t];
        turns[2 * SS_CHUNK + tid] = steps[SM_INSIDE + 8 * t + (t & 7)];       // (a token's weight for itself: dt)
    }
    const float skip = load_as_f(a.d_skip, a.d_dtype, h);
    const float* turn = turns + (Walk::column() >> 6) * SS_CHUNK;
    __syncthreads();
#pragma unroll 1                                           // (few instructions: what runs here has not run before, and comes from L2 a line at a time)
    for (int t = 0; t < n; ++t) {
        const float4 x = *reinterpret_cast<const float4*>(xs + t * 128 + Walk::column());
        const float dt = turn[2 * SS_CHUNK + t], u[4] = {x.x * dt, x.y * dt, x.z * dt, x.w * dt};
        walk.step(bs + t * N, nullptr, turn[t], u);
        if (t < exact) continue;
        const float o = walk.output(cs + t * N);
        if (writes) y[(size_t)t * ld_y] = fmaf(skip, xs[t * 128 + Walk::written()], o);
    }
    if (to_state) walk.end(to_state);
    __syncthreads();                                       // (the shared memory has been read)
}

// Chunks and two heads at a time, contributions: the next unit's x is asked for while this one's products run.
__global__ void __launch_bounds__(SM_FEW, 2) sm_contribution_kernel(ScanArgs a, int vec, int units, int* status) {
    extern __shared__ unsigned char sm_raw[];
    __shared__ __align__(8) unsigned long long bar;
    __shared__ unsigned tmem_s, seen, odd;
    __shared__ float ws[2][SS_CHUNK];
    unsigned char* xs = sm_raw + (-at_smem(sm_raw) & 1023u);          // [part][head][64 s][64 p]
    unsigned char* bs = xs + 2 * SM_SLAB;                             // [slab][part][64 s][64 n]
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), H = a.H, N = a.N, pairs = H / 2, slabs = N / 64;
    const int q = warp & 3, hh = q >> 1, p = (q & 1) * 32 + lane, row = tid >> 3, group = tid & 7;      // a thread's runs of eight: this row and the one 32 behind, of either head
    if (tid == 0) odd = 0;
    const unsigned tmem = cm_begin(&tmem_s, &bar);
    const unsigned elected = warp == 0 ? pe_elect() : 0u;
    pdl_wait();
    unsigned phase = 0, known = 0;
    int2 place = a.chunk_rows[blockIdx.x / pairs];
    float4 v[4][2];
    float w = 0.f;
    auto fetch = [&](int unit, const int2& at) {
        const int h0 = unit % pairs * 2;
        const SMChunk chunk(a, at.x, at.y, h0, h0 / (H / a.G), vec);
#pragma unroll
        for (int e = 0; e < 4; ++e) chunk.eight(v[e][0], v[e][1], chunk.x + (e >> 1) * 64, row + (e & 1) * 32, 8 * group);
        if (tid < 2 * SS_CHUNK) w = a.chunk_steps[((size_t)(unit / pairs) * H + h0 + (tid >> 6)) * SS_MATRIX_STEP_FLOATS + SM_WS + (tid & 63)];
        if (tid == 0) known = a.chunk_seen[(size_t)(unit / pairs) * a.G + h0 / (H / a.G)] & 1u;      // (B)
    };
    if (place.y > 0) fetch(blockIdx.x, place);
    for (int unit = blockIdx.x; unit < units && place.y > 0; unit += gridDim.x) {
        const int c = unit / pairs, h0 = unit % pairs * 2, g = h0 / (H / a.G), n = place.y;
        cm_bring(bs, a.chunk_planes + ((size_t)c * a.G + g) * 2 * ss_plane_bytes(N), slabs * SM_SLAB);
        const int next = unit + gridDim.x;
        if (next < units) place = a.chunk_rows[next / pairs];
        if (tid < 2 * SS_CHUNK) ws[tid >> 6][tid & 63] = w;
        if (tid == 0) seen = known;
        __syncthreads();
        unsigned most = 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float by = ws[e >> 1][row + (e & 1) * 32];          // (times x before the power of two: either product alone stays in range)
            cm_put<true>(xs + (e >> 1) * CM_PLANE + cm_at(row + (e & 1) * 32, group), 2 * CM_PLANE, sm_times(sm_times(v[e][0], by), CM_UP), sm_times(sm_times(v[e][1], by), CM_UP), most);
        }
        cm_report(&seen, cm_seen(most, 2));
        cm_landed();
        cm_ready();
        const bool parts = !seen;
        if (parts && warp == 0) {
            cm_products(elected, tmem, tmem + N, cm_across(at_smem(xs), 2 * CM_PLANE, CM_PLANE), cm_across(at_smem(bs), CM_PLANE, SM_SLAB), cm_idesc(N, true, true));
            if (elected) at_commit(at_smem(&bar));
            __syncwarp();
        }
        if (next < units && place.y > 0) fetch(next, place);
        if (tid == 0) {
            a.unit_exact[unit] = parts ? n : 0;
            if (!parts) odd = 1;
        }
        float* state = a.chunk_state + ((size_t)c * H + h0) * N * 64;
        if (parts) {
            cm_done(&bar, phase, status);
            for (int j = 0; j < 2 * slabs; ++j) {
                const int column = (warp >> 2) * (N / 2) + 16 * j;
                const unsigned mine = tmem + ((unsigned)(q * 32) << 16) + column;
                float acc[16];
                cm_read(acc, mine + N);
                cm_take(acc, mine);
                cm_scale(acc, CM_DOWN * CM_DOWN);
                float* to = state + (size_t)hh * N * 64 + ((size_t)(column / 8) * 64 + p) * 8;
                cm_store8(to, *reinterpret_cast<const float (*)[8]>(acc));
                cm_store8(to + 512, *reinterpret_cast<const float (*)[8]>(acc + 8));
            }
        }
    }
    cm_end(tmem);
    if (!odd) return;                                      // (the walks behind the loop: inside they cost its registers)
    __shared__ ScanArgs args;
    if (tid == 0) args = a;
    __syncthreads();
#pragma unroll 1
    for (int unit = blockIdx.x; unit < units; unit += gridDim.x) {
        const int c = unit / pairs, h0 = unit % pairs * 2, g = h0 / (H / a.G);
        const int2 at = a.chunk_rows[c];
        if (at.y <= 0) break;
        const int exact = a.unit_exact[unit];
        float* state = a.chunk_state + ((size_t)c * H + h0) * N * 64;
        if (exact >= at.y) continue;
        if (N == 64) sm_walk<64>(args, c, at.x, at.y, h0, g, nullptr, at.y, state);
        else sm_walk<128>(args, c, at.x, at.y, h0, g, nullptr, at.y, state);
    }
}

// A block eight columns of a head's state, 2 N threads: a thread four entries (rows r .. r + 3 of a column) walks the sequence's chunks in order, leaves
// every chunk its incoming state where its own contribution was, and stores the sequence's new state.  The sequences' states have the order of
// state_space.cu's threads (a thread's four entries lie in four lines there), so they go through shared memory.
__global__ void __launch_bounds__(256) sm_carry_kernel(ScanArgs a) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) unsigned char sm_mem[];
    float* tile = reinterpret_cast<float*>(sm_mem);       // [NR][8 columns][NS]
    pdl_wait();
    const int b = blockIdx.y, h = blockIdx.x / 8, p0 = blockIdx.x % 8 * 8, tid = threadIdx.x;
    int base = 0;
    for (int i = 0; i < b; ++i) base += (a.row_lens[i] + SS_CHUNK - 1) / SS_CHUNK;
    int nc = (a.row_lens[b] + SS_CHUNK - 1) / SS_CHUNK;
    const int end = min(base + nc - a.first_chunk, a.slab);              // the sequence's chunks of this slab, by their places in it
    base = max(base - a.first_chunk, 0);
    nc = end - base;
    if (nc <= 0) return;
    const int run = 8 * a.NS / 4;                         // vectors of a state row's eight columns
    float* sp = a.state + (size_t)a.slots[b] * a.state_stride + ((size_t)h * a.NR + tid / run) * 64 * a.NS + (size_t)p0 * a.NS + tid % run * 4;
    const size_t per = (size_t)a.N * 16 * a.H;
    float4* chunks = reinterpret_cast<float4*>(a.chunk_state) + (size_t)base * per + (size_t)h * a.N * 16 + (size_t)(tid / 16) * 128 + p0 * 2 + tid % 16;
    const float* decay = a.chunk_decay + (size_t)base * a.H + h;
    // Eight chunks' numbers in flight: they do not depend on the carry.  Whole runs of eight and what is left are loops of their own: with one loop whose
    // reads ask whether there is a chunk 43 us instead of 23 (22 and 11 chunks of 64 heads).
    float4 own[8];
    float d[8];
    auto ask = [&](int m) {
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (u < m) { own[u] = chunks[u * per]; d[u] = decay[u * a.H]; }
    };
    if (nc >= 8) ask(8);
    else ask(nc);
    float start[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) start[k] = sp[k];               // (rows of the state area need not start on 16 bytes)
#pragma unroll
    for (int k = 0; k < 4; ++k) tile[4 * tid + k] = start[k];
    __syncthreads();
    const int r = tid / 16 * 8 + tid % 2 * 4, p = tid / 2 % 8;
    auto at = [&](int n) { return (n % a.NR * 8 + p) * a.NS + n / a.NR; };
    float4 carry = make_float4(tile[at(r)], tile[at(r + 1)], tile[at(r + 2)], tile[at(r + 3)]);
    auto step = [&](int m) {
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (u < m) {
                chunks[u * per] = carry;
                carry = make_float4(fmaf(d[u], carry.x, own[u].x), fmaf(d[u], carry.y, own[u].y), fmaf(d[u], carry.z, own[u].z), fmaf(d[u], carry.w, own[u].w));
            }
    };
    while (nc >= 8) {
        step(8);
        nc -= 8; chunks += 8 * per; decay += 8 * a.H;
        if (nc >= 8) ask(8);
        else ask(nc);
    }
    step(nc);
    tile[at(r)] = carry.x; tile[at(r + 1)] = carry.y; tile[at(r + 2)] = carry.z; tile[at(r + 3)] = carry.w;      // (the places that this thread read)
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) sp[k] = tile[4 * tid + k];
}

// Chunks and two heads at a time, outputs: the next unit's first rows of the state are asked for while this one's last products run.
__global__ void __launch_bounds__(SM_FEW, 2) sm_output_kernel(ScanArgs a, int vec, int units, int* status) {
    extern __shared__ unsigned char sm_raw[];
    __shared__ __align__(8) unsigned long long bar;
    __shared__ unsigned tmem_s, seen, from, odd;
    __shared__ __align__(16) float es[2][SS_CHUNK];
    unsigned char* mem = sm_raw + (-at_smem(sm_raw) & 1023u);
    unsigned char* ss = mem;                                          // [part][head][64 p][64 n] of the state
    unsigned char* cs = mem + 2 * SM_SLAB;                            // [slab][part][64 t][64 n]
    unsigned char* xs = mem;                                          // [part][head][64 s][64 p]
    unsigned char* wgt = mem + 2 * SM_SLAB;                           // [part][head][64 t][64 s]
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), H = a.H, N = a.N, inner = H * 64, pairs = H / 2, slabs = N / 64;
    const int q = warp & 3, hh = q >> 1, p = (q & 1) * 32 + lane, column = (warp >> 2) * 32, row = tid >> 3, group = tid & 7;
    if (tid == 0) odd = 0;
    const unsigned tmem = cm_begin(&tmem_s, &bar), mine = tmem + ((unsigned)(q * 32) << 16) + column;
    const unsigned elected = warp == 0 ? pe_elect() : 0u;
    pdl_wait();
    unsigned phase = 0, known = 0;
    int2 place = a.chunk_rows[blockIdx.x / pairs];
    float4 v[4][2];
    float step = 0.f;
    auto fetch_state = [&](int unit, int slab) {
        const float* state = a.chunk_state + ((size_t)(unit / pairs) * H + unit % pairs * 2) * N * 64 + ((size_t)(slab * 8 + (tid >> 6)) * 64 + (tid & 63)) * 8;
#pragma unroll
        for (int e = 0; e < 4; ++e) cm_load8(v[e][0], v[e][1], state + (size_t)(e >> 1) * N * 64 + (e & 1) * 4 * 512);
    };
    auto fetch = [&](int unit) {                           // what a unit begins with
        fetch_state(unit, 0);
        if (tid < 2 * SS_CHUNK) step = a.chunk_steps[((size_t)(unit / pairs) * H + unit % pairs * 2 + (tid >> 6)) * SS_MATRIX_STEP_FLOATS + SM_ES + (tid & 63)];
        if (tid == 0) known = a.chunk_seen[(size_t)(unit / pairs) * a.G + unit % pairs * 2 / (H / a.G)];
    };
    fetch(blockIdx.x);
    for (int unit = blockIdx.x; unit < units && place.y > 0; unit += gridDim.x) {
        const int c = unit / pairs, h0 = unit % pairs * 2, g = h0 / (H / a.G), first = place.x, n = place.y;
        const SMChunk chunk(a, first, n, h0, g, vec);
        cm_bring(cs, a.chunk_planes + (((size_t)c * a.G + g) * 2 + 1) * ss_plane_bytes(N), slabs * SM_SLAB);
        const int next = unit + gridDim.x;
        if (next < units) place = a.chunk_rows[next / pairs];
        if (tid < 2 * SS_CHUNK) es[tid >> 6][tid & 63] = step;
        if (tid == 0) { seen = 0; from = known >> 16; }
        const float* scores = a.chunk_scores + ((size_t)c * a.G + g) * SS_CHUNK * SS_CHUNK;
        unsigned most_s = 0, most_x = 0, most_w = 0;
        const float skips[2] = {load_as_f(a.d_skip, a.d_dtype, h0), load_as_f(a.d_skip, a.d_dtype, h0 + 1)}, skip = skips[hh];
        for (int slab = 0; slab < slabs; ++slab) {
#pragma unroll
            for (int e = 0; e < 4; ++e) cm_put<true>(ss + (e >> 1) * CM_PLANE + cm_at(tid & 63, (e & 1) * 4 + (tid >> 6)), 2 * CM_PLANE, sm_times(v[e][0], CM_UP), sm_times(v[e][1], CM_UP), most_s);
            if (slab == 0) cm_landed();
            cm_ready();
            if (warp == 0) {
                cm_products(elected, tmem + 128 * slab, tmem + 128 * slab + 64, cm_along(at_smem(ss), 2 * CM_PLANE), cm_along(at_smem(cs) + slab * SM_SLAB, CM_PLANE), cm_idesc(64, false, false));
                if (elected) at_commit(at_smem(&bar));
                __syncwarp();
            }
            if (slab + 1 < slabs) fetch_state(unit, 1);
            else {
#pragma unroll
                for (int e = 0; e < 4; ++e) chunk.eight(v[e][0], v[e][1], chunk.x + (e >> 1) * 64, row + (e & 1) * 32, 8 * group);
            }
            cm_done(&bar, phase, status);
        }
        float4 score[2][2];                                // (both heads')
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int t = row + 32 * e;
            score[e][0] = score[e][1] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (8 * group <= t && t < n) {
                score[e][0] = *reinterpret_cast<const float4*>(scores + t * SS_CHUNK + 8 * group);
                score[e][1] = *reinterpret_cast<const float4*>(scores + t * SS_CHUNK + 8 * group + 4);
            }
        }
        float acc[32];
        cm_read(acc, mine + 64);
        cm_take(acc, mine);
        if (slabs > 1) { cm_take(acc, mine + 192); cm_take(acc, mine + 128); }
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
            const float4 d = *reinterpret_cast<const float4*>(&es[hh][column + i]);
            acc[i] *= d.x; acc[i + 1] *= d.y; acc[i + 2] *= d.z; acc[i + 3] *= d.w;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) cm_put(xs + (e >> 1) * CM_PLANE + cm_at(row + (e & 1) * 32, group), 2 * CM_PLANE, sm_times(v[e][0], CM_UP), sm_times(v[e][1], CM_UP), most_x);
        // weights: scores times a factor of s and one of its run of eight and t, or (t's own run) one of both.  With 128 state rows D x_t joins as a weight of the
        // token itself; with 64 it is most of many outputs and comes as a multiply-add at the end: cut with the others' products it left errors of 6.4 to 6.8e-8 of the
        // outputs' norm where multiply-adds have 4.7 to 5.8 (with 128 rows 7.8e-8 for 1.15e-7)
        float by[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int t = row + (e & 1) * 32;
            const float* steps = a.chunk_steps + ((size_t)c * H + h0 + (e >> 1)) * SS_MATRIX_STEP_FLOATS;
            const float4* from8 = reinterpret_cast<const float4*>(steps + (group < t >> 3 ? SM_FACTOR + 8 * group : SM_INSIDE + 8 * t));
            by[e] = group < t >> 3 ? steps[SM_RUNS + 8 * t + group] : 1.f;
            v[e][0] = from8[0]; v[e][1] = from8[1];
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int k = e >> 1, t = row + (e & 1) * 32;
            const float4 (&sc)[2] = score[e & 1];
            float w[8] = {sc[0].x, sc[0].y, sc[0].z, sc[0].w, sc[1].x, sc[1].y, sc[1].z, sc[1].w};
            const float factor[8] = {v[e][0].x, v[e][0].y, v[e][0].z, v[e][0].w, v[e][1].x, v[e][1].y, v[e][1].z, v[e][1].w};
#pragma unroll
            for (int i = 0; i < 8; ++i) w[i] = 8 * group + i > t ? 0.f : fmaf(w[i], factor[i] * by[e], 8 * group + i == t && slabs > 1 ? skips[k] : 0.f);
            cm_put(wgt + k * CM_PLANE + cm_at(t, group), 2 * CM_PLANE, sm_times(make_float4(w[0], w[1], w[2], w[3]), CM_UP), sm_times(make_float4(w[4], w[5], w[6], w[7]), CM_UP), most_w);
        }
        cm_report(&seen, cm_seen(most_s, 2) | cm_seen(most_x, 3) | cm_seen(most_w, 4));
        cm_ready();
        if (seen & 0x18u) {
#pragma unroll 1
            for (int k = 0; k < 2; ++k) {
                cm_mend(xs + k * CM_PLANE, 2 * CM_PLANE, CM_PARTS, &from);
                cm_mend(wgt + k * CM_PLANE, 2 * CM_PLANE, CM_PARTS, &from);
            }
            cm_ready();
        }
        if (warp == 0) {
            cm_products(elected, tmem, tmem + 128, cm_across(at_smem(xs), 2 * CM_PLANE, CM_PLANE), cm_along(at_smem(wgt), 2 * CM_PLANE), cm_idesc(128, true, false));
            if (elected) at_commit(at_smem(&bar));
            __syncwarp();
        }
        float* y = a.y + (size_t)(first + column) * inner + (h0 + hh) * 64 + p;
        const int exact = seen >> 2 & 1u ? 0 : min(n, (int)from);      // tokens in front of it have their outputs from the parts
        if (next < units) fetch(next);
        cm_done(&bar, phase, status);
        cm_take(acc, mine + hh * 64);
        cm_take(acc, mine + hh * 64 + 128);
        cm_scale(acc, CM_DOWN * CM_DOWN);
        if (slabs == 1) {                                  // D x_t, from its parts
            const unsigned char* xt = xs + hh * CM_PLANE + column * 128 + (p & 7) * 2;
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                const unsigned char* at = xt + cm_at(i, p >> 3);
                const auto part = [&](int q) { return __uint_as_float((unsigned)*reinterpret_cast<const unsigned short*>(at + q * 2 * CM_PLANE) << 16); };
                acc[i] = fmaf(skip, ((part(2) + part(1)) + part(0)) * CM_DOWN, acc[i]);
            }
        }
        if (exact == SS_CHUNK) {
#pragma unroll
            for (int i = 0; i < 32; ++i) y[i * inner] = acc[i];
        } else {
#pragma unroll
            for (int i = 0; i < 32; ++i)
                if (column + i < exact) y[i * inner] = acc[i];
        }
        if (tid == 0) {
            a.unit_exact[unit] = exact;
            if (exact < n) odd = 1;
        }
    }
    cm_end(tmem);
    if (!odd) return;                                      // (the walks behind the loop: inside they cost its registers)
    __shared__ ScanArgs args;
    if (tid == 0) args = a;
    __syncthreads();
#pragma unroll 1
    for (int unit = blockIdx.x; unit < units; unit += gridDim.x) {
        const int c = unit / pairs, h0 = unit % pairs * 2, g = h0 / (H / a.G);
        const int2 at = a.chunk_rows[c];
        if (at.y <= 0) break;
        const int exact = a.unit_exact[unit];
        float* state = a.chunk_state + ((size_t)c * H + h0) * N * 64;
        if (exact >= at.y) continue;
        if (N == 64) sm_walk<64>(args, c, at.x, at.y, h0, g, state, exact, nullptr);
        else sm_walk<128>(args, c, at.x, at.y, h0, g, state, exact, nullptr);
    }
}

template <typename T>
static int sm_run(ScanArgs a, int* status, cudaStream_t s) {
    const int vec = a.xbc_ld % 4 == 0 && (uintptr_t)a.xbc % 16 == 0;
    PE_TRY(cudaFuncSetAttribute(sm_steps_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * SM_SLAB));
    PE_TRY(cudaFuncSetAttribute(sm_contribution_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SM_CONTRIBUTION_SMEM));
    PE_TRY(cudaFuncSetAttribute(sm_output_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SM_OUTPUT_SMEM));
    const int units = a.slab * (a.H / 2), blocks = units < 2 * pe_sm_count() ? units : 2 * pe_sm_count();
    for (; a.first_chunk < a.chunks; a.first_chunk += a.slab) {      // (the carry between two slabs lies in the sequences' states)
        PE_TRY(pe_launch(sm_steps_kernel<T>, dim3(a.slab, a.G + (a.H + 7) / 8), SM_THREADS, 2 * SM_SLAB, s, a, vec));
        PE_LAUNCH_CHECK();
        PE_TRY(pe_launch(sm_contribution_kernel, blocks, SM_FEW, SM_CONTRIBUTION_SMEM, s, a, vec, units, status));
        PE_LAUNCH_CHECK();
        PE_TRY(pe_launch(sm_carry_kernel, dim3(a.H * 8, a.B), 2 * a.N, a.N * 8 * 4, s, a));
        PE_LAUNCH_CHECK();
        PE_TRY(pe_launch(sm_output_kernel, blocks, SM_FEW, SM_OUTPUT_SMEM, s, a, vec, units, status));
        PE_LAUNCH_CHECK();
    }
    return 0;
}

int ss_tensor_tiles(const ScanArgs& a, int dtype, int* status, cudaStream_t s) {
    if (a.H + a.G > 65535) return PE_ERR_UNSUPPORTED;
    return dtype == PE_F32 ? sm_run<float>(a, status, s) : sm_run<bf16>(a, status, s);
}
