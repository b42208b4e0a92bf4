// The recurrence of retention.cu over portions of prompts, in chunks of 64 tokens on the tensor cores:
//     S_t = a_t S_(t-1) + s_t k_t v_t^T,   o_t = S_t^T q_t        (a_t: a decay of the head or of the token, s_t: a key scale)
// With L_i = a_1 ... a_i inside a chunk and S the state before it,
//     o_i = L_i S^T q_i + sum_{j <= i} (L_i / L_j) s_j (q_i . k_j) v_j,      S' = L_64 S + sum_j (L_64 / L_j) s_j k_j v_j^T
// so that what a chunk adds to the state, and its outputs once its first state is known, are products of matrices; only the
// states themselves are a chain, of one multiply-add an element and chunk.  Three kernels:
//   chunk_states    a block per (chunk, head): what the chunk adds to the state, [v_dim x k_dim], into scratch memory
//   chunk_prefix    a thread per four state elements walks the request's chunks: leaves the state before each in place
//   chunk_outputs   a block per (chunk, head, half of the value dims): scores q_i . k_j times the decays between, the outputs
// The token-by-token scan is a chain of as many links as there are tokens, with one block of four warps an SM.  Measured, 16
// heads of 128 x 128, 16-bit values: 2,048 tokens of one request 332 -> 119 us (states 29, prefix 13, outputs 75), 512 tokens
// 88 -> 41, 256 tokens 47 -> 38, 8 requests of 128 99 -> 65; 32 heads 439 -> 232.  What bounds it: chunk_outputs issues an
// instruction in 29 of 100 cycles, seven warps an SM that wait for one another's products (registers hold no more).
//
// Everything stays 32-bit: a product of 32-bit numbers is three tensor-core products of their leading and trailing halves
// (x = hi + lo, each 11 bits wide: hi hi + hi lo + lo hi, 2^-22 of a product left out), a 16-bit value is a leading half by
// itself, and the sums are 32-bit.  Ratios of decays come from sums of their logarithms in 64-bit, so they are exact to a
// rounding however far apart the two tokens are.  Relative error against 64-bit, here and token by token, 2,048 tokens, decays
// of 1 - 2^-5 to 1 - 2^-11.6: outputs 3.2e-7 and 5.0e-7, state 3.4e-7 and 6.0e-7.  It grows less with the number of tokens
// that a state remembers and starts higher: equal at a decay of 0.99 (1.9e-7), 1.8e-7 and 1.3e-7 at 0.97.
//
// A value that is not finite leaves the outputs of its request undefined from its chunk of 16 tokens on.
#include "common.cuh"

namespace {

constexpr int CHUNK = 64, THREADS = 256;

struct ChunkParams {
    const float* q; const float* k;          // [tokens, qk_heads * DK]
    const void* v; int v_ld;                 // [tokens, H * DV], 16-bit or 32-bit
    const float* decay;                      // [H] or null
    const float* decay_tok;                  // [tokens, H] or null
    const float* kscale_tok;                 // [tokens, H] or null
    float* state;                            // [slots, H, DV, DK]
    const int* q_start; const int* q_len; const int* state_slots;
    float* out;                              // [tokens, H * DV]
    float* adds;                             // [chunks, H, DV, DK]: what a chunk adds, then the state before it
    float* spans;                            // [chunks, H]: L_64 of the chunk
    int n_requests, H, qk_heads;
};

// Chunk `place` of all requests' chunks laid end to end: its request (-1: none), its first token within it.
struct Where { int request, token; };
__device__ __forceinline__ int chunks_of(const ChunkParams& p, int r) {
    return p.state_slots[r] >= 0 ? (max(p.q_len[r], 0) + CHUNK - 1) / CHUNK : 0;
}
__device__ __forceinline__ Where find_chunk(const ChunkParams& p, int place) {      // by a whole warp
    const int lane = threadIdx.x & 31;
    int base = 0;
    for (int r0 = 0; r0 < p.n_requests; r0 += 32) {
        const int n = r0 + lane < p.n_requests ? chunks_of(p, r0 + lane) : 0;
        int upto = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int x = __shfl_up_sync(0xffffffffu, upto, o); if (lane >= o) upto += x; }
        const unsigned here = __ballot_sync(0xffffffffu, base + upto > place);
        if (here) {
            const int l = __ffs(here) - 1;
            const int first = __shfl_sync(0xffffffffu, base + upto - n, l);
            return {r0 + l, (place - first) * CHUNK};
        }
        base += __shfl_sync(0xffffffffu, upto, 31);
    }
    return {-1, 0};
}

// x = hi + lo: hi is x rounded to the 11 bits of a tensor-core operand, lo the rest cut to as many.  Bit operations: the
// conversion instruction runs at a quarter of their rate.
struct Halves { uint32_t hi, lo; };
__device__ __forceinline__ Halves halves(float x) {
    Halves h;
    h.hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
    h.lo = __float_as_uint(x - __uint_as_float(h.hi)) & 0xffffe000u;      // a NaN becomes a zero and a NaN
    return h;
}
struct HalvesA { Halves x0, x1, x2, x3; };
__device__ __forceinline__ void mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_from_zero(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void add(float (&sums)[4], const float (&x)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) sums[i] += x[i];
}
// sums += A B over one step of eight, and over two steps whose B is four neighbouring numbers of a lane.  The tensor cores cut
// the sums they form where an ordinary addition rounds them, a bias that adds up along a chain of products.  So a product of
// one or two steps starts from zero, small terms first, and is added to the running sums by ordinary additions (chained through
// the accumulators, the outputs' error was three times the token-by-token scan's).
__device__ __forceinline__ void add_one(float (&sums)[4], const HalvesA& a, const Halves& b0, const Halves& b1) {
    float t[4];
    mma_from_zero(t, a.x0.lo, a.x1.lo, a.x2.lo, a.x3.lo, b0.hi, b1.hi);
    mma(t, a.x0.hi, a.x1.hi, a.x2.hi, a.x3.hi, b0.lo, b1.lo);
    mma(t, a.x0.hi, a.x1.hi, a.x2.hi, a.x3.hi, b0.hi, b1.hi);
    add(sums, t);
}
__device__ __forceinline__ void add_two(float (&sums)[4], const HalvesA& a, const HalvesA& b, float4 with) {
    const Halves x = halves(with.x), y = halves(with.y), z = halves(with.z), w = halves(with.w);
    float t[4];
    mma_from_zero(t, a.x0.lo, a.x1.lo, a.x2.lo, a.x3.lo, x.hi, y.hi);
    mma(t, a.x0.hi, a.x1.hi, a.x2.hi, a.x3.hi, x.lo, y.lo);
    mma(t, b.x0.lo, b.x1.lo, b.x2.lo, b.x3.lo, z.hi, w.hi);
    mma(t, b.x0.hi, b.x1.hi, b.x2.hi, b.x3.hi, z.lo, w.lo);
    mma(t, a.x0.hi, a.x1.hi, a.x2.hi, a.x3.hi, x.hi, y.hi);
    mma(t, b.x0.hi, b.x1.hi, b.x2.hi, b.x3.hi, z.hi, w.hi);
    add(sums, t);
}

// The chunk's decays: logs[i] = log2 |L_i| in 64-bit, signs[i] = the sign of L_i, scales[i] = s_i (0 from n on).  By one warp.
// A decay of zero counts as 2^-1100: what lies before it is lost below any 32-bit number.
__device__ __forceinline__ void chunk_decays(const ChunkParams& p, int h, size_t token0, int n, double* logs, float* signs, float* scales) {
    const int lane = threadIdx.x & 31;
    double upto = 0.0;
    float sign = 1.f;
#pragma unroll
    for (int half = 0; half < CHUNK / 32; ++half) {
        const int i = half * 32 + lane;
        float a = 1.f, s = 0.f;
        if (i < n) {
            a = p.decay_tok ? p.decay_tok[(token0 + i) * p.H + h] : p.decay[h];
            s = p.kscale_tok ? p.kscale_tok[(token0 + i) * p.H + h] : 1.f;
        }
        double x = a == 0.f ? -1100.0 : log2((double)fabsf(a));
        float sg = a < 0.f ? -1.f : 1.f;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double y = __shfl_up_sync(0xffffffffu, x, o);
            const float z = __shfl_up_sync(0xffffffffu, sg, o);
            if (lane >= o) { x += y; sg *= z; }
        }
        logs[i] = upto + x; signs[i] = sign * sg; scales[i] = s;
        upto += __shfl_sync(0xffffffffu, x, 31);
        sign *= __shfl_sync(0xffffffffu, sg, 31);
    }
}

// Rows [CHUNK] x WIDTH of a matrix into shared memory as floats, rows from n on zero: 32-bit rows by asynchronous copies (the
// caller waits for them), 16-bit ones through registers, all loads of a thread in flight at once.
template <typename T, int WIDTH, int NTHREADS>
__device__ __forceinline__ void stage(float* dst, int pitch, const T* src, size_t ld, int n) {
    constexpr int PER = WIDTH / 4, MINE = CHUNK * PER / NTHREADS;
    static_assert(MINE * NTHREADS == CHUNK * PER, "the threads share the rows evenly");
    if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (int i = 0; i < MINE; ++i) {
            const int e = threadIdx.x + i * NTHREADS, r = e / PER, c = (e % PER) * 4;
            const uint32_t to = (uint32_t)__cvta_generic_to_shared(dst + r * pitch + c);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(to), "l"(src + (size_t)(r < n ? r : 0) * ld + c), "r"(r < n ? 16 : 0) : "memory");
        }
    } else {
        uint2 raw[MINE];
#pragma unroll
        for (int i = 0; i < MINE; ++i) {
            const int e = threadIdx.x + i * NTHREADS, r = e / PER, c = (e % PER) * 4;
            raw[i] = r < n ? *(const uint2*)(src + (size_t)r * ld + c) : make_uint2(0, 0);
        }
#pragma unroll
        for (int i = 0; i < MINE; ++i) {
            const int e = threadIdx.x + i * NTHREADS, r = e / PER, c = (e % PER) * 4;
            const float2 a = h16x2_to_float2(*(const h16x2*)&raw[i].x), b = h16x2_to_float2(*(const h16x2*)&raw[i].y);
            *(float4*)(dst + r * pitch + c) = make_float4(a.x, a.y, b.x, b.y);
        }
    }
}
__device__ __forceinline__ void staged() { asm volatile("cp.async.wait_all;" ::: "memory"); __syncthreads(); }

// What the chunk adds to the state: [DV x DK] = V^T (w K), w_j = (L_64 / L_j) s_j, by eight warps of 32 x (DK / WN) each.
// Rows of 8 more than a multiple of 32 floats: the lanes' reads down four tokens and along eight dims meet no bank twice.
template <typename T, int DK, int DV>
__global__ void __launch_bounds__(THREADS, 2)
chunk_states_kernel(const ChunkParams p) {
    constexpr int PK = DK + 8, PV = DV + 8, WM = DV / 32, WN = 8 / WM, NT = DK / WN / 8;
    extern __shared__ __align__(16) float sm[];
    float* ks = sm;
    float* vs = ks + CHUNK * PK;
    __shared__ double logs[CHUNK];
    __shared__ float signs[CHUNK], scales[CHUNK], w[CHUNK];
    pdl_launch_dependents();
    pdl_wait();
    const int place = blockIdx.x, h = blockIdx.y, hq = h / (p.H / p.qk_heads);
    const Where at = find_chunk(p, place);
    if (at.request < 0) return;
    const int n = min(CHUNK, p.q_len[at.request] - at.token);
    const size_t token0 = (size_t)p.q_start[at.request] + at.token;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
    stage<float, DK, THREADS>(ks, PK, p.k + (token0 * p.qk_heads + hq) * DK, (size_t)p.qk_heads * DK, n);
    stage<T, DV, THREADS>(vs, PV, (const T*)p.v + token0 * p.v_ld + (size_t)h * DV, p.v_ld, n);
    if (warp == 0) chunk_decays(p, h, token0, n, logs, signs, scales);
    staged();
    if (tid < CHUNK) w[tid] = exp2f((float)(logs[CHUNK - 1] - logs[tid])) * signs[CHUNK - 1] * signs[tid] * scales[tid];
    if (tid == 0) p.spans[(size_t)place * p.H + h] = exp2f((float)logs[CHUNK - 1]) * signs[CHUNK - 1];
    __syncthreads();
    const int m0 = (warp % WM) * 32, n0 = (warp / WM) * (DK / WN);
    float acc[2][NT][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[m][t][i] = 0.f;
#pragma unroll 2
    for (int j = 0; j < CHUNK; j += 8) {
        HalvesA a[2];
        const float *va = vs + (j + c) * PV + m0 + g, *vb = va + 4 * PV;
#pragma unroll
        for (int m = 0; m < 2; ++m) a[m] = {halves(va[16 * m]), halves(va[16 * m + 8]), halves(vb[16 * m]), halves(vb[16 * m + 8])};
        const float w0 = w[j + c], w1 = w[j + c + 4];
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const Halves b0 = halves(ks[(j + c) * PK + n0 + 8 * t + g] * w0), b1 = halves(ks[(j + c + 4) * PK + n0 + 8 * t + g] * w1);
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                if constexpr (sizeof(T) == 4) {
                    add_one(acc[m][t], a[m], b0, b1);
                } else {                                     // a 16-bit value has no trailing half
                    float x[4];
                    mma_from_zero(x, a[m].x0.hi, a[m].x1.hi, a[m].x2.hi, a[m].x3.hi, b0.lo, b1.lo);
                    mma(x, a[m].x0.hi, a[m].x1.hi, a[m].x2.hi, a[m].x3.hi, b0.hi, b1.hi);
                    add(acc[m][t], x);
                }
            }
        }
    }
    float* dst = p.adds + ((size_t)place * p.H + h) * DV * DK;
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            float* at0 = dst + (size_t)(m0 + 16 * m + g) * DK + n0 + 8 * t + 2 * c;
            *(float2*)at0 = make_float2(acc[m][t][0], acc[m][t][1]);
            *(float2*)(at0 + 8 * DK) = make_float2(acc[m][t][2], acc[m][t][3]);
        }
}

// Four elements of a head's state through the chunks of one request.  The loads of four chunks are in flight at a time.
__global__ void __launch_bounds__(THREADS)
chunk_prefix_kernel(const ChunkParams p, int elements) {
    pdl_launch_dependents();
    pdl_wait();
    const int req = blockIdx.z, h = blockIdx.y, e = (blockIdx.x * THREADS + threadIdx.x) * 4, lane = threadIdx.x & 31;
    const int len = p.q_len[req], slot = p.state_slots[req];
    if (len <= 0 || slot < 0) return;
    int before = 0;                                          // chunks of the requests before this one
    for (int r0 = 0; r0 < req; r0 += 32) {
        int n = r0 + lane < req ? chunks_of(p, r0 + lane) : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
        before += n;
    }
    if (e >= elements) return;
    const int chunks = (len + CHUNK - 1) / CHUNK;
    float4* st = (float4*)(p.state + ((size_t)slot * p.H + h) * elements + e);
    float4* add = (float4*)(p.adds + ((size_t)before * p.H + h) * elements + e);
    const float* span = p.spans + (size_t)before * p.H + h;
    const size_t step = (size_t)p.H * elements / 4;
    float4 s = *st;
    for (int i0 = 0; i0 < chunks; i0 += 4) {
        float4 x[4];
        float l[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (i0 + i < chunks) { x[i] = add[(i0 + i) * step]; l[i] = span[(size_t)(i0 + i) * p.H]; }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (i0 + i < chunks) {
                add[(i0 + i) * step] = s;
                s.x = fmaf(l[i], s.x, x[i].x); s.y = fmaf(l[i], s.y, x[i].y);
                s.z = fmaf(l[i], s.z, x[i].z); s.w = fmaf(l[i], s.w, x[i].w);
            }
    }
    *st = s;
}

// The outputs of half of the value dims: a warp owns 16 tokens; it forms its tokens' scores against the keys up to them,
// which are then its 16-row operand as they lie in its registers: step t of the contraction takes tokens 8t + 2c and
// 8t + 2c + 1 for the k of lane c.  Contractions over the key dims take four neighbouring dims a lane and two steps, so that
// queries, keys and the state come as 16-byte pieces; the state's come straight from memory, a step ahead.
constexpr int OUT_THREADS = 128;
template <typename T, int DK, int DV>
__global__ void __launch_bounds__(OUT_THREADS, 2)
chunk_outputs_kernel(const ChunkParams p) {
    constexpr int PK = DK + 16, HV = DV / 2, PV = HV + 4, NT = HV / 8;
    extern __shared__ __align__(16) float sm[];
    float* qs = sm;
    float* ks = qs + CHUNK * PK;
    float* vs = ks + CHUNK * PK;
    __shared__ double logs[CHUNK];
    __shared__ float signs[CHUNK], scales[CHUNK];
    pdl_launch_dependents();
    pdl_wait();
    const int place = blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * HV, hq = h / (p.H / p.qk_heads);
    const Where at = find_chunk(p, place);
    if (at.request < 0) return;
    const int n = min(CHUNK, p.q_len[at.request] - at.token);
    const size_t token0 = (size_t)p.q_start[at.request] + at.token;
    const int tid = threadIdx.x, m = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
    stage<float, DK, OUT_THREADS>(qs, PK, p.q + (token0 * p.qk_heads + hq) * DK, (size_t)p.qk_heads * DK, n);
    stage<float, DK, OUT_THREADS>(ks, PK, p.k + (token0 * p.qk_heads + hq) * DK, (size_t)p.qk_heads * DK, n);
    stage<T, HV, OUT_THREADS>(vs, PV, (const T*)p.v + token0 * p.v_ld + (size_t)h * DV + v0, p.v_ld, n);
    const int i0 = 16 * m + g, i1 = i0 + 8;
    const float* before = p.adds + ((size_t)place * p.H + h) * DV * DK + (size_t)(v0 + g) * DK;
    float4 s[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t) s[t] = *(const float4*)(before + (size_t)8 * t * DK + 4 * c);
    if (m == 0) chunk_decays(p, h, token0, n, logs, signs, scales);
    staged();
    if (16 * m >= n) return;
    const float *qa = qs + i0 * PK, *qb = qs + i1 * PK;
    float sc[8][4], acc[NT][4];
#pragma unroll
    for (int t = 0; t < 8; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i) sc[t][i] = 0.f;
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[t][i] = 0.f;
#pragma unroll 1
    for (int d = 4 * c; d < DK; d += 16) {
        const float4 a = *(const float4*)(qa + d), b = *(const float4*)(qb + d);
        const HalvesA q0 = {halves(a.x), halves(b.x), halves(a.y), halves(b.y)}, q1 = {halves(a.z), halves(b.z), halves(a.w), halves(b.w)};
        float4 now[NT];
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            now[t] = s[t];
            if (d + 16 < DK) s[t] = *(const float4*)(before + (size_t)8 * t * DK + d + 16);
        }
#pragma unroll
        for (int t = 0; t < 8; ++t)
            if (t < 2 * (m + 1)) add_two(sc[t], q0, q1, *(const float4*)(ks + (8 * t + g) * PK + d));
#pragma unroll
        for (int t = 0; t < NT; ++t) add_two(acc[t], q0, q1, now[t]);
    }
    const double la = logs[i0], lb = logs[i1];
    const float fa = exp2f((float)la) * signs[i0], fb = exp2f((float)lb) * signs[i1];
#pragma unroll
    for (int t = 0; t < NT; ++t) { acc[t][0] *= fa; acc[t][1] *= fa; acc[t][2] *= fb; acc[t][3] *= fb; }
#pragma unroll
    for (int t = 0; t < 8; ++t)
        if (t < 2 * (m + 1)) {
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const int j = 8 * t + 2 * c + x;
                const double lj = logs[j];
                const float sj = scales[j] * signs[j];
                sc[t][x] = j <= i0 ? sc[t][x] * (exp2f((float)(la - lj)) * signs[i0] * sj) : 0.f;
                sc[t][2 + x] = j <= i1 ? sc[t][2 + x] * (exp2f((float)(lb - lj)) * signs[i1] * sj) : 0.f;
            }
            const HalvesA a = {halves(sc[t][0]), halves(sc[t][2]), halves(sc[t][1]), halves(sc[t][3])};
            const float* vr = vs + (8 * t + 2 * c) * PV + g;
#pragma unroll
            for (int u = 0; u < NT; ++u) {
                if constexpr (sizeof(T) == 4) {
                    add_one(acc[u], a, halves(vr[8 * u]), halves(vr[PV + 8 * u]));
                } else {
                    const uint32_t b0 = __float_as_uint(vr[8 * u]), b1 = __float_as_uint(vr[PV + 8 * u]);
                    float x[4];
                    mma_from_zero(x, a.x0.lo, a.x1.lo, a.x2.lo, a.x3.lo, b0, b1);
                    mma(x, a.x0.hi, a.x1.hi, a.x2.hi, a.x3.hi, b0, b1);
                    add(acc[u], x);
                }
            }
        }
    float* dst = p.out + (token0 * p.H + h) * DV + v0 + 2 * c;
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        if (i0 < n) *(float2*)(dst + (size_t)i0 * p.H * DV + 8 * t) = make_float2(acc[t][0], acc[t][1]);
        if (i1 < n) *(float2*)(dst + (size_t)i1 * p.H * DV + 8 * t) = make_float2(acc[t][2], acc[t][3]);
    }
}

template <typename K>
int allow_smem(K kernel, size_t smem) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) cudaGetLastError();
    return (int)e;
}

template <typename T, int DK, int DV>
int launch(const ChunkParams& p, int chunks, cudaStream_t stream) {
    const size_t s1 = sizeof(float) * CHUNK * (DK + 8 + DV + 8), s3 = sizeof(float) * CHUNK * (2 * (DK + 16) + DV / 2 + 4);
    if (const int rc = allow_smem(chunk_states_kernel<T, DK, DV>, s1)) return rc;
    if (const int rc = allow_smem(chunk_outputs_kernel<T, DK, DV>, s3)) return rc;
    if (const int rc = tnx_launch_in_order(chunk_states_kernel<T, DK, DV>, dim3(chunks, p.H), dim3(THREADS), s1, stream, p)) return rc;
    if (const int rc = tnx_launch_in_order(chunk_prefix_kernel, dim3(DK * DV / (4 * THREADS), p.H, p.n_requests), dim3(THREADS), 0, stream, p, DK * DV)) return rc;
    return tnx_launch_in_order(chunk_outputs_kernel<T, DK, DV>, dim3(chunks, p.H, 2), dim3(OUT_THREADS), s3, stream, p);
}
template <typename T>
int launch_sizes(const ChunkParams& p, int dk, int dv, int chunks, cudaStream_t stream) {
    if (dk == 128 && dv == 128) return launch<T, 128, 128>(p, chunks, stream);
    if (dk == 128 && dv == 64) return launch<T, 128, 64>(p, chunks, stream);
    if (dk == 64 && dv == 64) return launch<T, 64, 64>(p, chunks, stream);
    if (dk == 64 && dv == 128) return launch<T, 64, 128>(p, chunks, stream);
    return TNX_ERR_UNSUPPORTED;
}

}  // namespace

// The most chunks that `tokens` tokens of `n_requests` requests can be cut into.
TNX_EXPORT int tnx_retention_chunks(int tokens, int n_requests) { return tokens / CHUNK + n_requests; }

// As tnx_retention_scan; adds holds tnx_retention_chunks x H x dv x dk floats, spans tnx_retention_chunks x H.
TNX_EXPORT int tnx_retention_chunked(const float* q, const float* k, const void* v, int v_ld, const float* decay, float* state,
                                     const int* q_start, const int* q_len, const int* state_slots, float* out, int tokens,
                                     int n_requests, int H, int dk, int dv, int v_h16, const float* decay_tok,
                                     const float* kscale_tok, int qk_heads, float* adds, float* spans, cudaStream_t stream) {
    if (n_requests <= 0 || tokens <= 0) return 0;
    if (H <= 0 || H > 65535 || n_requests > 65535 || qk_heads <= 0 || H % qk_heads || (!decay && !decay_tok) || !adds || !spans)
        return TNX_ERR_BAD_ARG;
    const int vsize = v_h16 ? 2 : 4;
    if ((((uintptr_t)q | (uintptr_t)k | (uintptr_t)state | (uintptr_t)out | (uintptr_t)adds) & 15) || ((uintptr_t)v % (4 * vsize)) || v_ld % 4)
        return TNX_ERR_UNSUPPORTED;
    const ChunkParams p{q, k, v, v_ld, decay, decay_tok, kscale_tok, state, q_start, q_len, state_slots, out, adds, spans, n_requests, H, qk_heads};
    const int chunks = tnx_retention_chunks(tokens, n_requests);
    return v_h16 ? launch_sizes<h16>(p, dk, dv, chunks, stream) : launch_sizes<float>(p, dk, dv, chunks, stream);
}
