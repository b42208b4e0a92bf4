// The recurrence of retention.cu over portions of prompts, in chunks of 64 tokens on the tensor cores:
//     S_t = a S_(t-1) + k_t v_t^T,   o_t = S_t^T q_t        (a: the head's decay)
// With tokens numbered from 0 inside a chunk of n and S the state before it,
//     o_i = a^(i+1) S^T q_i + sum_{j <= i} a^(i-j) (q_i . k_j) v_j,      S' = a^n S + sum_j a^(n-1-j) k_j v_j^T
// so that what a chunk adds to the state, and its outputs once its first state is known, are products of matrices; only the
// states themselves are a chain, of one multiply-add an element and chunk.  Three kernels:
//   chunk_states    a block per (chunk, head): what the chunk adds to the state, [v_dim x k_dim], into scratch memory
//   chunk_prefix    a thread per four state elements walks the request's chunks: leaves the state before each in place
//   chunk_outputs   a block per (chunk, head, half of the value dims): scores q_i . k_j times the decays between, the outputs
// The token-by-token scan is a chain of as many links as there are tokens, with one block of four warps an SM.  Measured, 16
// heads of 128 x 128, 16-bit values: 2,048 tokens of one request 332 -> 122 us, 512 tokens 88 -> 39, four requests of 512
// 122; 32 heads 439 -> 243.  What bounds it: chunk_outputs, seven warps an SM that wait for one another's products (registers
// hold no more).
//
// Everything stays 32-bit: a 32-bit number is the sum of three bfloat16 numbers, all its 24 bits, a product of two of them six
// products of the terms (what is left out is 2^-25 of it), and the sums are 32-bit.  A power of the decay is formed in 64-bit
// and rounded once.  Relative error against 64-bit, token by token and here, 1,024 tokens (with operands of two times 11 bits
// and powers from 32-bit logarithms): outputs at a decay of 0.5 8.8e-8 and 8.6e-8 (1.5e-7), at 0.9 1.0e-7 and 8.9e-8 (1.7e-7),
// at 0.97 1.3e-7 and 9.4e-8 (1.9e-7), at 0.99 2.0e-7 and 1.0e-7 (1.9e-7), at 0.9997 4.7e-7 and 1.2e-7 (2.3e-7); the state at
// 0.5 4.0e-8 and 6.0e-8, at 0.9 6.4e-8 and 6.3e-8, at 0.97 1.1e-7 and 6.5e-8, at 0.9997 5.8e-7 and 1.1e-7.
#include "common.cuh"

namespace {

constexpr int CHUNK = 64, THREADS = 256;

struct ChunkParams {
    const float* q; const float* k;          // [tokens, H * DK]
    const void* v; int v_ld;                 // [tokens, H * DV], 16-bit or 32-bit
    const float* decay;                      // [H]
    float* state;                            // [slots, H, DV, DK]
    const int* q_start; const int* q_len; const int* state_slots;
    float* out;                              // [tokens, H * DV]
    float* adds;                             // [chunks, H, DV, DK]: what a chunk adds, then the state before it
    float* spans;                            // [chunks, H]: the chunk's decay, a to its number of tokens
    int n_requests, H;
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

// Two numbers as pairs of bfloat16 numbers, one pair a term: eight bits each, so that three terms are a 32-bit number exactly,
// two a float16 number and one a bfloat16 number.
template <int TERMS> __device__ __forceinline__ void split(float x, float y, uint32_t (&out)[TERMS]) {
#pragma unroll
    for (int i = 0; i < TERMS; ++i) {
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(out[i]) : "f"(y), "f"(x));
        if (i + 1 < TERMS) { x -= __uint_as_float(out[i] << 16); y -= __uint_as_float(out[i] & 0xffff0000u); }
    }
}
// Operands of a product over sixteen: a lane has rows g and g + 8 (or column g) at four places, which may be any four as long as
// both operands agree on them.
template <int TERMS> struct Rows { uint32_t x[4][TERMS]; };
template <int TERMS> struct Columns { uint32_t x[2][TERMS]; };
template <int TERMS> __device__ __forceinline__ Rows<TERMS> rows(float4 a, float4 b) {
    Rows<TERMS> r;
    split<TERMS>(a.x, a.y, r.x[0]); split<TERMS>(b.x, b.y, r.x[1]); split<TERMS>(a.z, a.w, r.x[2]); split<TERMS>(b.z, b.w, r.x[3]);
    return r;
}
template <int TERMS> __device__ __forceinline__ Columns<TERMS> columns(float4 a) {
    Columns<TERMS> c;
    split<TERMS>(a.x, a.y, c.x[0]); split<TERMS>(a.z, a.w, c.x[1]);
    return c;
}
template <bool FROM_ZERO, int TA, int TB>
__device__ __forceinline__ void mma(float (&d)[4], const Rows<TA>& a, int i, const Columns<TB>& b, int j) {
    if constexpr (FROM_ZERO)
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
            : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a.x[0][i]), "r"(a.x[1][i]), "r"(a.x[2][i]), "r"(a.x[3][i]), "r"(b.x[0][j]), "r"(b.x[1][j]), "f"(0.f));
    else
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a.x[0][i]), "r"(a.x[1][i]), "r"(a.x[2][i]), "r"(a.x[3][i]), "r"(b.x[0][j]), "r"(b.x[1][j]));
}
// sums += A B over sixteen: the terms' products whose places add up to two, one and none (2^-16, 2^-8 and 1 of the whole; beyond
// two they are 2^-25 and less) each from zero, then added by ordinary additions, small ones first.  The tensor cores cut the sums
// they form where an ordinary addition rounds them, a bias that adds up along a chain of products (chained through the
// accumulators, the outputs' error was three times the token-by-token scan's).
template <int TA, int TB>
__device__ __forceinline__ void add_product(float (&sums)[4], const Rows<TA>& a, const Columns<TB>& b) {
    float lead[4], next[4], last[4];
    mma<true>(lead, a, 0, b, 0);
    if constexpr (TB > 1) {
        mma<true>(next, a, 0, b, 1);
        if constexpr (TA > 1) mma<false>(next, a, 1, b, 0);
    } else if constexpr (TA > 1) {
        mma<true>(next, a, 1, b, 0);
    }
    if constexpr (TA > 1 && TB > 1) {
        mma<true>(last, a, 1, b, 1);
        if constexpr (TB > 2) mma<false>(last, a, 0, b, 2);
        if constexpr (TA > 2) mma<false>(last, a, 2, b, 0);
    } else if constexpr (TA > 2) {
        mma<true>(last, a, 2, b, 0);
    } else if constexpr (TB > 2) {
        mma<true>(last, a, 0, b, 2);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if constexpr (TA > 2 || TB > 2 || (TA > 1 && TB > 1)) next[i] += last[i];
        if constexpr (TA > 1 || TB > 1) lead[i] += next[i];
        sums[i] += lead[i];
    }
}
// Terms of a value of the stored type.
#ifdef TNX_F16
constexpr int H16_TERMS = 2;
#else
constexpr int H16_TERMS = 1;
#endif
template <typename T> __host__ __device__ constexpr int terms_of() { return sizeof(T) == 4 ? 3 : H16_TERMS; }

// powers[n] = a^n for n up to CHUNK, formed in 64-bit and rounded once, by the block's first threads (the caller synchronises).
__device__ __forceinline__ void chunk_decays(float a, float* powers) {
    if (threadIdx.x > CHUNK) return;
    double p = 1.0, square = (double)a;
#pragma unroll
    for (int bit = 1; bit <= CHUNK; bit <<= 1, square *= square)
        if ((int)threadIdx.x & bit) p *= square;
    powers[threadIdx.x] = (float)p;
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

// What a chunk of n tokens adds to the state: [DV x DK] = V^T (w K), w_j = a^(n - 1 - j), by eight warps of 32 x (DK / WN) each.
// Rows of 4 more than a multiple of 32 floats: the lanes' reads down every second of eight tokens and along eight dims meet no
// bank twice.
template <typename T, int DK, int DV>
__global__ void __launch_bounds__(THREADS, 2)
chunk_states_kernel(const ChunkParams p) {
    constexpr int PK = DK + 4, PV = DV + 4, WM = DV / 32, WN = 8 / WM, NT = DK / WN / 8;
    extern __shared__ __align__(16) float sm[];
    float* ks = sm;
    float* vs = ks + CHUNK * PK;
    __shared__ float powers[CHUNK + 1];
    pdl_launch_dependents();
    pdl_wait();
    const int place = blockIdx.x, h = blockIdx.y;
    const Where at = find_chunk(p, place);
    if (at.request < 0) return;
    const int n = min(CHUNK, p.q_len[at.request] - at.token);
    const size_t token0 = (size_t)p.q_start[at.request] + at.token;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
    stage<float, DK, THREADS>(ks, PK, p.k + (token0 * p.H + h) * DK, (size_t)p.H * DK, n);
    stage<T, DV, THREADS>(vs, PV, (const T*)p.v + token0 * p.v_ld + (size_t)h * DV, p.v_ld, n);
    chunk_decays(p.decay[h], powers);
    staged();
    if (tid == 0) p.spans[(size_t)place * p.H + h] = powers[n];
    const int m0 = (warp % WM) * 32, n0 = (warp / WM) * (DK / WN);
    float acc[2][NT][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[m][t][i] = 0.f;
#pragma unroll 2
    for (int j = 0; j < CHUNK; j += 16) {
        const int j0 = j + 2 * c;                    // the lane's tokens: j0, j0 + 1, j0 + 8, j0 + 9
        Rows<terms_of<T>()> a[2];
        const float* va = vs + j0 * PV + m0 + g;
#pragma unroll
        for (int m = 0; m < 2; ++m, va += 16)
            a[m] = rows<terms_of<T>()>(make_float4(va[0], va[PV], va[8 * PV], va[9 * PV]),
                                       make_float4(va[8], va[PV + 8], va[8 * PV + 8], va[9 * PV + 8]));
        const float w0 = powers[max(n - 1 - j0, 0)], w1 = powers[max(n - 2 - j0, 0)];              // keys from n on are zero
        const float w2 = powers[max(n - 9 - j0, 0)], w3 = powers[max(n - 10 - j0, 0)];
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const float* ka = ks + j0 * PK + n0 + 8 * t + g;
            const Columns<3> b = columns<3>(make_float4(ka[0] * w0, ka[PK] * w1, ka[8 * PK] * w2, ka[9 * PK] * w3));
#pragma unroll
            for (int m = 0; m < 2; ++m) add_product(acc[m][t], a[m], b);
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
// which are then its 16-row operand as they lie in its registers (tokens 8t + 2c and 8t + 2c + 1 of two tiles t).
// Contractions over the key dims take four neighbouring dims a lane, so that queries, keys and the state come as 16-byte pieces; the state's come straight from memory, a step ahead.
constexpr int OUT_THREADS = 128;
template <typename T, int DK, int DV>
__global__ void __launch_bounds__(OUT_THREADS, 2)
chunk_outputs_kernel(const ChunkParams p) {
    constexpr int PK = DK + 16, HV = DV / 2, PV = HV + 4, NT = HV / 8;
    extern __shared__ __align__(16) float sm[];
    float* qs = sm;
    float* ks = qs + CHUNK * PK;
    float* vs = ks + CHUNK * PK;
    __shared__ float powers[CHUNK + 1];
    pdl_launch_dependents();
    pdl_wait();
    const int place = blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * HV;
    const Where at = find_chunk(p, place);
    if (at.request < 0) return;
    const int n = min(CHUNK, p.q_len[at.request] - at.token);
    const size_t token0 = (size_t)p.q_start[at.request] + at.token;
    const int tid = threadIdx.x, m = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
    stage<float, DK, OUT_THREADS>(qs, PK, p.q + (token0 * p.H + h) * DK, (size_t)p.H * DK, n);
    stage<float, DK, OUT_THREADS>(ks, PK, p.k + (token0 * p.H + h) * DK, (size_t)p.H * DK, n);
    stage<T, HV, OUT_THREADS>(vs, PV, (const T*)p.v + token0 * p.v_ld + (size_t)h * DV + v0, p.v_ld, n);
    const int i0 = 16 * m + g, i1 = i0 + 8;
    const float* before = p.adds + ((size_t)place * p.H + h) * DV * DK + (size_t)(v0 + g) * DK;
    float4 s[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t) s[t] = *(const float4*)(before + (size_t)8 * t * DK + 4 * c);
    chunk_decays(p.decay[h], powers);
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
        const Rows<3> q = rows<3>(a, b);
        float4 now[NT];
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            now[t] = s[t];
            if (d + 16 < DK) s[t] = *(const float4*)(before + (size_t)8 * t * DK + d + 16);
        }
#pragma unroll
        for (int t = 0; t < 8; ++t)
            if (t < 2 * (m + 1)) add_product(sc[t], q, columns<3>(*(const float4*)(ks + (8 * t + g) * PK + d)));
#pragma unroll
        for (int t = 0; t < NT; ++t) add_product(acc[t], q, columns<3>(now[t]));
    }
    const float fa = powers[i0 + 1], fb = powers[i1 + 1];
#pragma unroll
    for (int t = 0; t < NT; ++t) { acc[t][0] *= fa; acc[t][1] *= fa; acc[t][2] *= fb; acc[t][3] *= fb; }
#pragma unroll
    for (int t = 0; t < 8; ++t)
        if (t < 2 * (m + 1)) {
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const int j = 8 * t + 2 * c + x;
                sc[t][x] = j <= i0 ? sc[t][x] * powers[max(i0 - j, 0)] : 0.f;
                sc[t][2 + x] = j <= i1 ? sc[t][2 + x] * powers[max(i1 - j, 0)] : 0.f;
            }
        }
#pragma unroll
    for (int t = 0; t < 8; t += 2)
        if (t < 2 * (m + 1)) {
            const Rows<3> a = rows<3>(make_float4(sc[t][0], sc[t][1], sc[t + 1][0], sc[t + 1][1]),
                                      make_float4(sc[t][2], sc[t][3], sc[t + 1][2], sc[t + 1][3]));
            const float* vr = vs + (8 * t + 2 * c) * PV + g;
#pragma unroll
            for (int u = 0; u < NT; ++u) {
                float4 y = make_float4(vr[8 * u], vr[PV + 8 * u], vr[8 * PV + 8 * u], vr[9 * PV + 8 * u]);
                if (t == 2 * m && __any_sync(0xffffffffu, !(isfinite(y.x) && isfinite(y.y) && isfinite(y.z) && isfinite(y.w)))) {
                    // The tiles have later tokens beside earlier ones, whose scores are zeros, and zero times such a value is
                    // none: it is left out of the product and marks its own and later tokens by itself.
                    y.x = isfinite(y.x) ? y.x : 0.f; y.y = isfinite(y.y) ? y.y : 0.f;
                    y.z = isfinite(y.z) ? y.z : 0.f; y.w = isfinite(y.w) ? y.w : 0.f;
#pragma unroll 1
                    for (int j = 8 * t; j < 8 * t + 16; ++j)
#pragma unroll
                        for (int x = 0; x < 2; ++x)
                            if (!isfinite(vs[j * PV + 8 * u + 2 * c + x])) {
                                if (j <= i0) acc[u][x] = NAN;
                                if (j <= i1) acc[u][2 + x] = NAN;
                            }
                }
                add_product(acc[u], a, columns<terms_of<T>()>(y));
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
    const size_t s1 = sizeof(float) * CHUNK * (DK + 4 + DV + 4), s3 = sizeof(float) * CHUNK * (2 * (DK + 16) + DV / 2 + 4);
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

// As tnx_retention_scan with a decay per head; adds holds (tokens / 64 + n_requests) x H x dv x dk floats, spans
// (tokens / 64 + n_requests) x H.
TNX_EXPORT int tnx_retention_chunked(const float* q, const float* k, const void* v, int v_ld, const float* decay, float* state,
                                     const int* q_start, const int* q_len, const int* state_slots, float* out, int tokens,
                                     int n_requests, int H, int dk, int dv, int v_h16, float* adds, float* spans, cudaStream_t stream) {
    if (n_requests <= 0 || tokens <= 0) return 0;
    if (H <= 0 || H > 65535 || n_requests > 65535 || !decay || !adds || !spans)
        return TNX_ERR_BAD_ARG;
    const int vsize = v_h16 ? 2 : 4;
    if ((((uintptr_t)q | (uintptr_t)k | (uintptr_t)state | (uintptr_t)out | (uintptr_t)adds) & 15) || ((uintptr_t)v % (4 * vsize)) || v_ld % 4)
        return TNX_ERR_UNSUPPORTED;
    const ChunkParams p{q, k, v, v_ld, decay, state, q_start, q_len, state_slots, out, adds, spans, n_requests, H};
    const int chunks = tokens / CHUNK + n_requests;          // the most that the tokens can be cut into
    return v_h16 ? launch_sizes<h16>(p, dk, dv, chunks, stream) : launch_sizes<float>(p, dk, dv, chunks, stream);
}
