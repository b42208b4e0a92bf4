// 32-bit activations times a 16-bit matrix on the 5th-generation tensor cores, with every bit of the activations:
//
//   C[m, n] = epilogue( sum_k A[m, k] * W[n, k] )        A: [M, K] float, W: [N, K] h16 (both row-major)
//   epilogue: + bias[n]; activation (by code, common.cuh); + residual[m, n] (32-bit); stored as float or in the 16-bit type.
//
// An activation is the sum of three 16-bit terms, and a product of two 16-bit numbers is exact in 32 bits:
//   bfloat16   a = h + m + l, each the next eight leading bits (cut off, not rounded: 8 + 8 + 8 = 24 bits, the whole number)
//   float16    a row is scaled by a power of two so that its largest element lies in [2^14, 2^15); then a = h + m/2^11 + l/2^22,
//              each rounded to nearest (11 bits a term).  An element down to 2^-37 of the row's largest keeps all 24 bits, a smaller one
//              is off by less than 2^-61 of the largest.
// The three terms' rows are staged one under the other as one operand of 3 BN rows, so one MMA multiplies all of them by a tile
// of 128 features and the weights pass through shared memory once.
//
// The sums.  The tensor cores cut off what an addition to their accumulator shifts out (measured: 1.04e-9 of the sum for every
// element of K, towards zero, while a chain of 32-bit FMAs stays at 1.8e-8 sqrt(K)).  So nothing is left in an accumulator for
// more than CHUNK = 128 elements of K: four warps (eight with two tiles) then take the three terms' sums out, join them and
// go on in registers, chunks to segments of four, segments to the result.  Errors against 64 bits, relative, standard normal
// activations, chain of FMAs -> here: K = 256 2.9e-7 -> 1.9e-7, 768 5.0e-7 -> 1.9e-7, 2048 8.1e-7 -> 2.0e-7, 8192 1.6e-6 -> 2.1e-7.
// The order is the same whatever M, the tile and the split of K are, so a row's result does not depend on the other rows
// of the call, bit for bit.
//
// Infinities and NaN come out as from 32-bit multiplications: such an element is its own first term (and the terms of the
// others in its row are cut to a representable size, they cannot matter beside it, but opposite an infinite weight, so that none
// but zero becomes zero); a sum of first terms that is not finite stands, whatever the other terms say.
//
// Warp roles as in gemm_tc.cu: warp 0 TMA, warp 1 MMAs, warps from 2 on the accumulators; every wait is bounded.  Persistent
// CTAs, one an SM, walk over tiles of 128 NT features by BN tokens (tokens fastest: the CTAs at work share weights in the
// second-level cache).  The two accumulator buffers of 3 BN columns let the MMAs run on while one is taken out; with NT = 2
// they are the two feature tiles', which share the staged activations.
// What bounds it: the issue of MMAs and commits and the operands' way through the second-level cache; 2,048 tokens by
// [8192 x 2048] run at 1.1 PFLOP/s of 16-bit products.  Measured against gemm_simt, 16-bit weights, us, captured calls:
//   tokens   [6144 x 2048]   [2048 x 2048]   [8192 x 2048]   [2048 x 8192]
//   1             -            55 ->  9         71 -> 12           -
//   64        104 -> 17           -               -            323 -> 23
//   502       337 -> 59       149 -> 23        420 -> 60       595 -> 70
//   2,048         -               -         1,440 -> 196          -
// Tried: K blocks of 64 as the rings' unit (a third more waits and commits: 502 tokens by [6144 x 2048] 76 us), a barrier of its
// own for every ring (66), one thread instead of the whole warp along the MMAs' loop (94).
#include "common.cuh"
#include "tc_common.cuh"

namespace {

constexpr int BLOCK_K = 64, UMMA_K = 16, TILE_N = 128;
constexpr int CHUNK_KB = 2;          // K blocks of 64 in a chunk
constexpr int SEG_CHUNKS = 4;        // chunks in a segment: the unit by which K may be split over CTAs
constexpr int SEG_K = SEG_CHUNKS * CHUNK_KB * BLOCK_K;

#ifdef TNX_F16
constexpr float TERM = 4.8828125e-4f;        // 2^-11: what a unit of a term is worth in units of the one before
#else
constexpr float TERM = 1.f;
#endif

__host__ __device__ constexpr uint32_t instr_desc(int n) {
    return (1u << 4) | IDESC_H16_AB | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TILE_N >> 4) << 24);
}

struct Params {
    int M, N, K, ldc, act, c_is_h16;
    int tiles_m, items, splits, segs_per_split;
    const float* bias;
    const float* residual;       // may alias C
    const float* unscale;        // float16: what a row's sums are multiplied by, a power of two
    void* C;
    float* parts;                // K split: [segment][M][N] sums; else null
    int* err;
};

// What every output goes through, in the product itself or after its segments are added.
__device__ __forceinline__ float finish(float sum, float unscale, float bias, int act, float res) {
#ifdef TNX_F16
    sum *= unscale;
#endif
    return apply_activation(sum + bias, act) + res;
}

// A use: the MMAs of one chunk and one feature tile, numbered through a CTA's work.  Use u takes slot u % SLOTS of the weights'
// ring and accumulator buffer u % 2.  The chunk's activations come with its first use.
template <int BN, int NT> struct Shape {
    static constexpr int W_BYTES = CHUNK_KB * TILE_N * BLOCK_K * 2, X_BYTES = CHUNK_KB * 3 * BN * BLOCK_K * 2;       // a chunk
    static constexpr int SLOTS = BN == 16 ? 5 : 4;
    static constexpr int X_SLOTS = BN == 64 ? 2 : SLOTS;
    static constexpr int SMEM = SLOTS * W_BYTES + X_SLOTS * X_BYTES + 1024;
    static constexpr int GROUPS = BN == 64 ? 2 : 1;              // groups of four warps that take the accumulators out:
    static constexpr int TOKENS = NT == 2 ? BN : BN / GROUPS;    // one a feature tile, or each half of the tokens
    static constexpr int THREADS = 64 + GROUPS * 128;
    static constexpr int BUF_COLS = BN == 64 ? 256 : BN == 32 ? 128 : 64;       // columns from one accumulator buffer to the other
    static constexpr int TMEM_COLS = 2 * BUF_COLS;
    static_assert(3 * BN <= BUF_COLS && SMEM <= 232448 - 512, "an accumulator buffer; the shared memory of an SM");
    // A wait tells a phase from the one after it, not from later ones: the activations' slot of chunk c is waited for (by the end
    // of use NT (c - X_SLOTS) + NT - 1) before the weights of SLOTS uses later are asked for.
    static_assert(NT * X_SLOTS <= SLOTS, "one barrier serves both rings");
};

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_u32(dst)), "l"((unsigned long long)map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z) : "memory");
}

template <int BN, int NT>
__global__ void __launch_bounds__(Shape<BN, NT>::THREADS, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const Params p) {
    using S = Shape<BN, NT>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem_w = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* smem_x = smem_w + S::SLOTS * S::W_BYTES;
    __shared__ uint64_t full[S::SLOTS], done[S::SLOTS], empty_acc[2];       // operands are there; MMAs have ended; accumulators are taken out
    __shared__ uint32_t tmem_base_smem;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kbs = (p.K + BLOCK_K - 1) / BLOCK_K;

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < S::SLOTS; ++s) { mbar_init(&full[s], 1); mbar_init(&done[s], 1); }
        for (int b = 0; b < 2; ++b) mbar_init(&empty_acc[b], NT == 2 ? 4 : 4 * S::GROUPS);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&map_w) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&map_x) : "memory");
    }
    if (warp == 1) {
        tmem_alloc(&tmem_base_smem, S::TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_smem;
    bool ok = true;

    // An item: a tile of features (by NT), a tile of tokens, a range of segments; as K blocks [kb0, kb1).
    struct Item { int n0, m0, kb0, kb1; };
    auto item = [&](int i) {
        Item t;
        const int tile = i / p.splits, split = i - tile * p.splits;
        t.m0 = tile % p.tiles_m * BN;
        t.n0 = tile / p.tiles_m * (NT * TILE_N);
        t.kb0 = split * p.segs_per_split * (SEG_CHUNKS * CHUNK_KB);
        t.kb1 = min(kbs, t.kb0 + p.segs_per_split * (SEG_CHUNKS * CHUNK_KB));
        return t;
    };

    if (warp == 0) {
        if (lane == 0) {
            // The weights are no kernel's output: the first ones are asked for before the wait for the kernel ahead.
            // (What lies beyond K is filled with zeros.)
            Ring<S::SLOTS> wr;                           // the use's slot; pass is also that of the use SLOTS before it, inverted
            Ring<S::X_SLOTS> xr;
            int use = 0;
            auto load_w = [&](int kb, int n0, bool with_x) {
                if (!mbar_wait(&done[wr.slot], wr.pass ^ 1, p.err, 61)) return false;
                mbar_expect_tx(&full[wr.slot], S::W_BYTES + (with_x ? S::X_BYTES : 0));
                uint8_t* dst = smem_w + (size_t)wr.slot * S::W_BYTES;
#pragma unroll
                for (int q = 0; q < CHUNK_KB; ++q)
                    tma_load_2d(dst + q * (S::W_BYTES / CHUNK_KB), &map_w, &full[wr.slot], (kb + q) * BLOCK_K, n0);
                wr.next();
                return true;
            };
            auto load_x = [&](int kb, int m0) {          // of the chunk whose first use is `use`
                uint8_t* dst = smem_x + (size_t)xr.slot * S::X_BYTES;
#pragma unroll
                for (int q = 0; q < CHUNK_KB; ++q)
                    tma_load_3d(dst + q * (S::X_BYTES / CHUNK_KB), &map_x, &full[use % S::SLOTS], (kb + q) * BLOCK_K, m0, 0);
                xr.next();
            };
            int early = 0;               // uses of the first item whose weights are asked for ahead of the wait
            if ((int)blockIdx.x < p.items) {
                const Item t = item(blockIdx.x);
                for (; early < S::SLOTS && t.kb0 + early / NT * CHUNK_KB < t.kb1; ++early)
                    load_w(t.kb0 + early / NT * CHUNK_KB, t.n0 + early % NT * TILE_N, early % NT == 0);
            }
            pdl_wait();
            for (int i = blockIdx.x; i < p.items && ok; i += gridDim.x) {
                const Item t = item(i);
                for (int c = t.kb0; c < t.kb1 && ok; c += CHUNK_KB) {
                    // (in this order: the wait for the activations' slot goes ahead of that for the weights')
                    const int before = use - NT * S::X_SLOTS + NT - 1;
                    ok = before < 0 || mbar_wait(&done[before % S::SLOTS], (before / S::SLOTS) & 1, p.err, 62);
                    if (early > 0) --early; else ok = ok && load_w(c, t.n0, true);
                    if (ok) load_x(c, t.m0);
                    ++use;
                    if (NT == 2) {
                        if (early > 0) --early; else ok = ok && load_w(c, t.n0 + TILE_N, false);
                        ++use;
                    }
                }
            }
        } else {
            pdl_wait();
        }
    } else if (warp == 1) {
        // The whole warp walks along, one lane issues.  What an issue costs is what bounds this kernel, or nearly: a wait that
        // is already over takes about 100 cycles, a commit 160, eight MMAs 260 to issue and 768 to run; so there is one barrier
        // for what a use needs and one for its end.
        pdl_wait();
        constexpr uint32_t idesc = instr_desc(3 * BN);
        const uint64_t wdesc0 = smem_desc_sw128(smem_u32(smem_w)), xdesc0 = smem_desc_sw128(smem_u32(smem_x));
        Ring<S::SLOTS> wr;
        Ring<S::X_SLOTS> xr;
        Ring<2> ar;
        for (int i = blockIdx.x; i < p.items && ok; i += gridDim.x) {
            const Item t = item(i);
            for (int c = t.kb0; c < t.kb1 && ok; c += CHUNK_KB) {
#pragma unroll
                for (int half = 0; half < NT; ++half) {
                    ok = ok && mbar_wait(&empty_acc[ar.slot], ar.pass ^ 1, p.err, 63) && mbar_wait(&full[wr.slot], wr.pass, p.err, 64);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t acc = tmem_base + (uint32_t)(ar.slot * S::BUF_COLS);
                    const uint64_t wdesc = wdesc0 + (uint64_t)(wr.slot * (S::W_BYTES >> 4)), xdesc = xdesc0 + (uint64_t)(xr.slot * (S::X_BYTES >> 4));
                    if (elected()) {
#pragma unroll
                        for (int q = 0; q < CHUNK_KB; ++q)
#pragma unroll
                            for (int k = 0; k < BLOCK_K / UMMA_K; ++k)
                                umma_h16(acc, wdesc + (uint64_t)(q * (S::W_BYTES / CHUNK_KB >> 4) + 2 * k),
                                         xdesc + (uint64_t)(q * (S::X_BYTES / CHUNK_KB >> 4) + 2 * k), idesc, (q > 0 || k > 0) ? 1u : 0u);
                        umma_commit(&done[wr.slot]);
                    }
                    __syncwarp();
                    wr.next();
                    ar.next();
                }
                xr.next();
            }
        }
    } else {
        pdl_wait();
        const int group = (warp - 2) >> 2;
        const int tile = NT == 2 ? group : 0, col0 = NT == 2 ? 0 : group * S::TOKENS;       // its feature tile, its tokens
        const int quad = warp & 3;                       // the tensor-memory lanes it may read
        const uint32_t lanes = (uint32_t)(quad * 32) << 16;
        constexpr int T = S::TOKENS;
        Ring<S::SLOTS> wr;
        Ring<2> ar;
        if (tile) { wr.next(); ar.next(); }
        for (int i = blockIdx.x; i < p.items && ok; i += gridDim.x) {
            const Item t = item(i);
            const int n = t.n0 + tile * TILE_N + quad * 32 + lane, m0 = t.m0 + col0;
            const bool live = n < p.N;
            const float bias = live && p.bias && !p.parts ? __ldg(p.bias + n) : 0.f;
            float seg[T], tot[T];
#pragma unroll
            for (int j = 0; j < T; ++j) seg[j] = tot[j] = 0.f;
            int chunk = 0;                               // of the segment
            for (int c = t.kb0; c < t.kb1; c += CHUNK_KB) {
                ok = __all_sync(0xffffffffu, mbar_wait(&done[wr.slot], wr.pass, p.err, 66));
                if (!ok) break;
                tc_fence_after();
                const uint32_t acc = tmem_base + lanes + (uint32_t)(ar.slot * S::BUF_COLS + col0);
#pragma unroll
                for (int j0 = 0; j0 < T; j0 += 16) {
                    uint32_t h[32], m[32], l[32];        // (the loads fill the first 16)
                    float low[16];
                    tmem_ld16(acc + BN + j0, m);
                    tmem_ld16(acc + 2 * BN + j0, l);
                    tmem_ld_wait();
                    // the lower terms' part is kept finite, so that a first term that is not decides
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        low[j] = fminf(fmaxf(fmaf(__uint_as_float(l[j]), TERM, __uint_as_float(m[j])), -3.402823466e38f), 3.402823466e38f);
                    tmem_ld16(acc + j0, h);
                    tmem_ld_wait();
                    if (j0 + 16 == T) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&empty_acc[ar.slot])) : "memory");
                    }
#pragma unroll
                    for (int j = 0; j < 16; ++j) seg[j0 + j] += fmaf(low[j], TERM, __uint_as_float(h[j]));
                }
                if (++chunk == SEG_CHUNKS || c + CHUNK_KB >= t.kb1) {
                    if (p.parts) {
                        float* dst = p.parts + ((size_t)(c / (SEG_CHUNKS * CHUNK_KB)) * p.M + m0) * p.N + n;
                        if (live)
#pragma unroll
                            for (int j = 0; j < T; ++j)
                                if (m0 + j < p.M) __stcg(dst + (size_t)j * p.N, seg[j]);
                    }
#pragma unroll
                    for (int j = 0; j < T; ++j) { tot[j] += seg[j]; seg[j] = 0.f; }
                    chunk = 0;
                }
#pragma unroll
                for (int u = 0; u < NT; ++u) { wr.next(); ar.next(); }
            }
            const bool store = ok && !p.parts && live;
#pragma unroll
            for (int j0 = 0; j0 < T; j0 += 16) {
                if (!store) break;
                float res[16], un[16];                   // all loads ahead of the first store: the residual may be C itself
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int m = m0 + j0 + j;
                    res[j] = m < p.M && p.residual ? __ldcg(p.residual + (size_t)m * p.ldc + n) : 0.f;
#ifdef TNX_F16
                    un[j] = m < p.M ? __ldcg(p.unscale + m) : 0.f;
#else
                    un[j] = 1.f;
#endif
                }
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int m = m0 + j0 + j;
                    if (m >= p.M) break;
                    const float v = finish(tot[j0 + j], un[j], bias, p.act, res[j]);
                    const size_t o = (size_t)m * p.ldc + n;
                    if (p.c_is_h16) ((h16*)p.C)[o] = float_to_h16(v);
                    else ((float*)p.C)[o] = v;
                }
            }
            __syncwarp();
        }
    }
    if (!ok) {                           // a wait ran out: let the copies in flight land before the shared memory goes
        const unsigned long long t0 = global_ns();
        while (global_ns() - t0 < 1000000ull) __nanosleep(1000);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, S::TMEM_COLS);
    }
}

// The segments of a product whose K was split, added in their order.  A thread takes VEC neighbouring outputs.
template <int VEC>
__global__ void __launch_bounds__(128) split_sum_kernel(const Params p, int segs) {
    pdl_launch_dependents();
    const int per_row = p.N / VEC;
    const long long i = (long long)blockIdx.x * 128 + threadIdx.x;
    const int m = (int)(i / per_row), n = (int)(i - (long long)m * per_row) * VEC;
    float b[VEC];
#pragma unroll
    for (int e = 0; e < VEC; ++e) b[e] = m < p.M && p.bias ? __ldg(p.bias + n + e) : 0.f;
    pdl_wait();
    if (m >= p.M) return;
    float v[VEC], res[VEC];
#pragma unroll
    for (int e = 0; e < VEC; ++e) { v[e] = 0.f; res[e] = p.residual ? __ldcg(p.residual + (size_t)m * p.ldc + n + e) : 0.f; }
    const float* src = p.parts + (size_t)m * p.N + n;
    const size_t step = (size_t)p.M * p.N;
    for (int s0 = 0; s0 < segs; s0 += 4) {               // four round trips at a time
        float f[4][VEC];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int e = 0; e < VEC; ++e) f[u][e] = 0.f;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (s0 + u < segs) {
                if constexpr (VEC == 4) {
                    const float4 q = __ldcg((const float4*)(src + (s0 + u) * step));
                    f[u][0] = q.x; f[u][1] = q.y; f[u][2] = q.z; f[u][3] = q.w;
                } else {
                    f[u][0] = __ldcg(src + (s0 + u) * step);
                }
            }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (s0 + u < segs)
#pragma unroll
                for (int e = 0; e < VEC; ++e) v[e] += f[u][e];
    }
#ifdef TNX_F16
    const float un = __ldcg(p.unscale + m);
#else
    const float un = 1.f;
#endif
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
        const float x = finish(v[e], un, b[e], p.act, res[e]);
        const size_t o = (size_t)m * p.ldc + n + e;
        if (p.c_is_h16) ((h16*)p.C)[o] = float_to_h16(x);
        else ((float*)p.C)[o] = x;
    }
}

// The terms of the activations: planes [3][M][K].  A block a row; up to KEEP elements a thread stay in registers between
// the search for the row's largest and the split, the rest is read again.
constexpr int SPLIT_THREADS = 256;
__device__ __forceinline__ bool not_finite(float v) { return (__float_as_uint(v) & 0x7f800000u) == 0x7f800000u; }

// h, m, l of one element v; odd: its row holds an element that is not finite.
__device__ __forceinline__ void terms(float v, float scale, bool odd, h16& h, h16& m, h16& l) {
#ifdef TNX_F16
    const float x = v * scale;
    h = __float2half_rn(odd && !not_finite(x) ? fminf(fmaxf(x, -1.f), 1.f) : x);
    // no element but zero becomes zero: an infinite weight tells them apart
    if ((uint16_t)(__half_as_ushort(h) << 1) == 0 && v != 0.f) h = __ushort_as_half(v < 0.f ? 0x8001 : 0x0001);
    if (odd) {
        m = l = __float2half_rn(0.f);
        return;
    }
    const float r = (x - __half2float(h)) * 2048.f;
    m = __float2half_rn(r);
    l = __float2half_rn((r - __half2float(m)) * 2048.f);
#else
    const float x = v;
    const uint32_t u = __float_as_uint(x);
    if (not_finite(x)) {                 // infinities keep their sign; a NaN stays one when its low bits go
        h = __ushort_as_bfloat16((unsigned short)((u >> 16) | ((u & 0x7fffffu) ? 0x40u : 0u)));
        m = l = __ushort_as_bfloat16(0);
        return;
    }
    if ((u & 0x7fff0000u) == 0 && x != 0.f) {        // below 2^-133: rounded away from zero (an infinite weight times a small number)
        h = __ushort_as_bfloat16((unsigned short)((u >> 16) | 1u));
        m = l = __ushort_as_bfloat16(0);
        return;
    }
    const float hf = __uint_as_float(u & 0xffff0000u), r = x - hf;
    const float mf = __uint_as_float(__float_as_uint(r) & 0xffff0000u);
    h = __ushort_as_bfloat16((unsigned short)(u >> 16));
    m = __ushort_as_bfloat16((unsigned short)(__float_as_uint(r) >> 16));
    l = __ushort_as_bfloat16((unsigned short)(__float_as_uint(r - mf) >> 16));
#endif
}

template <bool VECTOR>
__global__ void __launch_bounds__(SPLIT_THREADS)
split_terms_kernel(const float* __restrict__ A, h16* __restrict__ planes, float* __restrict__ unscale, int M, int K, int lda) {
    constexpr int KEEP = 4;              // pieces of four
    pdl_launch_dependents();
    pdl_wait();
    const int row = blockIdx.x, quads = K / 4, tid = threadIdx.x;
    const float* src = A + (size_t)row * lda;
    auto load = [&](int q) {
        if (VECTOR) return __ldg((const float4*)src + q);
        return make_float4(src[4 * q], src[4 * q + 1], src[4 * q + 2], src[4 * q + 3]);
    };
    float4 keep[KEEP];
#pragma unroll
    for (int i = 0; i < KEEP; ++i) {
        const int q = tid + i * SPLIT_THREADS;
        keep[i] = q < quads ? load(q) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float scale = 1.f;
    bool odd = false;
#ifdef TNX_F16
    // the row's largest as bits: a number's bits grow with its size, and those of infinities and NaN are above all others
    uint32_t top = 0;
    auto see = [&](float4 v) {
        top = max(max(top, __float_as_uint(v.x) & 0x7fffffffu), __float_as_uint(v.y) & 0x7fffffffu);
        top = max(max(top, __float_as_uint(v.z) & 0x7fffffffu), __float_as_uint(v.w) & 0x7fffffffu);
    };
#pragma unroll
    for (int i = 0; i < KEEP; ++i) see(keep[i]);
    for (int q = tid + KEEP * SPLIT_THREADS; q < quads; q += SPLIT_THREADS) see(load(q));
    __shared__ uint32_t tops[SPLIT_THREADS / 32];
    top = __reduce_max_sync(0xffffffffu, top);
    if ((tid & 31) == 0) tops[tid >> 5] = top;
    __syncthreads();
    top = 0;
#pragma unroll
    for (int w = 0; w < SPLIT_THREADS / 32; ++w) top = max(top, tops[w]);
    odd = top >= 0x7f800000u;
    // 2^(14 - exponent of the largest), at most 2^126 (its reciprocal is then a normal number too)
    const int e = odd ? 0 : min(141 - (int)(top >> 23), 126);
    scale = __uint_as_float((uint32_t)(e + 127) << 23);
    if (tid == 0) unscale[row] = __uint_as_float((uint32_t)(127 - e) << 23);
#endif
    const size_t plane = (size_t)M * K;
    auto put = [&](int q, float4 v) {
        const float x[4] = {v.x, v.y, v.z, v.w};
        __align__(8) h16 h[4], m[4], l[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) terms(x[i], scale, odd, h[i], m[i], l[i]);
        h16* dst = planes + (size_t)row * K + 4 * (size_t)q;
        *(uint2*)dst = *(const uint2*)h;
        *(uint2*)(dst + plane) = *(const uint2*)m;
        *(uint2*)(dst + 2 * plane) = *(const uint2*)l;
    };
#pragma unroll
    for (int i = 0; i < KEEP; ++i) {
        const int q = tid + i * SPLIT_THREADS;
        if (q < quads) put(q, keep[i]);
    }
    for (int q = tid + KEEP * SPLIT_THREADS; q < quads; q += SPLIT_THREADS) put(q, load(q));
}

template <int BN, int NT>
int launch_product(const CUtensorMap& mw, const CUtensorMap& mx, const Params& p, int sms, cudaStream_t stream) {
    using S = Shape<BN, NT>;
    static TnxSmemLimit limit;
    if (const int rc = limit.allow(gemm_split_kernel<BN, NT>, S::SMEM)) return rc;
    const int grid = p.items < sms ? p.items : sms;
    return tnx_launch_ex(1, gemm_split_kernel<BN, NT>, dim3(grid), dim3(S::THREADS), S::SMEM, stream, mw, mx, p);
}

// The planes of the terms, [3][M][K], in boxes of 3 x bn x 64: a K block of a tile's three terms, one under the other.
bool make_terms_map(CUtensorMap* out, const void* planes, int M, int K, int bn) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)M, 3}, strides[2] = {(cuuint64_t)K * 2, (cuuint64_t)K * 2 * M};
    const cuuint32_t box[3] = {64u, (cuuint32_t)bn, 3u}, estr[3] = {1, 1, 1};
    return fn(out, TNX_TMA_H16, 3, const_cast<void*>(planes), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct Plan { int bn, nt, splits, segs, segs_per_split; };

// Tokens a tile: as few as hold all rows, 64 at most.  Two feature tiles a CTA where that leaves the SMs as busy (the
// staged activations then serve twice the features).  K is split, by whole segments, while that fills more SMs.
Plan plan_for(int M, int N, int K, int sms) {
    Plan q;
    q.bn = M <= 16 ? 16 : M <= 32 ? 32 : 64;
    q.segs = (K + SEG_K - 1) / SEG_K;
    const long long tm = (M + q.bn - 1) / q.bn;
    const long long t1 = tm * ((N + TILE_N - 1) / TILE_N), t2 = tm * ((N + 2 * TILE_N - 1) / (2 * TILE_N));
    const long long r1 = (t1 + sms - 1) / sms, r2 = (t2 + sms - 1) / sms;
    q.nt = q.bn == 64 && 3 * r2 <= 2 * r1 ? 2 : 1;
    q.splits = 1;
    q.segs_per_split = q.segs;
    if (q.nt == 1 && 2 * t1 <= sms && q.segs > 1) {
        long long s = sms / t1;
        if (s > q.segs) s = q.segs;
        q.segs_per_split = (int)((q.segs + s - 1) / s);
        q.splits = (q.segs + q.segs_per_split - 1) / q.segs_per_split;
    }
    return q;
}

}  // namespace

// Scratch memory that tnx_gemm_split needs for these sizes, in bytes: the terms, the rows' scales, the segments' sums.
TNX_EXPORT long long tnx_gemm_split_scratch(int M, int N, int K, int sms) {
    if (M <= 0 || N <= 0 || K <= 0 || sms <= 0) return 0;
    const Plan q = plan_for(M, N, K, sms);
    const long long planes = (3ll * M * K * 2 + 255) / 256 * 256, scales = (4ll * M + 255) / 256 * 256;
    return planes + scales + (q.splits > 1 ? 4ll * q.segs * M * N : 0);
}

// A [M, lda] float, W [N, ldw] h16 with ldw and K multiples of 8 and a 16-byte aligned base; scratch: 256-byte aligned,
// tnx_gemm_split_scratch bytes.  residual (32-bit, C's leading dimension) may alias C when C is float.  Returns the number
// of kernels launched, or an error: negative, or a CUDA error code + 1000.
TNX_EXPORT int tnx_gemm_split(const float* A, const void* W, const float* bias, const float* residual, void* C, int M, int N,
                              int K, int lda, int ldw, int ldc, int act, int c_h16, int sms, void* scratch, int* err_word,
                              cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || lda < K || ldw < K || ldc < N || sms <= 0 || !scratch || !err_word) return TNX_ERR_BAD_ARG;
    if (residual && c_h16) return TNX_ERR_BAD_ARG;
    if (act < 0 || act >= TNX_ACT_COUNT) return TNX_ERR_BAD_ARG;
    if (K % 8 || ldw % 8 || ((uintptr_t)W & 15) || ((uintptr_t)scratch & 255) || 3ll * M >= (1ll << 31)) return TNX_ERR_UNSUPPORTED;
    const Plan q = plan_for(M, N, K, sms);
    const size_t planes_bytes = (3ull * M * K * 2 + 255) / 256 * 256, scales_bytes = (4ull * M + 255) / 256 * 256;
    h16* planes = (h16*)scratch;
    float* scales = (float*)((char*)scratch + planes_bytes);
    Params p{};
    p.M = M; p.N = N; p.K = K; p.ldc = ldc; p.act = act; p.c_is_h16 = c_h16;
    p.tiles_m = (M + q.bn - 1) / q.bn;
    const long long items = (long long)p.tiles_m * ((N + q.nt * TILE_N - 1) / (q.nt * TILE_N)) * q.splits;
    if (items >= (1ll << 31)) return TNX_ERR_UNSUPPORTED;
    p.items = (int)items; p.splits = q.splits; p.segs_per_split = q.segs_per_split;
    p.bias = bias; p.residual = residual; p.unscale = scales; p.C = C; p.err = err_word;
    p.parts = q.splits > 1 ? (float*)((char*)scales + scales_bytes) : nullptr;
    CUtensorMap mw, mx;
    if (!make_map(&mw, W, N, K, ldw, TILE_N) || !make_terms_map(&mx, planes, M, K, q.bn)) return TNX_ERR_UNSUPPORTED;
    const bool vec = lda % 4 == 0 && ((uintptr_t)A & 15) == 0;
    int rc = vec ? tnx_launch_in_order(split_terms_kernel<true>, dim3(M), dim3(SPLIT_THREADS), 0, stream, A, planes, scales, M, K, lda)
                 : tnx_launch_in_order(split_terms_kernel<false>, dim3(M), dim3(SPLIT_THREADS), 0, stream, A, planes, scales, M, K, lda);
    if (rc) return rc > 0 ? 1000 + rc : rc;
    if (q.bn == 16) rc = launch_product<16, 1>(mw, mx, p, sms, stream);
    else if (q.bn == 32) rc = launch_product<32, 1>(mw, mx, p, sms, stream);
    else if (q.nt == 1) rc = launch_product<64, 1>(mw, mx, p, sms, stream);
    else rc = launch_product<64, 2>(mw, mx, p, sms, stream);
    if (rc) return rc > 0 ? 1000 + rc : rc;
    if (q.splits == 1) return 2;
    const int vec4 = N % 4 == 0;
    const long long work = (long long)M * (vec4 ? N / 4 : N);
    const dim3 grid((unsigned)((work + 127) / 128));
    rc = vec4 ? tnx_launch_ex(1, split_sum_kernel<4>, grid, dim3(128), 0, stream, p, q.segs)
              : tnx_launch_ex(1, split_sum_kernel<1>, grid, dim3(128), 0, stream, p, q.segs);
    if (rc) return rc > 0 ? 1000 + rc : rc;
    return 3;
}
