// Decode attention on the tensor cores (mma.sync), above all where several query heads share a key/value head: one query token per request, the keys and values of
// its request streamed from the pages named by its block table.
//
//   s_j = scale * <q, k_j>  (32-bit; less a distance bias where one is given),  out = sum_j exp(s_j - max) v_j / sum_j exp(s_j - max)
//   (with a sink, exp(sink - max) more in the denominator: the first warp of the first split starts from it)
//
// Bound by the pages' bytes.  With one block per query head (attention_decode.cu) the heads of a group each read the
// group's pages, and with all of a group's dot products in one block on the multiply-add units that arithmetic is what a
// block waits for.  Here a block takes up to 16 query heads of a key/value head, reads every page once, and a page of 16
// keys costs a warp D/16 products for the scores and two or three times as many for the values.
//   scores   S^T [16 keys x 8 heads] = K Q^T: the keys are the 16-row operand.  A contraction may take its dims in any
//            order, so a lane's 16-byte pieces of its two key rows ARE its operand registers (no shared memory).
//   softmax  a lane holds two keys of two heads; the maximum runs over eight lanes
//   values   O^T [16 dims x 8 heads] += V^T P^T: a lane's 16-byte pieces of four value rows, two rows' halves merged by a
//            byte permutation, are the 16-row operand; P is turned by movmatrix.
// A page's probabilities are formed against the page's own largest score, and its products, which start from zero, are added
// to the running sums times exp(page's maximum - running maximum) by ordinary 32-bit multiply-adds: the tensor cores cut the
// sums they form where those round, a bias that adds up along a chain of pages.  (The scores likewise, two 16-dim steps at a
// time.)  A probability enters the products as a sum of 16-bit numbers cut towards zero and a rounded last one: three in bfloat16,
// to within 2^-22 of itself, and two in float16, to within 2^-21 of itself down to 2^-18 of its page's largest and to 2^-39 of
// the page's largest below (in multiples of 2^-15, which takes float16's smallest number to 2^-39); the denominator sums it in
// 32-bit.  No term is zero or less: an infinite value stays infinite (infinity x 0 has no value).  Results rounded otherwise
// than the 64-bit ones are, of float16 results, 48 rows of 32 heads on 8: 1.3 in 1,000 (a block a head: 1.8; with sums chained
// through the accumulators and unscaled terms 4.6).
// Measured, pages beyond the second-level cache, us a call in float16 / bfloat16 (with one block a head): 48 rows of 32 heads on
// 8 over 950 to 1,900 tokens 60 / 63 (165 / 171; 45 would be the copy rate), 64 rows over 1,024 to 2,048 77 / 80 (215 / 227), 8
// rows of 32 heads on 2 over 950 to 1,900 14.5 / 16.5 (39 / 41); 64 rows of 16 heads on one over 500 to 1,000 18.6 / 19.4 (65 / 68).
// With as many key/value heads as heads: 80 dims, 8 rows of 32 heads over 700 to 1,400 29 / 31 (33 / 35).
//
// Grid (key/value heads x head tiles, rows, splits), 4, 8 or 12 warps; a warp takes every WARPS-th page of the split's range,
// its next keys and values in flight while it works.  Warps are merged in shared memory.  The splits of a (row, head tile)
// are a thread-block cluster: each block reads the others' merged states from their shared memory and writes its share of
// the output (through scratch memory and a counter two splits cost 10 us).  The kernel can append the rows' own keys and
// values, as attention_decode.cu does.
#include "common.cuh"

namespace {

constexpr int PAGE = 16;

struct GroupedParams {
    const h16* q; int q_stride;
    const h16* cache;
    const int* block_tables; int bt_stride;
    const int* rows;                 // rows of the batch that are decode tokens (null: all rows)
    const int* token_request;
    const int* positions;
    h16* out; int out_stride;
    int n_heads, n_kv_heads, head_tiles;
    int window;                      // the mask rule of common.cuh: first_visible_key
    float scale;
    int keep_first;                  // with a window: the first positions that stay visible
    DistanceBias bias;
    SoftmaxSink sink;
    int n_splits, pages_per_split;   // a cluster's blocks
    const h16* k_new;                // [rows, kv_heads * D] keys of the rows' own tokens, or null: the cache holds them
    const h16* v_new;
    int kv_stride;
    h16* cache_w;
};

#ifdef TNX_F16
#define MMA_KIND "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 "
#else
#define MMA_KIND "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
#endif
__device__ __forceinline__ void mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm(MMA_KIND "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_from_zero(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm(MMA_KIND "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
#undef MMA_KIND
// An 8 x 8 matrix of 16-bit numbers turned: lane (g, c) gives row g, columns 2c and 2c + 1, and receives those of the transpose.
__device__ __forceinline__ uint32_t turned(uint32_t v) {
    uint32_t r;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}

// Two numbers cut to 16 bits: towards zero, so that what is left has no other sign.
__device__ __forceinline__ h16x2 cut(float a, float b) {
    uint32_t v;
#ifdef TNX_F16
    asm("cvt.rz.f16x2.f32 %0, %1, %2;" : "=r"(v) : "f"(b), "f"(a));
#else
    asm("cvt.rz.bf16x2.f32 %0, %1, %2;" : "=r"(v) : "f"(b), "f"(a));
#endif
    return *(const h16x2*)&v;
}

#ifdef TNX_F16
constexpr int TERMS = 2;
constexpr float SCALE = 0x1p15f;             // of the probabilities in the products: float16 has no small numbers to spare
constexpr float LEAST = 0x1p-24f;            // the smallest positive number of the 16-bit type
#else
constexpr int TERMS = 3;
constexpr float SCALE = 1.f;
constexpr float LEAST = 0x1p-133f;
#endif

__device__ __forceinline__ uint32_t shared_address(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ float remote_float(const float* local, int rank) {       // the same place in another block's shared memory
    uint32_t at;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(shared_address(local)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at));
    return v;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// NT: tiles of eight query heads (1 or 2) that the block's heads fill.  An SM's registers hold twelve warps of the first
// kind and eight of the second.
template <int D, int NT, int WARPS, bool BIAS>
__global__ void __launch_bounds__(WARPS * 32, (NT == 1 ? 12 : 8) / WARPS)
attention_decode_grouped_kernel(const GroupedParams p) {
    constexpr int STEPS = D / 16;                       // 16-dim steps of the scores' contraction, 16-dim tiles of the output
    constexpr int N32 = D / 32, N64 = D / 64, REST = (D % 64) / 16;
    constexpr int HEADS = 8 * NT;
    constexpr int PITCH = D + 4;
    __shared__ float sm_m[WARPS][HEADS], sm_l[WARPS][HEADS], block_m[HEADS], block_l[HEADS];
    extern __shared__ __align__(16) float sm_o[];       // [WARPS][HEADS][PITCH]
    pdl_launch_dependents();
    pdl_wait();

    const int kvh = blockIdx.x / p.head_tiles, tile = blockIdx.x % p.head_tiles, ri = blockIdx.y, split = blockIdx.z;
    const int group = p.n_heads / p.n_kv_heads;
    const int h0 = kvh * group + tile * HEADS, n_mine = min(HEADS, group - tile * HEADS);     // the block's query heads
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
    const int row = p.rows ? p.rows[ri] : ri;
    if (row < 0) return;                                        // a padded entry of the row list of a captured step
    const int req = p.token_request[row];
    if (req < 0) return;                                        // a padded row of a captured batch
    const int pos = p.positions[row];
    const int* bt = p.block_tables + (size_t)req * p.bt_stride;

    // the queries as the 8-column operand: lane (g, c) holds head g's dims in the order its key pieces come in, kept where the
    // warp's results go in the end (in registers they spilled others: 88 us for the first measurement above)
    uint2* const qs = (uint2*)(sm_o + (size_t)warp * HEADS * PITCH) + lane;
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        const bool has = t * 8 + g < n_mine;
        const h16* src = p.q + (size_t)row * p.q_stride + (size_t)(h0 + t * 8 + g) * D;
#pragma unroll
        for (int i = 0; i < N32; ++i) {
            const uint4 v = has ? *(const uint4*)(src + 32 * i + 8 * c) : make_uint4(0, 0, 0, 0);
            qs[(t * STEPS + 2 * i) * 32] = make_uint2(v.x, v.y); qs[(t * STEPS + 2 * i + 1) * 32] = make_uint2(v.z, v.w);
        }
        if constexpr (D % 32 != 0) {
            const uint2 v = has ? *(const uint2*)(src + 32 * N32 + 4 * c) : make_uint2(0, 0);
            qs[(t * STEPS + STEPS - 1) * 32] = v;
        }
    }

    const int kv_len = pos + 1;
    const int first_key = first_visible_key(pos, p.window);
    const int n_pages = (kv_len + PAGE - 1) / PAGE;
    const BlockWalk walk = walk_blocks(first_key, p.keep_first, PAGE);       // pages are numbered along the visible ones
    const int page_lo = split * p.pages_per_split;
    const int page_hi = min(walk.count(n_pages - 1), (split + 1) * p.pages_per_split);
    const size_t head_block = (size_t)PAGE * D;
    const bool own_here = p.k_new != nullptr && walk.place(pos / PAGE) / p.pages_per_split == split;    // one answer for the block
    const int cached_len = p.k_new != nullptr ? pos : kv_len;
    const int my_pages = page_hi > page_lo + warp ? (page_hi - page_lo - warp + WARPS - 1) / WARPS : 0;
    const int n_chunks = my_pages + (own_here && warp == 0 ? 1 : 0);         // the token's own key is a chunk of one key

    float m[NT][2], l[NT][2], acc[NT][STEPS][4];                             // of heads 2c and 2c + 1 of each tile
    float bias_mul[NT][2], bias_rate[NT][2];                                 // of a logarithm to base 2
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        const bool sink_here = p.sink.on && split == 0 && warp == 0;
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            m[t][x] = sink_here ? p.sink.score : -INFINITY;
            l[t][x] = sink_here && g == 0 ? 1.f : 0.f;                       // counted once: the sum runs over the lanes of a head
            if constexpr (BIAS) {
                const int h = h0 + min(t * 8 + 2 * c + x, n_mine - 1);
                bias_mul[t][x] = p.bias.mul[h] * 0.6931471805599453f; bias_rate[t][x] = p.bias.rate[h];
            }
        }
#pragma unroll
        for (int s = 0; s < STEPS; ++s)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[t][s][i] = 0.f;
    }

    auto seen = [&](int j) { return (j >= first_key || j < p.keep_first) && j < cached_len; };
    // chunk t of the warp: its first key and its key and value rows
    auto first_of = [&](int t) { return t < my_pages ? walk.at(page_lo + warp + t * WARPS) * PAGE : pos; };
    auto page_of = [&](int t) { return t < my_pages ? bt[walk.at(page_lo + warp + t * WARPS)] : 0; };
    auto rows_of = [&](int t, int page, int which) -> const h16* {
        if (t < my_pages) return p.cache + (((size_t)page * 2 + which) * p.n_kv_heads + kvh) * head_block;
        return (which ? p.v_new : p.k_new) + (size_t)row * p.kv_stride + (size_t)kvh * D;
    };
    uint32_t kr[2][2 * STEPS], vr[4][STEPS];                                 // two key rows, four value rows
    auto load_keys = [&](int t, int page) {
        const h16* base = rows_of(t, page, 0);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int key = g + 8 * r;
            const bool there = t < my_pages || key == 0;
            const h16* src = base + (size_t)key * D;
#pragma unroll
            for (int i = 0; i < N32; ++i) {
                const uint4 v = there ? __ldg((const uint4*)(src + 32 * i + 8 * c)) : make_uint4(0, 0, 0, 0);
                kr[r][4 * i] = v.x; kr[r][4 * i + 1] = v.y; kr[r][4 * i + 2] = v.z; kr[r][4 * i + 3] = v.w;
            }
            if constexpr (D % 32 != 0) {
                const uint2 v = there ? __ldg((const uint2*)(src + 32 * N32 + 4 * c)) : make_uint2(0, 0);
                kr[r][4 * N32] = v.x; kr[r][4 * N32 + 1] = v.y;
            }
        }
    };
    // rows that no query may see, and rows never written, which may hold anything, stay zero: p = 0 times them is 0
    auto load_values = [&](int t, int page) {
        const h16* base = rows_of(t, page, 1);
        const int j0 = first_of(t);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int key = 2 * c + (r & 1) + 8 * (r >> 1);
            const bool there = t < my_pages ? seen(j0 + key) : key == 0;
            const h16* src = base + (size_t)key * D;
#pragma unroll
            for (int i = 0; i < N64; ++i) {
                const uint4 v = there ? __ldg((const uint4*)(src + 64 * i + 8 * g)) : make_uint4(0, 0, 0, 0);
                vr[r][4 * i] = v.x; vr[r][4 * i + 1] = v.y; vr[r][4 * i + 2] = v.z; vr[r][4 * i + 3] = v.w;
            }
            if constexpr (REST == 1) {
                vr[r][4 * N64] = there ? __ldg((const uint32_t*)(src + 64 * N64 + 2 * g)) : 0u;
            } else if constexpr (REST == 2) {
                const uint2 v = there ? __ldg((const uint2*)(src + 64 * N64 + 4 * g)) : make_uint2(0, 0);
                vr[r][4 * N64] = v.x; vr[r][4 * N64 + 1] = v.y;
            } else if constexpr (REST == 3) {
#pragma unroll
                for (int w = 0; w < 3; ++w) vr[r][4 * N64 + w] = there ? __ldg((const uint32_t*)(src + 64 * N64 + 6 * g) + w) : 0u;
            }
        }
    };

    int page = 0, next_page = 0;
    if (n_chunks > 0) {
        page = page_of(0);
        load_keys(0, page);
        load_values(0, page);
        next_page = page_of(1);
    }
    for (int t = 0; t < n_chunks; ++t) {
        const bool more = t + 1 < n_chunks;
        float s[NT][4];                                  // [0], [1]: key g of heads 2c, 2c + 1;  [2], [3]: key g + 8
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            float x[4];
#pragma unroll
            for (int k = 0; k < STEPS; ++k) {
                const uint2 q = qs[(n * STEPS + k) * 32];
                if (k % 2 == 0) mma_from_zero(x, kr[0][2 * k], kr[1][2 * k], kr[0][2 * k + 1], kr[1][2 * k + 1], q.x, q.y);
                else mma(x, kr[0][2 * k], kr[1][2 * k], kr[0][2 * k + 1], kr[1][2 * k + 1], q.x, q.y);
                if (k % 2 == 0 && k + 1 < STEPS) continue;
#pragma unroll
                for (int i = 0; i < 4; ++i) s[n][i] = k >= 2 ? s[n][i] + x[i] : x[i];
            }
        }
        if (more) load_keys(t + 1, next_page);
        const int j0 = first_of(t);
        const bool paged = t < my_pages;
        const bool see0 = paged ? seen(j0 + g) : g == 0, see1 = paged && seen(j0 + g + 8);
        float here[NT][2], top[NT][2];                   // the page's largest score, the largest so far
        bool grew = false;
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                float a = s[n][x] * p.scale, b = s[n][2 + x] * p.scale;
                if constexpr (BIAS) {
                    a -= bias_mul[n][x] * log2_approx(fmaf(bias_rate[n][x], (float)(pos - j0 - g), 1.f));
                    b -= bias_mul[n][x] * log2_approx(fmaf(bias_rate[n][x], (float)(pos - j0 - g - 8), 1.f));
                }
                s[n][x] = a = see0 ? a : -INFINITY;
                s[n][2 + x] = b = see1 ? b : -INFINITY;
                float v = fmaxf(a, b);
                v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 4));
                v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 8));
                v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 16));
                here[n][x] = v;
                top[n][x] = fmaxf(v, m[n][x]);
                grew = grew || top[n][x] > m[n][x];
            }
        if (__any_sync(0xffffffffu, grew)) {
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const float corr = m[n][x] == -INFINITY ? 0.f : __expf(m[n][x] - top[n][x]);
                    m[n][x] = top[n][x];
                    l[n][x] *= corr;
#pragma unroll
                    for (int k = 0; k < STEPS; ++k) { acc[n][k][x] *= corr; acc[n][k][2 + x] *= corr; }
                }
        }
        // the probabilities against the page's maximum, split into 16-bit terms and turned: lane (g, c) gets head g's keys
        // 2c, 2c + 1 (and + 8).  times: the page's share of the sums
        uint32_t pt[NT][TERMS][2];
        float times[NT][2];
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            float e[4];
#pragma unroll
            for (int x = 0; x < 2; ++x) times[n][x] = here[n][x] == -INFINITY ? 0.f : __expf(here[n][x] - m[n][x]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                e[i] = s[n][i] == -INFINITY ? 0.f : __expf(s[n][i] - here[n][i & 1]);
                l[n][i & 1] = fmaf(e[i], times[n][i & 1], l[n][i & 1]);
                e[i] *= SCALE;
            }
#pragma unroll
            for (int k = 0; k < TERMS; ++k)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    float &a = e[2 * r], &b = e[2 * r + 1];
                    const float ta = fmaxf(a, LEAST), tb = fmaxf(b, LEAST);
                    const h16x2 term = k + 1 < TERMS ? cut(ta, tb) : floats_to_h16x2(ta, tb);
                    if (k + 1 < TERMS) { const float2 f = h16x2_to_float2(term); a -= f.x; b -= f.y; }
                    pt[n][k][r] = turned(*(const uint32_t*)&term);
                }
        }
#pragma unroll
        for (int k = 0; k < STEPS; ++k) {
            const uint32_t a0 = __byte_perm(vr[0][k], vr[1][k], 0x5410), a1 = __byte_perm(vr[0][k], vr[1][k], 0x7632);
            const uint32_t a2 = __byte_perm(vr[2][k], vr[3][k], 0x5410), a3 = __byte_perm(vr[2][k], vr[3][k], 0x7632);
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                float x[4];                              // small terms first
                mma_from_zero(x, a0, a1, a2, a3, pt[n][TERMS - 1][0], pt[n][TERMS - 1][1]);
#pragma unroll
                for (int y = TERMS - 2; y >= 0; --y) mma(x, a0, a1, a2, a3, pt[n][y][0], pt[n][y][1]);
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[n][k][i] = fmaf(x[i], times[n][i & 1], acc[n][k][i]);
            }
        }
        if (more) {
            load_values(t + 1, next_page);
            next_page = t + 2 < n_chunks ? page_of(t + 2) : 0;
        }
    }
    if (own_here && tile == 0) {
        // The token's own key and value go into their page for later steps; after the pages have been streamed, so that
        // these loads do not stand between the block's start and its first page.
        const int where = bt[pos / PAGE];
        constexpr int PIECES = D / 8;
        for (int i = threadIdx.x; i < 2 * PIECES; i += WARPS * 32) {
            const int which = i / PIECES, piece = i % PIECES;
            const h16* src = (which ? p.v_new : p.k_new) + (size_t)row * p.kv_stride + (size_t)kvh * D;
            h16* dst = p.cache_w + (((size_t)where * 2 + which) * p.n_kv_heads + kvh) * head_block + (size_t)(pos % PAGE) * D;
            ((uint4*)dst)[piece] = ((const uint4*)src)[piece];
        }
    }
    __syncwarp();
    // the warps' states into shared memory: tile k of the output holds dims d_k (rows g) and d_k + 1 (rows g + 8)
#pragma unroll
    for (int n = 0; n < NT; ++n) {
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            float v = l[n][x];
            v += __shfl_xor_sync(0xffffffffu, v, 4);
            v += __shfl_xor_sync(0xffffffffu, v, 8);
            v += __shfl_xor_sync(0xffffffffu, v, 16);
            if (g == 0) { sm_m[warp][n * 8 + 2 * c + x] = m[n][x]; sm_l[warp][n * 8 + 2 * c + x] = v; }
#pragma unroll
            for (int k = 0; k < STEPS; ++k) {
                const int dim = k < 4 * N64 ? 64 * (k / 4) + 8 * g + 2 * (k % 4) : 64 * N64 + 2 * REST * g + 2 * (k - 4 * N64);
                *(float2*)&sm_o[(warp * HEADS + n * 8 + 2 * c + x) * PITCH + dim] = make_float2(acc[n][k][x], acc[n][k][2 + x]);
            }
        }
    }
    __syncthreads();
    // one factor per warp and head, then every output element is a sum over the warps
    const int tid = threadIdx.x;
    if (tid < HEADS) {
        float M = -INFINITY, L = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) M = fmaxf(M, sm_m[w][tid]);
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            const float f = sm_m[w][tid] == -INFINITY ? 0.f : __expf(sm_m[w][tid] - M);
            L += sm_l[w][tid] * f;
            sm_m[w][tid] = f;
        }
        block_m[tid] = M; block_l[tid] = L;
    }
    __syncthreads();
    for (int i = tid; i < n_mine * D; i += WARPS * 32) {
        const int x = i / D, dim = i % D;
        float o = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            const float f = sm_m[w][x];
            o += f == 0.f ? 0.f : sm_o[(w * HEADS + x) * PITCH + dim] * f;
        }
        if (p.n_splits == 1) {
            p.out[(size_t)row * p.out_stride + (size_t)(h0 + x) * D + dim] = float_to_h16(o * (1.f / SCALE) / block_l[x]);
        } else {
            sm_o[x * PITCH + dim] = o;                   // only this thread reads the warps' numbers of this place
        }
    }
    if (p.n_splits == 1) return;
    cluster_arrive();                                    // every block's merged state is there ...
    cluster_wait();
    for (int i = split * WARPS * 32 + tid; i < n_mine * D; i += p.n_splits * WARPS * 32) {
        const int x = i / D, dim = i % D;
        float ms[8], ls[8], os[8], M = -INFINITY, L = 0.f, o = 0.f;
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            const bool there = s < p.n_splits;
            ms[s] = there ? remote_float(&block_m[x], s) : -INFINITY;
            ls[s] = there ? remote_float(&block_l[x], s) : 0.f;
            os[s] = there ? remote_float(&sm_o[x * PITCH + dim], s) : 0.f;
        }
#pragma unroll
        for (int s = 0; s < 8; ++s) M = fmaxf(M, ms[s]);
#pragma unroll
        for (int s = 0; s < 8; ++s)
            if (ms[s] != -INFINITY) { const float f = __expf(ms[s] - M); L += ls[s] * f; o += os[s] * f; }
        p.out[(size_t)row * p.out_stride + (size_t)(h0 + x) * D + dim] = float_to_h16(o * (1.f / SCALE) / L);
    }
    cluster_arrive();                                    // ... and stays until all have read it
    cluster_wait();
}

template <int D, int NT, int WARPS, bool BIAS>
int launch_as(dim3 grid, cudaStream_t stream, const GroupedParams& p) {
    const size_t smem = sizeof(float) * WARPS * 8 * NT * (D + 4);
    auto kernel = attention_decode_grouped_kernel<D, NT, WARPS, BIAS>;
    if (smem > 40 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) { cudaGetLastError(); return (int)e; }
    }
    if (p.n_splits == 1) return tnx_launch_in_order(kernel, grid, dim3(WARPS * 32), smem, stream, p);
    return tnx_launch_cluster(0, dim3(1, 1, p.n_splits), kernel, grid, dim3(WARPS * 32), smem, stream, p);
}
template <int D, int NT>
int launch(int warps, dim3 grid, cudaStream_t stream, const GroupedParams& p) {
    constexpr int MOST = NT == 1 ? 12 : 8;
    if (warps == 4) return p.bias.mul ? launch_as<D, NT, 4, true>(grid, stream, p) : launch_as<D, NT, 4, false>(grid, stream, p);
    if (warps == MOST) return p.bias.mul ? launch_as<D, NT, MOST, true>(grid, stream, p) : launch_as<D, NT, MOST, false>(grid, stream, p);
    return TNX_ERR_BAD_ARG;
}
template <int D>
int launch_tiles(int nt, int warps, dim3 grid, cudaStream_t stream, const GroupedParams& p) {
    return nt == 1 ? launch<D, 1>(warps, grid, stream, p) : launch<D, 2>(warps, grid, stream, p);
}

// Query heads a block takes (8 or 16), 0 where the kernel does not take these sizes.
int heads_of_a_block(int n_heads, int n_kv_heads, int head_dim) {
    if (n_heads <= 0 || n_kv_heads <= 0 || n_heads % n_kv_heads) return 0;
    if (head_dim != 64 && head_dim != 80 && head_dim != 96 && head_dim != 112 && head_dim != 128) return 0;
    return n_heads / n_kv_heads <= 8 ? 8 : 16;
}

}  // namespace

// Arguments as tnx_attention_decode_append; n_splits 1 .. 8; warps a block: 4, or all that an SM holds (12 with up to 8 query
// heads a key/value head, else 8).
TNX_EXPORT int tnx_attention_decode_grouped(const void* q, int q_stride, void* cache, const int* block_tables, int bt_stride,
                                            const int* rows, const int* token_request, const int* positions, void* out,
                                            int out_stride, int n_rows, int n_heads, int n_kv_heads, int head_dim,
                                            int page_size, int window, float scale, int n_splits, int pages_per_split,
                                            const void* k_new, const void* v_new, int kv_stride, int warps, int keep_first, const float* bias_mul, const float* bias_rate,
                                            int has_sink, float sink_score, cudaStream_t stream) {
    if (n_rows <= 0) return 0;
    const int heads = heads_of_a_block(n_heads, n_kv_heads, head_dim);
    if (!heads || page_size != PAGE || q_stride % 8 || ((uintptr_t)q & 15) || ((uintptr_t)cache & 15)) return TNX_ERR_UNSUPPORTED;
    if ((k_new == nullptr) != (v_new == nullptr)) return TNX_ERR_BAD_ARG;
    if (k_new && (kv_stride % 8 || (((uintptr_t)k_new | (uintptr_t)v_new) & 15))) return TNX_ERR_UNSUPPORTED;
    if (n_splits < 1 || n_splits > 8 || pages_per_split < 1 || n_rows > 65535) return TNX_ERR_BAD_ARG;
    if (keep_first < 0 || (bias_mul && !bias_rate)) return TNX_ERR_BAD_ARG;
    GroupedParams p;
    p.keep_first = keep_first; p.bias.mul = bias_mul; p.bias.rate = bias_rate;
    p.sink.on = has_sink; p.sink.score = sink_score;
    p.q = (const h16*)q; p.q_stride = q_stride; p.cache = (const h16*)cache;
    p.block_tables = block_tables; p.bt_stride = bt_stride; p.rows = rows; p.token_request = token_request;
    p.positions = positions; p.out = (h16*)out; p.out_stride = out_stride;
    p.n_heads = n_heads; p.n_kv_heads = n_kv_heads; p.head_tiles = (n_heads / n_kv_heads + heads - 1) / heads;
    p.window = window; p.scale = scale;
    p.n_splits = n_splits; p.pages_per_split = pages_per_split;
    p.k_new = (const h16*)k_new; p.v_new = (const h16*)v_new; p.kv_stride = kv_stride; p.cache_w = (h16*)cache;
    const dim3 grid(n_kv_heads * p.head_tiles, n_rows, n_splits);
    switch (head_dim) {
        case 64: return launch_tiles<64>(heads / 8, warps, grid, stream, p);
        case 80: return launch_tiles<80>(heads / 8, warps, grid, stream, p);
        case 96: return launch_tiles<96>(heads / 8, warps, grid, stream, p);
        case 112: return launch_tiles<112>(heads / 8, warps, grid, stream, p);
        default: return launch_tiles<128>(heads / 8, warps, grid, stream, p);
    }
}
