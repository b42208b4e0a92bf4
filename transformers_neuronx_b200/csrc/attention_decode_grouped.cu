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
// What a warp waits for is its pages, so they are asked for two and more ahead, by asynchronous copies into a ring of its own in
// shared memory (the next page's in registers, asked for once this one's are used up, keep half as many bytes on their way: 48 rows
// of 32 heads on 8 over 950 to 1,900 tokens 61.7 us, with the ring 53.8; 43.5 would be the copy rate).
// Measured, pages beyond the second-level cache, us a call (with one block a head): the same 54 (165), 64 rows over 950 to 1,900
// 71 (223), 40 rows of 32 heads on 2 27 (147), 64 32 (216).  With as many key/value heads as heads: 80 dims, 8 rows of 32 heads over
// 700 to 1,400 25 (33), 64 over 750 to 1,500 120 (180); 128 dims, 64 rows of 40 heads over 200 to 400 71 (77).
// Tried: all pages of all heads laid end to end and cut into equal runs, one a warp, partial sums through scratch memory and a
// second kernel: 10 us of fixed costs, at best level (64 rows of 40 heads over 400 tokens 76).
//
// Grid (key/value heads x head tiles, rows, splits), 4, 8 or 12 warps; a warp takes every WARPS-th page of the split's range.
// Warps are merged in shared memory.  The splits of a (row, head tile)
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
    int n_splits;                    // a cluster's blocks
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

// One warp's part of a (row, tile of query heads): its running maxima, sums and output, the page it holds, and the step over a page.
// NT: tiles of eight query heads (1 or 2) that the heads fill.  An SM's registers hold twelve warps of the first kind and eight of
// the second.
template <int D, int NT, bool BIAS>
struct Heads {
    static constexpr int STEPS = D / 16;                // 16-dim steps of the scores' contraction, 16-dim tiles of the output
    static constexpr int N32 = D / 32, N64 = D / 64, REST = (D % 64) / 16;
    int g, c;                                           // the lane as (row, column) of an 8-column operand
    float m[NT][2], l[NT][2], acc[NT][STEPS][4];        // of heads 2c and 2c + 1 of each tile
    float bias_mul[NT][2], bias_rate[NT][2];            // of a logarithm to base 2
    uint32_t kr[2][2 * STEPS], vr[4][STEPS];            // two key rows, four value rows

    // A warp's pages pass through a ring of its own in shared memory: copies (16 bytes a lane, asynchronous) of the next SLOTS
    // pages are on their way while one is worked on.  Rows lie so that the lanes' reads of them meet all banks: 64 bytes apart
    // modulo 128 (keys: eight lanes read four pieces of two neighbouring rows), or pieces exchanged by the row's number (112 dims: two
    // of four pieces meet).
    static constexpr int PIECES = D / 8;                                     // of 16 bytes in a row
    static constexpr int K_PITCH = D == 80 ? 192 : 2 * D, V_PITCH = D == 80 ? 192 : 2 * D;
    static constexpr int SLOT = PAGE * (K_PITCH + V_PITCH), SLOTS = D == 64 ? 3 : 2;
    static constexpr int QUERY_BYTES = NT * STEPS * 256, WARP_BYTES = SLOTS * SLOT + QUERY_BYTES;       // the ring, then the queries
    static_assert((NT == 1 ? 12 : 8) * WARP_BYTES + 2 * 1024 <= 232448, "the warps that an SM's registers hold");
    static __device__ __forceinline__ int key_at(int row, int piece) { return row * K_PITCH + (D % 64 == 0 ? piece ^ (row & 1) << 2 : piece) * 16; }
    static __device__ __forceinline__ int value_at(int row, int piece) {
        return PAGE * K_PITCH + row * V_PITCH + (piece < 8 * N64 ? piece ^ ((row >> 1 & 3) << 1) : piece) * 16;
    }
    // Copies of a page (paged) or of the token's own key and value (as row 0) into a slot.  Values that no query may see, which may
    // hold anything, are filled with zeros: p = 0 times them is 0.
    template <typename Seen>
    __device__ __forceinline__ void ask(uint32_t slot, const h16* keys, const h16* values, bool paged, int j0, int lane, Seen seen) const {
#pragma unroll
        for (int i = 0; i < (PAGE * PIECES + 31) / 32; ++i) {
            const int n = lane + 32 * i, row = n / PIECES, piece = n % PIECES;
            if (PAGE * PIECES % 32 != 0 && row >= PAGE) break;
            const int k_bytes = paged || row == 0 ? 16 : 0, v_bytes = (paged ? seen(j0 + row) : row == 0) ? 16 : 0;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(slot + key_at(row, piece)),
                         "l"(k_bytes ? keys + row * D + piece * 8 : keys), "r"(k_bytes) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(slot + value_at(row, piece)),
                         "l"(v_bytes ? values + row * D + piece * 8 : values), "r"(v_bytes) : "memory");
        }
    }
    static __device__ __forceinline__ void asked() { asm volatile("cp.async.commit_group;" ::: "memory"); }
    template <int PENDING> static __device__ __forceinline__ void landed() {     // all but the newest PENDING pages, for the whole warp
        asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
        __syncwarp();
    }

    // the queries as the 8-column operand: lane (g, c) holds head g's dims in the order its key pieces come in (in registers they
    // spilled others: 88 us for the first measurement above); qs: this lane's place
    __device__ __forceinline__ void load_queries(const GroupedParams& p, int row, int h0, int n_mine, uint2* qs) {
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
    }
    __device__ __forceinline__ void start(const GroupedParams& p, int h0, int n_mine, bool sink_here) {
#pragma unroll
        for (int t = 0; t < NT; ++t) {
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                m[t][x] = sink_here ? p.sink.score : -INFINITY;
                l[t][x] = sink_here && g == 0 ? 1.f : 0.f;                   // counted once: the sum runs over the lanes of a head
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
    }
    // A page's keys, or the token's own one (paged false) as row 0.
    __device__ __forceinline__ void load_keys(const h16* base, bool paged) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int key = g + 8 * r;
            const bool there = paged || key == 0;
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
    }
    // rows that no query may see, and rows never written, which may hold anything, stay zero: p = 0 times them is 0
    template <typename Seen>
    __device__ __forceinline__ void load_values(const h16* base, bool paged, int j0, Seen seen) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int key = 2 * c + (r & 1) + 8 * (r >> 1);
            const bool there = paged ? seen(j0 + key) : key == 0;
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
    }
    // The same from a slot of the ring.
    __device__ __forceinline__ void take_keys(const uint8_t* slot) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int row = g + 8 * r;
#pragma unroll
            for (int i = 0; i < N32; ++i) {
                const uint4 v = *(const uint4*)(slot + key_at(row, 4 * i + c));
                kr[r][4 * i] = v.x; kr[r][4 * i + 1] = v.y; kr[r][4 * i + 2] = v.z; kr[r][4 * i + 3] = v.w;
            }
            if constexpr (D % 32 != 0) {
                const uint2 v = *(const uint2*)(slot + row * K_PITCH + 64 * N32 + 8 * c);
                kr[r][4 * N32] = v.x; kr[r][4 * N32 + 1] = v.y;
            }
        }
    }
    __device__ __forceinline__ void take_values(const uint8_t* slot) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int row = 2 * c + (r & 1) + 8 * (r >> 1);
#pragma unroll
            for (int i = 0; i < N64; ++i) {
                const uint4 v = *(const uint4*)(slot + value_at(row, 8 * i + g));
                vr[r][4 * i] = v.x; vr[r][4 * i + 1] = v.y; vr[r][4 * i + 2] = v.z; vr[r][4 * i + 3] = v.w;
            }
            const uint8_t* rest = slot + PAGE * K_PITCH + row * V_PITCH + 128 * N64 + 4 * REST * g;
            if constexpr (REST == 1) {
                vr[r][4 * N64] = *(const uint32_t*)rest;
            } else if constexpr (REST == 2) {
                const uint2 v = *(const uint2*)rest;
                vr[r][4 * N64] = v.x; vr[r][4 * N64 + 1] = v.y;
            } else if constexpr (REST == 3) {
#pragma unroll
                for (int w = 0; w < 3; ++w) vr[r][4 * N64 + w] = ((const uint32_t*)rest)[w];
            }
        }
    }
    // The scores of the page whose keys the lane holds: [0], [1]: key g of heads 2c, 2c + 1;  [2], [3]: key g + 8.
    __device__ __forceinline__ void scores(const uint2* qs, float (&s)[NT][4]) const {
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
    }
    // The softmax step over them and the values' products; the page's first key is j0, the query's position pos.
    __device__ __forceinline__ void add_page(const GroupedParams& p, float (&s)[NT][4], int pos, int j0, bool see0, bool see1) {
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
    }
    // this lane's pair of neighbouring dims in tile k of the output
    __device__ __forceinline__ int dim_of(int k) const {
        return k < 4 * N64 ? 64 * (k / 4) + 8 * g + 2 * (k % 4) : 64 * N64 + 2 * REST * g + 2 * (k - 4 * N64);
    }
    __device__ __forceinline__ float denominator(int n, int x) const {       // in every lane of the head
        float v = l[n][x];
        v += __shfl_xor_sync(0xffffffffu, v, 4);
        v += __shfl_xor_sync(0xffffffffu, v, 8);
        v += __shfl_xor_sync(0xffffffffu, v, 16);
        return v;
    }
};

// Shared memory of a warp.  Without a ring (one row: the product that follows streams its weights through the first-level cache, which
// a large share of shared memory would leave 28 KB; a step of 4 layers of width 4096 502 us with rings, 438 without) the next page
// waits in registers, asked for when this one's numbers are used up.
template <int D, int NT, bool BIAS, bool RING> __host__ __device__ constexpr int warp_bytes() {
    using H = Heads<D, NT, BIAS>;
    return RING ? H::WARP_BYTES : (H::QUERY_BYTES > 32 * NT * (D + 4) ? H::QUERY_BYTES : 32 * NT * (D + 4));
}

template <int D, int NT, int WARPS, bool BIAS, bool RING>
__global__ void __launch_bounds__(WARPS * 32, (NT == 1 ? 12 : 8) / WARPS)
attention_decode_grouped_kernel(const GroupedParams p) {
    constexpr int HEADS = 8 * NT, STEPS = D / 16;
    constexpr int PITCH = D + 4;
    __shared__ float sm_m[WARPS][HEADS], sm_l[WARPS][HEADS], block_m[HEADS], block_l[HEADS];
    // a warp's ring and queries, and in the end its sums, [HEADS][PITCH]
    extern __shared__ __align__(128) uint8_t smem_raw[];
    float* const sm_o = (float*)smem_raw;
    constexpr int WARP_BYTES = warp_bytes<D, NT, BIAS, RING>(), O_STEP = WARP_BYTES / 4;
    static_assert(HEADS * PITCH <= O_STEP, "a warp's sums fit where its ring and queries were");
    pdl_launch_dependents();
    pdl_wait();

    const int kvh = blockIdx.x / p.head_tiles, tile = blockIdx.x % p.head_tiles, ri = blockIdx.y, split = blockIdx.z;
    const int group = p.n_heads / p.n_kv_heads;
    const int h0 = kvh * group + tile * HEADS, n_mine = min(HEADS, group - tile * HEADS);     // the block's query heads
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
    const int row = p.rows ? p.rows[ri] : ri;
    if (row < 0) return;                                        // a padded entry of the row list of a captured step
    const int req = p.token_request[row], pos = p.positions[row];       // asked for together, and the queries beside them
    Heads<D, NT, BIAS> w;
    w.g = g; w.c = c;
    uint8_t* const ring = smem_raw + warp * WARP_BYTES;
    uint2* const qs = (uint2*)(ring + (RING ? w.SLOTS * w.SLOT : 0)) + lane;
    w.load_queries(p, row, h0, n_mine, qs);
    if (req < 0) return;                                        // a padded row of a captured batch
    const int* bt = p.block_tables + (size_t)req * p.bt_stride;
    const int kv_len = pos + 1;
    const int first_key = first_visible_key(pos, p.window);
    const int n_pages = (kv_len + PAGE - 1) / PAGE;
    const BlockWalk walk = walk_blocks(first_key, p.keep_first, PAGE);       // pages are numbered along the visible ones
    // the row's own pages in equal parts: the plan's bound on the contexts may be far above them (a captured step's)
    const int pages_all = walk.count(n_pages - 1), per_split = (pages_all + p.n_splits - 1) / p.n_splits;
    const int page_lo = split * per_split, page_hi = min(pages_all, (split + 1) * per_split);
    const size_t head_block = (size_t)PAGE * D;
    const bool own_here = p.k_new != nullptr && walk.place(pos / PAGE) / per_split == split;    // one answer for the block
    const int cached_len = p.k_new != nullptr ? pos : kv_len;
    const int my_pages = page_hi > page_lo + warp ? (page_hi - page_lo - warp + WARPS - 1) / WARPS : 0;
    // the token's own key is a chunk of one key, of the warp whose turn comes after the pages' (warp 0 may have one page more)
    const int n_chunks = my_pages + (own_here && warp == max(page_hi - page_lo, 0) % WARPS ? 1 : 0);

    w.start(p, h0, n_mine, p.sink.on && split == 0 && warp == 0);

    auto seen = [&](int j) { return (j >= first_key || j < p.keep_first) && j < cached_len; };
    // chunk t of the warp: its first key and its key and value rows
    auto first_of = [&](int t) { return t < my_pages ? walk.at(page_lo + warp + t * WARPS) * PAGE : pos; };
    auto page_of = [&](int t) { return t < my_pages ? bt[walk.at(page_lo + warp + t * WARPS)] : 0; };
    auto rows_of = [&](int t, int page, int which) -> const h16* {
        if (t < my_pages) return p.cache + (((size_t)page * 2 + which) * p.n_kv_heads + kvh) * head_block;
        return (which ? p.v_new : p.k_new) + (size_t)row * p.kv_stride + (size_t)kvh * D;
    };
    auto ask = [&](int t, int page) {
        if (t < n_chunks) w.ask(shared_address(ring) + t % w.SLOTS * w.SLOT, rows_of(t, page, 0), rows_of(t, page, 1), t < my_pages, first_of(t), lane, seen);
        w.asked();
    };
    if constexpr (!RING) {
        auto load_keys = [&](int t, int page) { w.load_keys(rows_of(t, page, 0), t < my_pages); };
        auto load_values = [&](int t, int page) { w.load_values(rows_of(t, page, 1), t < my_pages, first_of(t), seen); };
        int next_page = 0;
        if (n_chunks > 0) {
            const int page = page_of(0);
            load_keys(0, page);
            load_values(0, page);
            next_page = page_of(1);
        }
        for (int t = 0; t < n_chunks; ++t) {
            const bool more = t + 1 < n_chunks;
            float s[NT][4];
            w.scores(qs, s);
            if (more) load_keys(t + 1, next_page);
            const int j0 = first_of(t);
            const bool paged = t < my_pages;
            w.add_page(p, s, pos, j0, paged ? seen(j0 + g) : g == 0, paged && seen(j0 + g + 8));
            if (more) {
                load_values(t + 1, next_page);
                next_page = t + 2 < n_chunks ? page_of(t + 2) : 0;
            }
        }
    } else {
        int pages[w.SLOTS];
#pragma unroll
        for (int i = 0; i < w.SLOTS; ++i) pages[i] = page_of(i);
#pragma unroll
        for (int i = 0; i < w.SLOTS; ++i) ask(i, pages[i]);
        int next_page = page_of(w.SLOTS);
        for (int t = 0; t < n_chunks; ++t) {
            const uint8_t* slot = ring + t % w.SLOTS * w.SLOT;
            w.template landed<w.SLOTS - 1>();
            float s[NT][4];
            w.take_keys(slot);
            w.scores(qs, s);
            w.take_values(slot);
            __syncwarp();                                        // the slot is read out
            ask(t + w.SLOTS, next_page);
            next_page = page_of(t + 1 + w.SLOTS);
            const int j0 = first_of(t);
            const bool paged = t < my_pages;
            w.add_page(p, s, pos, j0, paged ? seen(j0 + g) : g == 0, paged && seen(j0 + g + 8));
        }
        w.template landed<0>();
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
            const float v = w.denominator(n, x);
            if (g == 0) { sm_m[warp][n * 8 + 2 * c + x] = w.m[n][x]; sm_l[warp][n * 8 + 2 * c + x] = v; }
#pragma unroll
            for (int k = 0; k < STEPS; ++k) {
                *(float2*)&sm_o[warp * O_STEP + (n * 8 + 2 * c + x) * PITCH + w.dim_of(k)] = make_float2(w.acc[n][k][x], w.acc[n][k][2 + x]);
            }
        }
    }
    __syncthreads();
    // one factor per warp and head, then every output element is a sum over the warps
    const int tid = threadIdx.x;
    if (tid < HEADS) {
        float M = -INFINITY, L = 0.f;
#pragma unroll
        for (int i = 0; i < WARPS; ++i) M = fmaxf(M, sm_m[i][tid]);
#pragma unroll
        for (int i = 0; i < WARPS; ++i) {
            const float f = sm_m[i][tid] == -INFINITY ? 0.f : __expf(sm_m[i][tid] - M);
            L += sm_l[i][tid] * f;
            sm_m[i][tid] = f;
        }
        block_m[tid] = M; block_l[tid] = L;
    }
    __syncthreads();
    for (int i = tid; i < n_mine * D; i += WARPS * 32) {
        const int x = i / D, dim = i % D;
        float o = 0.f;
#pragma unroll
        for (int k = 0; k < WARPS; ++k) {
            const float f = sm_m[k][x];
            o += f == 0.f ? 0.f : sm_o[k * O_STEP + x * PITCH + dim] * f;
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

template <int D, int NT, int WARPS, bool BIAS, bool RING>
int launch_as(dim3 grid, cudaStream_t stream, const GroupedParams& p) {
    constexpr size_t smem = (size_t)WARPS * warp_bytes<D, NT, BIAS, RING>();
    auto kernel = attention_decode_grouped_kernel<D, NT, WARPS, BIAS, RING>;
    static TnxSmemLimit limit;
    if (const int rc = limit.allow(kernel, smem)) return rc;
    if (p.n_splits == 1) return tnx_launch_in_order(kernel, grid, dim3(WARPS * 32), smem, stream, p);
    return tnx_launch_cluster(0, dim3(1, 1, p.n_splits), kernel, grid, dim3(WARPS * 32), smem, stream, p);
}
template <int D, int NT, int WARPS, bool BIAS>
int launch_ring(dim3 grid, cudaStream_t stream, const GroupedParams& p) {
    return grid.y > 1 ? launch_as<D, NT, WARPS, BIAS, true>(grid, stream, p) : launch_as<D, NT, WARPS, BIAS, false>(grid, stream, p);
}
template <int D, int NT>
int launch(int warps, dim3 grid, cudaStream_t stream, const GroupedParams& p) {
    constexpr int MOST = NT == 1 ? 12 : 8;
    if (warps == 4) return p.bias.mul ? launch_ring<D, NT, 4, true>(grid, stream, p) : launch_ring<D, NT, 4, false>(grid, stream, p);
    if (warps == MOST) return p.bias.mul ? launch_ring<D, NT, MOST, true>(grid, stream, p) : launch_ring<D, NT, MOST, false>(grid, stream, p);
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
                                            int page_size, int window, float scale, int n_splits,
                                            const void* k_new, const void* v_new, int kv_stride, int warps, int keep_first, const float* bias_mul, const float* bias_rate,
                                            int has_sink, float sink_score, cudaStream_t stream) {
    if (n_rows <= 0) return 0;
    const int heads = heads_of_a_block(n_heads, n_kv_heads, head_dim);
    if (!heads || page_size != PAGE || q_stride % 8 || ((uintptr_t)q & 15) || ((uintptr_t)cache & 15)) return TNX_ERR_UNSUPPORTED;
    if ((k_new == nullptr) != (v_new == nullptr)) return TNX_ERR_BAD_ARG;
    if (k_new && (kv_stride % 8 || (((uintptr_t)k_new | (uintptr_t)v_new) & 15))) return TNX_ERR_UNSUPPORTED;
    if (n_splits < 1 || n_splits > 8 || n_rows > 65535) return TNX_ERR_BAD_ARG;
    if (keep_first < 0 || (bias_mul && !bias_rate)) return TNX_ERR_BAD_ARG;
    GroupedParams p;
    p.keep_first = keep_first; p.bias.mul = bias_mul; p.bias.rate = bias_rate;
    p.sink.on = has_sink; p.sink.score = sink_score;
    p.q = (const h16*)q; p.q_stride = q_stride; p.cache = (const h16*)cache;
    p.block_tables = block_tables; p.bt_stride = bt_stride; p.rows = rows; p.token_request = token_request;
    p.positions = positions; p.out = (h16*)out; p.out_stride = out_stride;
    p.n_heads = n_heads; p.n_kv_heads = n_kv_heads; p.head_tiles = (n_heads / n_kv_heads + heads - 1) / heads;
    p.window = window; p.scale = scale;
    p.n_splits = n_splits;
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
