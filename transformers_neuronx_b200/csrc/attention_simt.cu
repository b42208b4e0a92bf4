// Attention over the paged cache on CUDA cores, scores and softmax in 32-bit: the true 32-bit
// path, and the path for head sizes that the tensor-core kernels refuse.
//
// The query at position p of its request reads the keys at
// positions first_visible_key(p, window) .. p (a sliding window, a chunked mask or all: common.cuh), with a window also
// the first keep_first ones, all of which are in the cache when the kernel runs (this
// step's keys and values are written before it).  Keys are visited in ascending position, 32 at a
// time, with an online softmax; the result for a token therefore does not depend on how the
// request was cut into steps or on what else is in the batch.
//
//   s_j = scale * <q, k_j> (- the distance bias);  out = sum_j exp(s_j - max) v_j / sum_j exp(s_j - max)
//
// Three kernels with the same arithmetic, operation by operation, so that a row's result is the same bit for bit in each:
//   wide    one warp per (query token, head), any mask, head size and alignment
//   rows    one block per (query token, head), heads of up to 128 dims: 64 or 128 keys and values at a time are staged in
//           shared memory by all four warps; the dot products of the staged keys are formed side by side, the sums over the
//           keys stay in their order.  It is a chain of stages: load, score, rescale, add.
//   tiles   for portions of prompts without a mask: a block takes 64 neighbouring rows and one head, 64 staged keys and
//           values serve all of them; what a tile holds beside its largest portion goes to a kernel that runs beside it (others)
// Measured, 32 heads of 64, 32-bit: a portion of 499 tokens behind 256 beside three single rows of 500 to 700 keys, 2,417 us
// with `wide` for all rows, 1,200 with `rows`, 147 with `tiles` (in tiles of 32 rows with the single rows in a kernel
// after them 279); four single rows of 100 to 900 keys 382 us with `wide`, 53 with `rows`; 64 of 100 to 1,360 keys 1,106 and 434;
// a portion of 2,048 tokens, 16 heads of 128, 0.58 ms (tiles of 32 rows 1.66).
#include "common.cuh"

namespace {
constexpr int WIDE_DIMS_PER_LANE = 24;  // head_dim <= 768: rows wider than any 16-bit kernel takes (a wide latent)

// The wide kernel.  MAX_DIMS_PER_LANE: 8 (head_dim <= 256) or WIDE_DIMS_PER_LANE; a lane accumulates that many output dims.
template <typename T, int MAX_DIMS_PER_LANE>
__global__ void __launch_bounds__(128)
attention_simt_wide_kernel(const T* __restrict__ q, int q_stride, const T* __restrict__ cache,
                      const int* __restrict__ block_tables, int bt_stride,
                      const int* __restrict__ token_request, const int* __restrict__ positions,
                      T* __restrict__ out, int out_stride, int n_tokens, int n_heads, int n_kv_heads,
                      int head_dim, int page_size, int window, float scale, int keep_first, DistanceBias bias,
                      SoftmaxSink sink) {
    extern __shared__ float qsm[];                  // [warps per block][head_dim]
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long pair = (long long)blockIdx.x * (blockDim.x >> 5) + warp;
    if (pair >= (long long)n_tokens * n_heads) return;
    const int n = (int)(pair / n_heads), h = (int)(pair % n_heads);
    const int req = token_request[n];
    if (req < 0) return;                            // a padded row of a captured batch
    const int pos = positions[n];
    const int kvh = h / (n_heads / n_kv_heads);
    const int* bt = block_tables + (size_t)req * bt_stride;
    float* qs = qsm + warp * head_dim;
    const T* qrow = q + (size_t)n * q_stride + (size_t)h * head_dim;
    for (int c = lane; c < head_dim; c += 32) qs[c] = to_float(qrow[c]);
    __syncwarp();

    const size_t head_block = (size_t)page_size * head_dim;
    float m = sink.on ? sink.score : -INFINITY, l = sink.on ? 1.f : 0.f;
    float acc[MAX_DIMS_PER_LANE];
#pragma unroll
    for (int i = 0; i < MAX_DIMS_PER_LANE; ++i) acc[i] = 0.f;
    // the visible keys, numbered without the gap between the first ones that are kept and the window
    const int first = first_visible_key(pos, window);
    const int kept = keep_first < first ? keep_first : first, gap = first - kept;
    const int n_keys = pos + 1 - gap;
    const float mul = bias.mul ? bias.mul[h] : 0.f, rate = bias.mul ? bias.rate[h] : 0.f;

    for (int c0 = 0; c0 < n_keys; c0 += 32) {
        const int i = c0 + lane, j = i < kept ? i : i + gap;
        float s = -INFINITY;
        if (i < n_keys) {
            const int page = bt[j / page_size];
            const T* krow = cache + (((size_t)page * 2 + 0) * n_kv_heads + kvh) * head_block +
                            (size_t)(j % page_size) * head_dim;
            float dot = 0.f;
            for (int c = 0; c < head_dim; ++c) dot = fmaf(qs[c], to_float(krow[c]), dot);
            s = dot * scale;
            if (bias.mul) s -= mul * log1pf(rate * (float)(pos - j));
        }
        const float m_new = fmaxf(m, warp_max(s));
        const float p = (i < n_keys) ? expf(s - m_new) : 0.f;
        const float corr = (m == -INFINITY) ? 0.f : expf(m - m_new);
        l = l * corr + warp_sum(p);
        m = m_new;
#pragma unroll
        for (int i = 0; i < MAX_DIMS_PER_LANE; ++i) acc[i] *= corr;
        const int cnt = min(32, n_keys - c0);
        for (int jj = 0; jj < cnt; ++jj) {
            const float pj = __shfl_sync(0xffffffffu, p, jj);
            const int jk = c0 + jj < kept ? c0 + jj : c0 + jj + gap;
            const int page = bt[jk / page_size];
            const T* vrow = cache + (((size_t)page * 2 + 1) * n_kv_heads + kvh) * head_block +
                            (size_t)(jk % page_size) * head_dim;
#pragma unroll
            for (int i = 0; i < MAX_DIMS_PER_LANE; ++i) {
                const int c = lane + 32 * i;
                if (c < head_dim) acc[i] = fmaf(pj, to_float(vrow[c]), acc[i]);
            }
        }
    }
    const float inv = 1.0f / l;
    T* orow = out + (size_t)n * out_stride + (size_t)h * head_dim;
#pragma unroll
    for (int i = 0; i < MAX_DIMS_PER_LANE; ++i) {
        const int c = lane + 32 * i;
        if (c < head_dim) orow[c] = from_float<T>(acc[i] * inv);
    }
}

template <typename T>
struct SimtParams {
    const T* q; int q_stride;
    const T* cache;
    const int* block_tables; int bt_stride;
    const int* token_request;
    const int* positions;
    T* out; int out_stride;
    int n_tokens, n_heads, n_kv_heads, head_dim, page_size, window;
    float scale;
    int keep_first;
    DistanceBias bias;
    SoftmaxSink sink;
    int page_shift;                      // page_size = 2^page_shift, or -1
};

constexpr int TILE_ROWS = 64;            // rows of a tile: tile t holds rows 64 t .. 64 t + 63 of the batch

__device__ __forceinline__ float4 load4(const float* p) { return *(const float4*)p; }
__device__ __forceinline__ float4 load4(const h16* p) {
    const uint2 raw = *(const uint2*)p;
    const float2 a = h16x2_to_float2(*(const h16x2*)&raw.x), b = h16x2_to_float2(*(const h16x2*)&raw.y);
    return make_float4(a.x, a.y, b.x, b.y);
}

// One row and one head by THREADS threads (no fewer than KEYS and the head's dims): a block (part < 0), or part 0 or 1 of one.  (A named
// barrier where the block's own would do cost the rows kernel 4 %.)
template <typename T, int KEYS, int THREADS, bool WHOLE = true>
__device__ __forceinline__ void attend_row(const SimtParams<T>& p, float* sm, int n, int h, int part = -1) {
    auto meet = [&] {
        if (WHOLE) __syncthreads();
        else asm volatile("bar.sync %0, %1;" ::"r"(1 + part), "n"(THREADS) : "memory");
    };
    const int d = p.head_dim, d4 = d / 4;
    float* ks = sm;                                 // [KEYS][d + 4]: a warp's 16-byte reads down the rows meet all banks evenly
    float* vs = ks + KEYS * (d + 4);                // [KEYS][d]
    float* qs = vs + KEYS * d;                      // [d]
    float* ss = qs + d;                             // [KEYS] the staged keys' scores
    const int tid = WHOLE ? threadIdx.x : threadIdx.x % THREADS, lane = tid & 31;
    const int kvh = h / (p.n_heads / p.n_kv_heads);
    const size_t head_block = (size_t)p.page_size * d;
    const float mul = p.bias.mul ? p.bias.mul[h] : 0.f, rate = p.bias.mul ? p.bias.rate[h] : 0.f;
    const int req = p.token_request[n];
    if (req < 0) return;                            // a padded row of a captured batch
    const int pos = p.positions[n];
    const int* bt = p.block_tables + (size_t)req * p.bt_stride;
    // the visible keys, numbered without the gap between the first ones that are kept and the window
    const int first = first_visible_key(pos, p.window);
    const int kept = p.keep_first < first ? p.keep_first : first, gap = first - kept;
    const int n_keys = pos + 1 - gap;
    float m = p.sink.on ? p.sink.score : -INFINITY, l = p.sink.on ? 1.f : 0.f, acc = 0.f;
    const bool has_dim = tid < d;               // the thread owns dim `tid` of the output
    for (int k0 = 0; k0 < n_keys; k0 += KEYS) {
        const int staged = min(KEYS, n_keys - k0);
        meet();                        // the keys before are done with
        if (k0 == 0)
            for (int c = tid; c < d; c += THREADS) qs[c] = to_float(p.q[(size_t)n * p.q_stride + (size_t)h * d + c]);
#pragma unroll 8
        for (int i = tid; i < staged * d4; i += THREADS) {
            const int kk = i / d4, c = (i % d4) * 4, i_key = k0 + kk, j = i_key < kept ? i_key : i_key + gap;
            const T* krow = p.cache + ((size_t)bt[j / p.page_size] * 2 * p.n_kv_heads + kvh) * head_block
                            + (size_t)(j % p.page_size) * d + c;
            *(float4*)(ks + kk * (d + 4) + c) = load4(krow);
            *(float4*)(vs + kk * d + c) = load4(krow + (size_t)p.n_kv_heads * head_block);
        }
        meet();
        if (tid < staged) {
            const float* kr = ks + tid * (d + 4);
            float dot = 0.f;
#pragma unroll 4
            for (int c = 0; c < d; c += 4) {
                const float4 k4 = *(const float4*)(kr + c), q4 = *(const float4*)(qs + c);
                dot = fmaf(q4.x, k4.x, dot); dot = fmaf(q4.y, k4.y, dot);
                dot = fmaf(q4.z, k4.z, dot); dot = fmaf(q4.w, k4.w, dot);
            }
            float s = dot * p.scale;
            const int i_key = k0 + tid, j = i_key < kept ? i_key : i_key + gap;
            if (p.bias.mul) s -= mul * log1pf(rate * (float)(pos - j));
            ss[tid] = s;
        }
        meet();
        for (int c0 = 0; c0 < staged; c0 += 32) {               // every warp keeps the running maximum and sum for itself
            const int cnt = min(32, staged - c0);
            const float s = lane < cnt ? ss[c0 + lane] : -INFINITY;
            const float m_new = fmaxf(m, warp_max(s));
            const float e = lane < cnt ? expf(s - m_new) : 0.f;
            const float corr = (m == -INFINITY) ? 0.f : expf(m - m_new);
            l = l * corr + warp_sum(e);
            m = m_new;
            acc *= corr;
            const float* vr = vs + c0 * d + tid;
            if (cnt == 32) {
#pragma unroll
                for (int jj = 0; jj < 32; ++jj) {
                    const float pj = __shfl_sync(0xffffffffu, e, jj);
                    if (has_dim) acc = fmaf(pj, vr[jj * d], acc);
                }
            } else {
                for (int jj = 0; jj < cnt; ++jj) {
                    const float pj = __shfl_sync(0xffffffffu, e, jj);
                    if (has_dim) acc = fmaf(pj, vr[jj * d], acc);
                }
            }
        }
    }
    if (has_dim) p.out[(size_t)n * p.out_stride + (size_t)h * d + tid] = from_float<T>(acc * (1.0f / l));
}

template <typename T, int KEYS>
__global__ void __launch_bounds__(128)
attention_simt_rows_kernel(const SimtParams<T> p) {
    extern __shared__ __align__(16) float sm[];
    pdl_launch_dependents();
    pdl_wait();
    attend_row<T, KEYS, 128>(p, sm, blockIdx.x, blockIdx.y);
}

// A tile's portions: in 64 neighbouring rows, a request's rows.
struct Tile {
    int reqs[TILE_ROWS], poss[TILE_ROWS];                                                    // of the rows
    int rows_of[TILE_ROWS], place_of[TILE_ROWS], most_of[TILE_ROWS], least_of[TILE_ROWS];    // of their portions: rows, the row's place, keys
    int keys_of[TILE_ROWS], row_at[TILE_ROWS];                                               // of the slots: see attend_portion
    float corr_of[2][TILE_ROWS], m_of[TILE_ROWS], l_of[TILE_ROWS];
};
template <typename T>
__device__ __forceinline__ void load_tile(const SimtParams<T>& p, Tile& t, int tile) {       // by the whole block
    const int tid = threadIdx.x;
    __syncthreads();                                 // the tile before is done with
    if (tid < TILE_ROWS) {
        const int n = tile * TILE_ROWS + tid;
        t.reqs[tid] = n < p.n_tokens ? p.token_request[n] : -1;
        t.poss[tid] = n < p.n_tokens ? p.positions[n] : 0;
    }
    __syncthreads();
    if (tid < TILE_ROWS) {
        const int req = t.reqs[tid];
        int most = 0, least = 0x7fffffff, rows = 0, place = 0;
#pragma unroll 8
        for (int i = 0; i < TILE_ROWS; ++i) {
            if (t.reqs[i] != req) continue;
            place += i < tid; ++rows;
            most = max(most, t.poss[i] + 1); least = min(least, t.poss[i] + 1);
        }
        t.most_of[tid] = most; t.least_of[tid] = least; t.rows_of[tid] = rows; t.place_of[tid] = place;
    }
}
// The portion that a tile's own block takes: the one with the most rows, of equal ones the first; 0: the tile has single rows only.
__device__ __forceinline__ int portion_rank(int rows, int first) { return rows > 1 ? rows * TILE_ROWS + TILE_ROWS - 1 - first : 0; }
__device__ __forceinline__ int portion_first(int rank) { return TILE_ROWS - 1 - rank % TILE_ROWS; }

// The portion whose first row is row `lead` of the tile, in slots 0 .. of the tile's arrays; LIVE: no fewer than its rows.
// 64 keys and values are staged at a time:
//   scores   a thread owns PR rows and PK keys: PR + PK 16-byte reads of shared memory feed 4 PR PK multiply-adds, in the order
//            of the dims; they go to shared memory
//   softmax  a thread owns a row's 32-key step (maximum, sum, rescaling: those of the other kernels)
//   values   a thread owns PV_ROWS rows and four dims, the keys in their order
constexpr int STAGE_KEYS = 64;
template <typename T, int DIMS, int THREADS, int LIVE>
__device__ __forceinline__ void attend_portion(const SimtParams<T>& p, Tile& t, float* sm, int row0, int lead, int h) {
    constexpr int KEYS = STAGE_KEYS;
    constexpr int DG = DIMS / 4;                                  // groups of four dims
    constexpr int RG_V = THREADS / DG, PV_ROWS = LIVE / RG_V;     // thread: rows rv, rv + RG_V, ..; dims 4 dv ..
    constexpr int PK = 4, KG = KEYS / PK, RG = THREADS / KG, PR = LIVE > RG ? LIVE / RG : 1;       // thread: rows rq, rq + RG, ..; keys kq, kq + KG, ..
    constexpr int Q_ROWS = PR * RG;
    const int SP = max(p.head_dim, KEYS) + 4;
    const int tid = threadIdx.x, lane = tid & 31;
    const int d = p.head_dim, d4 = d / 4, dp = d + 4;
    float* qs = sm;                                 // [Q_ROWS][d + 4]
    float* ks = qs + Q_ROWS * dp;                   // [KEYS][d + 4]
    float* vs = ks + KEYS * SP;                     // [KEYS][d]
    float* ps = ks;                                 // [Q_ROWS][KEYS + 4]: scores, then probabilities, over the keys once these are used
    const int kvh = h / (p.n_heads / p.n_kv_heads);
    const size_t head_block = (size_t)p.page_size * d;
    const float mul = p.bias.mul ? p.bias.mul[h] : 0.f, rate = p.bias.mul ? p.bias.rate[h] : 0.f;
    const int rq = tid / KG, kq = tid % KG, rv = tid / DG, dv = tid % DG;
    const bool has_dims = 4 * dv < d;
    const int req = t.reqs[lead], most = t.most_of[lead], least = t.least_of[lead], rows = t.rows_of[lead];
    const int* bt = p.block_tables + (size_t)req * p.bt_stride;
    if (tid < TILE_ROWS) {
        if (t.reqs[tid] == req) { t.keys_of[t.place_of[tid]] = t.poss[tid] + 1; t.row_at[t.place_of[tid]] = row0 + tid; }
        if (tid >= rows) { t.keys_of[tid] = 0; t.row_at[tid] = -1; }
        t.m_of[tid] = p.sink.on ? p.sink.score : -INFINITY;
        t.l_of[tid] = p.sink.on ? 1.f : 0.f;
    }
    __syncthreads();
    for (int i = tid; i < Q_ROWS * d4; i += THREADS) {
        const int r = i / d4, c = (i % d4) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t.row_at[r] >= 0) {
            const T* src = p.q + (size_t)t.row_at[r] * p.q_stride + (size_t)h * d + c;
            v = make_float4(to_float(src[0]), to_float(src[1]), to_float(src[2]), to_float(src[3]));
        }
        *(float4*)(qs + r * dp + c) = v;
    }
    float4 acc[PV_ROWS];
#pragma unroll
    for (int r = 0; r < PV_ROWS; ++r) acc[r] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k0 = 0; k0 < most; k0 += KEYS) {
        __syncthreads();                        // the keys before are done with
        // thread: dims 4 dv .. of keys rv, rv + THREADS / DG, ..; 32-bit pages are copied without passing through registers, the
        // values still on their way while the scores are formed
#pragma unroll
        for (int which = 0; which < 2; ++which) {
#pragma unroll 8
            for (int it = 0; it < KEYS * DG / THREADS; ++it) {
                const int kk = rv + it * (THREADS / DG), j = min(k0 + kk, most - 1);     // (keys beyond: some key's numbers, none looks at them)
                const int page = p.page_shift >= 0 ? j >> p.page_shift : j / p.page_size, at = j - page * p.page_size;
                const T* src = p.cache + (((size_t)bt[page] * 2 + which) * p.n_kv_heads + kvh) * head_block + (size_t)at * d + 4 * dv;
                float* dst = (which ? vs + kk * d : ks + kk * dp) + 4 * dv;
                if (!has_dims) continue;
                if constexpr (sizeof(T) == 4) {
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
                } else {
                    *(float4*)dst = load4(src);
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        {
            float s[PR][PK];
#pragma unroll
            for (int r = 0; r < PR; ++r)
#pragma unroll
                for (int k = 0; k < PK; ++k) s[r][k] = 0.f;
            const float *qr = qs + rq * dp, *kr = ks + kq * dp;
#pragma unroll 2
            for (int c = 0; c < d; c += 4) {
                float4 b[PK];
#pragma unroll
                for (int k = 0; k < PK; ++k) b[k] = *(const float4*)(kr + k * KG * dp + c);
#pragma unroll
                for (int r = 0; r < PR; ++r) {
                    const float4 a = *(const float4*)(qr + r * RG * dp + c);
#pragma unroll
                    for (int k = 0; k < PK; ++k) {
                        s[r][k] = fmaf(a.x, b[k].x, s[r][k]); s[r][k] = fmaf(a.y, b[k].y, s[r][k]);
                        s[r][k] = fmaf(a.z, b[k].z, s[r][k]); s[r][k] = fmaf(a.w, b[k].w, s[r][k]);
                    }
                }
            }
            __syncthreads();
#pragma unroll
            for (int r = 0; r < PR; ++r)
#pragma unroll
                for (int k = 0; k < PK; ++k) ps[(rq + r * RG) * SP + kq + k * KG] = s[r][k];
        }
        __syncthreads();
        if (tid < (LIVE > 16 ? 2 * LIVE : 32)) {             // whole warps
            // A thread takes a row's 32-key step; the sum over its keys is the tree that a warp's exchanges form in the other
            // kernels.  Steps beyond a row's keys leave its numbers as they are.  (With a lane a key and a warp a row this took
            // twice as long as the scores: 9,000 cycles of a stage's 24,000.)
            const int row = tid >> 1, half = tid & 1, n_keys = t.keys_of[row], first = k0 + 32 * half;
            float* pr = ps + row * SP + 32 * half;
            float e[32], top = -INFINITY, scale = p.scale;
            if (p.bias.mul) {                                // apart, so that the loops below stay short
#pragma unroll 1
                for (int i = 0; i < 32; ++i)
                    pr[i] = fmaf(-mul, log1pf(rate * (float)(n_keys - 1 - first - i)), __fmul_rn(pr[i], scale));    // rounded as in the other kernels
                scale = 1.f;
            }
#pragma unroll
            for (int i = 0; i < 32; i += 4) { const float4 v = *(const float4*)(pr + i); e[i] = v.x; e[i + 1] = v.y; e[i + 2] = v.z; e[i + 3] = v.w; }
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                e[i] *= scale;
                if (first + i >= n_keys) e[i] = -INFINITY;
                top = fmaxf(top, e[i]);
            }
            const float m_old = t.m_of[row], l_old = t.l_of[row];
            const float top0 = __shfl_sync(0xffffffffu, top, lane & 30), top1 = __shfl_sync(0xffffffffu, top, lane | 1);
            const float m0 = fmaxf(m_old, top0), m1 = fmaxf(m0, top1), m_before = half ? m0 : m_old, m_new = half ? m1 : m0;
            const float corr = (m_before == -INFINITY) ? 0.f : expf(m_before - m_new);
#pragma unroll
            for (int i = 0; i < 32; ++i) e[i] = (first + i < n_keys) ? expf(e[i] - m_new) : 0.f;
#pragma unroll
            for (int i = 0; i < 32; i += 4) *(float4*)(pr + i) = make_float4(e[i], e[i + 1], e[i + 2], e[i + 3]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int i = 0; i < o; ++i) e[i] += e[i + o];
            const float corr0 = __shfl_sync(0xffffffffu, corr, lane & 30), sum0 = __shfl_sync(0xffffffffu, e[0], lane & 30);
            t.corr_of[half][row] = corr;
            if (half) {
                const float l0 = l_old * corr0 + sum0;
                t.l_of[row] = l0 * corr + e[0];
                t.m_of[row] = m1;
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (has_dims) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int c0 = k0 + 32 * half;
                if (c0 >= most) break;
                const float* vr = vs + 32 * half * d + 4 * dv;
                const float* pr = ps + rv * SP + 32 * half;
#pragma unroll
                for (int r = 0; r < PV_ROWS; ++r) {
                    const float corr = t.corr_of[half][rv + r * RG_V];
                    acc[r].x *= corr; acc[r].y *= corr; acc[r].z *= corr; acc[r].w *= corr;
                }
                if (c0 + 32 <= least) {                      // every row at work sees all 32 keys
#pragma unroll 2
                    for (int jj = 0; jj < 32; jj += 4) {
                        float4 v[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) v[u] = *(const float4*)(vr + (jj + u) * d);
#pragma unroll
                        for (int r = 0; r < PV_ROWS; ++r) {
                            const float4 e = *(const float4*)(pr + r * RG_V * SP + jj);
                            const float w[4] = {e.x, e.y, e.z, e.w};
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                acc[r].x = fmaf(w[u], v[u].x, acc[r].x); acc[r].y = fmaf(w[u], v[u].y, acc[r].y);
                                acc[r].z = fmaf(w[u], v[u].z, acc[r].z); acc[r].w = fmaf(w[u], v[u].w, acc[r].w);
                            }
                        }
                    }
                } else {
#pragma unroll 1
                    for (int jj = 0; jj < 32; jj += 4) {
                        float4 v[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) v[u] = *(const float4*)(vr + (jj + u) * d);
#pragma unroll
                        for (int r = 0; r < PV_ROWS; ++r) {
                            const int cnt = t.keys_of[rv + r * RG_V] - c0 - jj;
                            const float4 e = *(const float4*)(pr + r * RG_V * SP + jj);
                            const float w[4] = {e.x, e.y, e.z, e.w};
#pragma unroll
                            for (int u = 0; u < 4; ++u) {    // a key that the row does not see may hold anything
                                if (u >= cnt) continue;
                                acc[r].x = fmaf(w[u], v[u].x, acc[r].x); acc[r].y = fmaf(w[u], v[u].y, acc[r].y);
                                acc[r].z = fmaf(w[u], v[u].z, acc[r].z); acc[r].w = fmaf(w[u], v[u].w, acc[r].w);
                            }
                        }
                    }
                }
            }
        }
    }
    if (has_dims) {
#pragma unroll
        for (int r = 0; r < PV_ROWS; ++r) {
            const int slot = rv + r * RG_V, row = t.row_at[slot];
            if (row < 0) continue;
            const float inv = 1.0f / t.l_of[slot];
            T* orow = p.out + (size_t)row * p.out_stride + (size_t)h * d + 4 * dv;
            orow[0] = from_float<T>(acc[r].x * inv); orow[1] = from_float<T>(acc[r].y * inv);
            orow[2] = from_float<T>(acc[r].z * inv); orow[3] = from_float<T>(acc[r].w * inv);
        }
    }
}

// The tiles kernel.  Grid (heads, tiles): blocks of like length lie side by side, so the SMs get like shares.  A block takes its tile's
// largest portion, nearly always the tile.
// Of a stage's 17,800 cycles (64 rows, heads of 64, two blocks an SM) the scores take 6,000, the values 5,000, the softmax 3,500 and the
// wait for the keys 3,000; half of the issue slots are used, and the SMs' shares are uneven (256 blocks, 12 to 5 stages long).
template <typename T, int DIMS, int THREADS>
__global__ void __launch_bounds__(THREADS, DIMS == 64 ? 4 : 2)
attention_simt_tiles_kernel(const SimtParams<T> p, int first_tiles, int at_once) {
    extern __shared__ __align__(16) float sm[];
    __shared__ Tile t;
    __shared__ int own_of[2];
    pdl_launch_dependents();
    pdl_wait();
    // The tiles with the most keys first; where all blocks are on the GPU at once, those after the first round of it from the
    // fewest on, so that an SM's blocks add up to like sums.
    const int y = blockIdx.y, tiles = gridDim.y, tid = threadIdx.x;
    const int tile = y < first_tiles || !at_once ? tiles - 1 - y : y - first_tiles;
    load_tile(p, t, tile);
    if (tid < TILE_ROWS) {
        const int own = __reduce_max_sync(0xffffffffu, t.reqs[tid] >= 0 && t.place_of[tid] == 0 ? portion_rank(t.rows_of[tid], tid) : 0);
        if (tid % 32 == 0) own_of[tid / 32] = own;
    }
    __syncthreads();
    const int own = max(own_of[0], own_of[1]);
    if (own) attend_portion<T, DIMS, THREADS, 64>(p, t, sm, tile * TILE_ROWS, portion_first(own), blockIdx.x);
}

// The others kernel: what the tiles' blocks leave, i.e. the smaller portions of tiles with several and the rows that are alone with
// their request in their tile.  Grid (heads, blocks): every block looks all rows over, numbers what it finds and takes every
// gridDim.y-th.  Portions one after the other, in forms for up to 8, 16 and 32 rows (a tile's own is no smaller), then rows, one or
// two at a time.  A portion with a few rows and one stage of keys goes as rows: 128 portions of four rows without a
// past, 16 heads of 128, take 106 us as portions, 52 as rows.
// It runs beside the tiles kernel, from when that one's last block has started.  What both read was there before that one (which was
// launched in order) and they write different rows, so only one block waits for that one's end: a kernel ends after the one ahead.
// (The other way round the tiles' blocks crowd on the SMs that this one's leave first: one portion of 130 tokens 122 us, 64 so.)
// Measured, 32 heads of 64, 32-bit, us, where the tiles' blocks took their other portions one after the other in patches of 64 rows,
// in tiles of 32 rows, so: 256 portions of two tokens behind 300 2,920, 1,100, 700; 64 of eight 785, 392, 196; 11 of 45 270, 235, 122;
// without a past 64 of eight 148, 48, 58, 16 of 32 45, 28, 33.  100 dims: 300 single rows behind 300 1,140, 850, 1,010.
template <typename T, int DIMS, int THREADS>
__global__ void __launch_bounds__(THREADS, DIMS == 64 ? 4 : 2)
attention_simt_others_kernel(const SimtParams<T> p) {
    constexpr int WARPS = THREADS / 32, AT_ONCE = 16, EACH = AT_ONCE / WARPS;     // tiles that are looked over at a time, by a warp
    extern __shared__ __align__(16) float sm[];
    __shared__ Tile t;
    __shared__ int found[AT_ONCE], n_portions, n_rows;
    __shared__ unsigned short mine[AT_ONCE * TILE_ROWS];                          // portions from the front, rows from the back
    pdl_launch_dependents();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = blockIdx.x;
    const bool pairs = DIMS == 128 && p.head_dim <= 104;                          // of rows
    const int few = DIMS == 64 ? 3 : pairs ? 8 : 4;
    int before = 0;                                  // found in the tiles before
    for (int base = 0; base < p.n_tokens; base += AT_ONCE * TILE_ROWS) {          // (all of it the same for every thread)
        int req[EACH][2], is[EACH][2];               // of the lane's two rows of a tile: its request; 1: a row to take, 2: the first of a portion
#pragma unroll
        for (int e = 0; e < EACH; ++e)
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const int n = base + (warp * EACH + e) * TILE_ROWS + 32 * x + lane;
                req[e][x] = n < p.n_tokens ? p.token_request[n] : -1;
            }
        bool any = false;
#pragma unroll
        for (int e = 0; e < EACH; ++e) {
            const int row0 = base + (warp * EACH + e) * TILE_ROWS, a = req[e][0], b = req[e][1], lead = __shfl_sync(0xffffffffu, a, 0);
            is[e][0] = is[e][1] = 0;
            int n_found = 0;
            if (!__all_sync(0xffffffffu, a == lead && b == lead)) {
                const int ka = a >= 0 ? p.positions[row0 + lane] + 1 : 0, kb = b >= 0 ? p.positions[row0 + 32 + lane] + 1 : 0;
                int same_a = 0, same_b = 0, most_a = 0, most_b = 0;
                bool first_a = a >= 0, first_b = b >= 0;
#pragma unroll 4
                for (int i = 0; i < 32; ++i) {
                    const int oa = __shfl_sync(0xffffffffu, a, i), ob = __shfl_sync(0xffffffffu, b, i);
                    const int ja = __shfl_sync(0xffffffffu, ka, i), jb = __shfl_sync(0xffffffffu, kb, i);
                    same_a += (oa == a) + (ob == a); same_b += (oa == b) + (ob == b);
                    most_a = max(most_a, max(oa == a ? ja : 0, ob == a ? jb : 0)); most_b = max(most_b, max(oa == b ? ja : 0, ob == b ? jb : 0));
                    first_a = first_a && !(i < lane && oa == a);
                    first_b = first_b && oa != b && !(i < lane && ob == b);
                }
                const int own = __reduce_max_sync(0xffffffffu, max(first_a ? portion_rank(same_a, lane) : 0, first_b ? portion_rank(same_b, 32 + lane) : 0));
                const int at = portion_first(own), ra = __shfl_sync(0xffffffffu, a, at & 31), rb = __shfl_sync(0xffffffffu, b, at & 31);
                const int own_req = own == 0 ? -1 : at < 32 ? ra : rb;
                auto kind = [&](int r, int same, int most, bool first) {
                    return r < 0 || r == own_req ? 0 : same == 1 || (same <= few && most <= STAGE_KEYS) ? 1 : first ? 2 : 0;
                };
                is[e][0] = kind(a, same_a, most_a, first_a); is[e][1] = kind(b, same_b, most_b, first_b);
                n_found = __popc(__ballot_sync(0xffffffffu, is[e][0])) + __popc(__ballot_sync(0xffffffffu, is[e][1]));
            }
            if (lane == 0) found[warp * EACH + e] = n_found;
            any = any || n_found > 0;
        }
        if (tid == 0) n_portions = n_rows = 0;
        if (!__syncthreads_or(any)) continue;
        int number = before;
        for (int i = 0; i < AT_ONCE; ++i) { before += found[i]; if (i < warp * EACH) number += found[i]; }
#pragma unroll
        for (int e = 0; e < EACH; ++e)
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const unsigned all = __ballot_sync(0xffffffffu, is[e][x]);
                if (is[e][x] && (number + __popc(all & ((1u << lane) - 1))) % gridDim.y == blockIdx.y) {
                    const unsigned short row = (unsigned short)((warp * EACH + e) * TILE_ROWS + 32 * x + lane);
                    if (is[e][x] == 2) mine[atomicAdd(&n_portions, 1)] = row;
                    else mine[AT_ONCE * TILE_ROWS - 1 - atomicAdd(&n_rows, 1)] = row;
                }
                number += __popc(all);
            }
        __syncthreads();
        for (int i = 0; i < n_portions; ++i) {
            const int n = base + mine[i], lead = n % TILE_ROWS;
            load_tile(p, t, n / TILE_ROWS);
            __syncthreads();
            const int rows = t.rows_of[lead];
            if (rows <= 8) attend_portion<T, DIMS, THREADS, 8>(p, t, sm, n - lead, lead, h);
            else if (rows <= 16) attend_portion<T, DIMS, THREADS, 16>(p, t, sm, n - lead, lead, h);
            else attend_portion<T, DIMS, THREADS, 32>(p, t, sm, n - lead, lead, h);
        }
        __syncthreads();
        auto row = [&](int i) { return base + mine[AT_ONCE * TILE_ROWS - 1 - i]; };
        if (pairs) {                                 // two rows at a time (100 dims 0.89 of the time of one; 128 dims 1.2)
            const int part = tid / 128;
            for (int i = part; i < n_rows; i += 2) attend_row<T, 32, 128, false>(p, sm + part * (32 * (2 * p.head_dim + 4) + p.head_dim + 32), row(i), h, part);
        } else {
            for (int i = 0; i < n_rows; ++i) attend_row<T, 64, THREADS>(p, sm, row(i), h);
        }
        __syncthreads();
    }
    if (blockIdx.x == 0 && blockIdx.y == 0) pdl_wait();
}

template <typename T>
int launch_wide(const SimtParams<T>& p, cudaStream_t stream) {
    const int warps = 4;
    const long long pairs = (long long)p.n_tokens * p.n_heads;
    const int blocks = (int)((pairs + warps - 1) / warps);
    const size_t smem = (size_t)warps * p.head_dim * sizeof(float);
#define WIDE(DPL)                                                                                                       \
    return tnx_launch_in_order(attention_simt_wide_kernel<T, DPL>, dim3(blocks), dim3(warps * 32), smem, stream, p.q,   \
                               p.q_stride, p.cache, p.block_tables, p.bt_stride, p.token_request, p.positions, p.out,   \
                               p.out_stride, p.n_tokens, p.n_heads, p.n_kv_heads, p.head_dim, p.page_size, p.window,    \
                               p.scale, p.keep_first, p.bias, p.sink)
    if (p.head_dim <= 256) WIDE(8);
    WIDE(WIDE_DIMS_PER_LANE);
#undef WIDE
}

template <typename T, int KEYS>
int launch_rows(const SimtParams<T>& p, cudaStream_t stream) {
    auto smem_of = [](int d) { return sizeof(float) * (KEYS * (2 * d + 4) + d + KEYS); };
    static TnxSmemLimit limit;
    if (const int rc = limit.allow(attention_simt_rows_kernel<T, KEYS>, smem_of(KEYS == 128 ? 64 : 128))) return rc;
    const size_t smem = smem_of(p.head_dim);
    return tnx_launch_in_order(attention_simt_rows_kernel<T, KEYS>, dim3(p.n_tokens, p.n_heads), dim3(128), smem, stream, p);
}

template <typename T, int DIMS, int THREADS>
int launch_tiles(const SimtParams<T>& p, int sms, cudaStream_t stream) {
    constexpr int KEYS = STAGE_KEYS, PLACES = DIMS == 64 ? 4 : 2;      // blocks an SM
    auto smem_of = [](int rows, int d) { return sizeof(float) * (rows * (d + 4) + KEYS * ((d > KEYS ? d : KEYS) + 4) + KEYS * d); };
    static TnxSmemLimit limit, others_limit;
    if (const int rc = limit.allow(attention_simt_tiles_kernel<T, DIMS, THREADS>, smem_of(TILE_ROWS, DIMS))) return rc;
    if (const int rc = others_limit.allow(attention_simt_others_kernel<T, DIMS, THREADS>, smem_of(32, DIMS))) return rc;
    const size_t smem = smem_of(TILE_ROWS, p.head_dim), others_smem = smem_of(32, p.head_dim);
    const int tiles = (p.n_tokens + TILE_ROWS - 1) / TILE_ROWS;
    int others = PLACES * sms / p.n_heads;
    others = others < 1 ? 1 : others > p.n_tokens ? p.n_tokens : others;
    const int round = (sms + p.n_heads - 1) / p.n_heads, first_tiles = round < tiles ? round : tiles;
    if (const int rc = tnx_launch_in_order(attention_simt_tiles_kernel<T, DIMS, THREADS>, dim3(p.n_heads, tiles), dim3(THREADS), smem, stream, p, first_tiles,
                                           (int)((long long)tiles * p.n_heads <= PLACES * sms))) return rc;
    return tnx_launch_ex(1, attention_simt_others_kernel<T, DIMS, THREADS>, dim3(p.n_heads, others), dim3(THREADS), others_smem, stream, p);
}

// portions: some request may have several rows.  The tiles take them where no mask shifts the 32-key steps of neighbouring
// rows against one another and the rows are enough to give the SMs tiles.
template <typename T>
int launch_all(SimtParams<T> p, int portions, int sms, cudaStream_t stream) {
    const bool staged = p.head_dim % 4 == 0 && p.head_dim <= 128 && (uintptr_t)p.cache % (4 * sizeof(T)) == 0 && p.n_heads <= 65535;
    if (!staged) return launch_wide<T>(p, stream);
    if (portions && p.window == 0 && (long long)p.n_tokens * p.n_heads >= 2048 && p.n_tokens <= 2000000)      // (a grid's second axis)
        return p.head_dim <= 64 ? launch_tiles<T, 64, 128>(p, sms, stream) : launch_tiles<T, 128, 256>(p, sms, stream);
    return p.head_dim <= 64 ? launch_rows<T, 128>(p, stream) : launch_rows<T, 64>(p, stream);
}
}  // namespace

// portions: 0 where every request of the batch has one row (the rows kernel alone), else 1; sms: how many the device has.
TNX_EXPORT int tnx_attention_simt(const void* q, int q_stride, const void* cache, const int* block_tables,
                                  int bt_stride, const int* token_request, const int* positions, void* out,
                                  int out_stride, int n_tokens, int n_heads, int n_kv_heads, int head_dim,
                                  int page_size, int window, float scale, int keep_first, const float* bias_mul,
                                  const float* bias_rate, int has_sink, float sink_score, int is_h16, int portions, int sms,
                                  cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (head_dim <= 0 || head_dim > 32 * WIDE_DIMS_PER_LANE || n_kv_heads <= 0 || n_heads % n_kv_heads)
        return TNX_ERR_UNSUPPORTED;
    if (keep_first < 0 || (bias_mul && !bias_rate) || sms <= 0) return TNX_ERR_BAD_ARG;
    const DistanceBias bias{bias_mul, bias_rate};
    const SoftmaxSink sink{has_sink, sink_score};
    int page_shift = -1;
    for (int i = 0; i < 31; ++i) if (page_size == 1 << i) page_shift = i;
#define ASIMT(T)                                                                                                        \
    return launch_all<T>(SimtParams<T>{(const T*)q, q_stride, (const T*)cache, block_tables, bt_stride, token_request,  \
                                       positions, (T*)out, out_stride, n_tokens, n_heads, n_kv_heads, head_dim,         \
                                       page_size, window, scale, keep_first, bias, sink, page_shift}, portions, sms, stream)
    if (is_h16) ASIMT(h16);
    ASIMT(float);
#undef ASIMT
}
