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
//   tiles   for portions of prompts without a mask: a block takes 32 neighbouring rows and one head, 64 staged keys and
//           values serve all of them
// Measured, 32 heads of 64, 32-bit: a portion of 499 tokens behind 256 beside three single rows of 500 to 700 keys, 2,417 us
// with `wide` for all rows, 1,200 with `rows`, 279 with `tiles` and `rows`; four single rows of 100 to 900 keys 382 us with
// `wide`, 53 with `rows`; 64 of 100 to 1,360 keys 1,106 and 434; a portion of 2,048 tokens, 16 heads of 128, 17.2 and 1.66 ms.
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
    int tiled;                           // the tiles kernel takes the rows that share their request within a tile
};

constexpr int TILE_ROWS = 32;            // rows of a tile: tile t holds rows 32 t .. 32 t + 31 of the batch

__device__ __forceinline__ float4 load4(const float* p) { return *(const float4*)p; }
__device__ __forceinline__ float4 load4(const h16* p) {
    const uint2 raw = *(const uint2*)p;
    const float2 a = h16x2_to_float2(*(const h16x2*)&raw.x), b = h16x2_to_float2(*(const h16x2*)&raw.y);
    return make_float4(a.x, a.y, b.x, b.y);
}

// The rows kernel: 128 threads a (row, head).  With `tiled`, blockIdx.x names a tile and one of its SLOTS: the block takes
// every SLOTS-th of the rows that are alone with their request in that tile, which the tiles kernel leaves.
constexpr int SLOTS = 8;
template <typename T, int KEYS>
__global__ void __launch_bounds__(128)
attention_simt_rows_kernel(const SimtParams<T> p) {
    extern __shared__ __align__(16) float sm[];
    const int d = p.head_dim, d4 = d / 4;
    float* ks = sm;                                 // [KEYS][d + 4]: a warp's 16-byte reads down the rows meet all banks evenly
    float* vs = ks + KEYS * (d + 4);                // [KEYS][d]
    float* qs = vs + KEYS * d;                      // [d]
    float* ss = qs + d;                             // [KEYS] the staged keys' scores
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31;
    const int h = blockIdx.y, kvh = h / (p.n_heads / p.n_kv_heads);
    const size_t head_block = (size_t)p.page_size * d;
    const float mul = p.bias.mul ? p.bias.mul[h] : 0.f, rate = p.bias.mul ? p.bias.rate[h] : 0.f;
    unsigned todo = 1;                              // bit r: row row0 + r is still to do (the same in every thread)
    int row0 = blockIdx.x;
    if (p.tiled) {
        row0 = blockIdx.x / SLOTS * TILE_ROWS;
        const int mine = row0 + lane < p.n_tokens ? p.token_request[row0 + lane] : -1;
        bool alone = mine >= 0;
        for (int i = 0; i < TILE_ROWS; ++i) {
            const int other = __shfl_sync(0xffffffffu, mine, i);
            alone = alone && (i == lane || other != mine);
        }
        todo = __ballot_sync(0xffffffffu, alone);
        const int place = __popc(todo & ((1u << lane) - 1));
        todo = __ballot_sync(0xffffffffu, alone && place % SLOTS == (int)blockIdx.x % SLOTS);
    }
    for (; todo; todo &= todo - 1) {
        const int n = row0 + __ffs(todo) - 1;
        const int req = p.token_request[n];
        if (req < 0) continue;                      // a padded row of a captured batch
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
            __syncthreads();                        // the keys before are done with
            if (k0 == 0)
                for (int c = tid; c < d; c += 128) qs[c] = to_float(p.q[(size_t)n * p.q_stride + (size_t)h * d + c]);
#pragma unroll 8
            for (int i = tid; i < staged * d4; i += 128) {
                const int kk = i / d4, c = (i % d4) * 4, i_key = k0 + kk, j = i_key < kept ? i_key : i_key + gap;
                const T* krow = p.cache + ((size_t)bt[j / p.page_size] * 2 * p.n_kv_heads + kvh) * head_block
                                + (size_t)(j % p.page_size) * d + c;
                *(float4*)(ks + kk * (d + 4) + c) = load4(krow);
                *(float4*)(vs + kk * d + c) = load4(krow + (size_t)p.n_kv_heads * head_block);
            }
            __syncthreads();
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
            __syncthreads();
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
}

// The tiles kernel.  Grid (tiles, heads), four warps of eight rows.  The requests that have two rows and more in the tile
// are taken one after the other (nearly always there is one); rows of other requests idle meanwhile.
//   scores   a lane owns keys `lane` and `lane + 32` of the 64 staged, the row's q comes as a broadcast: two 16-byte
//            shared-memory reads of keys and eight of q feed 64 multiply-adds
//   values   a lane owns dims lane, lane + 32, ..; the row's probabilities come as a broadcast
// It is bound by those reads (16 bytes a thread take a warp four cycles, broadcast or not).  A row's own 32-key steps
// (maximum, sum, rescaling) are those of the other kernels.
template <typename T, int DPL>
__global__ void __launch_bounds__(128)
attention_simt_tiles_kernel(const SimtParams<T> p) {
    constexpr int KEYS = 64, RPW = TILE_ROWS / 4;
    extern __shared__ __align__(16) float sm[];
    const int d = p.head_dim;
    float* qs = sm;                                 // [TILE_ROWS][d]
    float* ks = qs + TILE_ROWS * d;                 // [KEYS][d + 4]
    float* vs = ks + KEYS * (d + 4);                // [KEYS][d]
    float* ps = vs + KEYS * d;                      // [TILE_ROWS][32]
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * TILE_ROWS, h = blockIdx.y;     // later rows have more keys: first
    const int kvh = h / (p.n_heads / p.n_kv_heads);
    const int my_n = row0 + lane;
    const int my_req = my_n < p.n_tokens ? p.token_request[my_n] : -1;
    const int my_pos = my_n < p.n_tokens ? p.positions[my_n] : 0;
    const size_t head_block = (size_t)p.page_size * d;
    const float mul = p.bias.mul ? p.bias.mul[h] : 0.f, rate = p.bias.mul ? p.bias.rate[h] : 0.f;
    const int d4 = d / 4;
    unsigned todo = __ballot_sync(0xffffffffu, my_req >= 0);
    while (todo) {                                  // the same for every warp of the block
        const int lead = __ffs(todo) - 1;
        const int req = __shfl_sync(0xffffffffu, my_req, lead);
        const unsigned mine = __ballot_sync(0xffffffffu, my_req == req);
        todo &= ~mine;
        if (!(mine & (mine - 1))) continue;         // a request's only row here: the rows kernel's
        int most = my_req == req ? my_pos + 1 : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
        const int* bt = p.block_tables + (size_t)req * p.bt_stride;
        __syncthreads();                            // the request before is done with q
        for (int i = tid; i < TILE_ROWS * d4; i += 128) {
            const int r = i / d4, c = (i % d4) * 4;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (mine >> r & 1) {
                const T* src = p.q + (size_t)(row0 + r) * p.q_stride + (size_t)h * d + c;
                v = make_float4(to_float(src[0]), to_float(src[1]), to_float(src[2]), to_float(src[3]));
            }
            *(float4*)(qs + r * d + c) = v;
        }
        float m[RPW], l[RPW], acc[RPW][DPL];
        int n_keys[RPW];
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
            const int row = warp * RPW + r, at = __shfl_sync(0xffffffffu, my_pos, row);
            n_keys[r] = (mine >> row & 1) ? at + 1 : 0;
            m[r] = p.sink.on ? p.sink.score : -INFINITY; l[r] = p.sink.on ? 1.f : 0.f;
#pragma unroll
            for (int i = 0; i < DPL; ++i) acc[r][i] = 0.f;
        }
        int warp_keys = 0;
#pragma unroll
        for (int r = 0; r < RPW; ++r) warp_keys = max(warp_keys, n_keys[r]);
        for (int k0 = 0; k0 < most; k0 += KEYS) {
            __syncthreads();                        // the keys before are done with
            for (int i = tid; i < KEYS * d4; i += 128) {
                const int kk = i / d4, c = (i % d4) * 4, j = k0 + kk;
                float4 k4 = make_float4(0.f, 0.f, 0.f, 0.f), v4 = k4;
                if (j < most) {
                    const T* krow = p.cache + ((size_t)bt[j / p.page_size] * 2 * p.n_kv_heads + kvh) * head_block
                                    + (size_t)(j % p.page_size) * d + c;
                    k4 = load4(krow);
                    v4 = load4(krow + (size_t)p.n_kv_heads * head_block);
                }
                *(float4*)(ks + kk * (d + 4) + c) = k4;
                *(float4*)(vs + kk * d + c) = v4;
            }
            __syncthreads();
            if (k0 >= warp_keys) continue;
            float s0[RPW], s1[RPW];
#pragma unroll
            for (int r = 0; r < RPW; ++r) s0[r] = s1[r] = 0.f;
            const float *ka = ks + lane * (d + 4), *kb = ka + 32 * (d + 4), *qw = qs + warp * RPW * d;
#pragma unroll 2
            for (int c = 0; c < d; c += 4) {
                const float4 a = *(const float4*)(ka + c), b = *(const float4*)(kb + c);
#pragma unroll
                for (int r = 0; r < RPW; ++r) {
                    const float4 q = *(const float4*)(qw + r * d + c);
                    s0[r] = fmaf(q.x, a.x, s0[r]); s0[r] = fmaf(q.y, a.y, s0[r]);
                    s0[r] = fmaf(q.z, a.z, s0[r]); s0[r] = fmaf(q.w, a.w, s0[r]);
                    s1[r] = fmaf(q.x, b.x, s1[r]); s1[r] = fmaf(q.y, b.y, s1[r]);
                    s1[r] = fmaf(q.z, b.z, s1[r]); s1[r] = fmaf(q.w, b.w, s1[r]);
                }
            }
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int c0 = k0 + 32 * half, i = c0 + lane;
                bool whole = true;                  // every row of the warp that is at work sees all 32 keys
#pragma unroll
                for (int r = 0; r < RPW; ++r) {
                    const int cnt = n_keys[r] - c0;
                    whole = whole && (cnt >= 32 || n_keys[r] == 0);
                    if (cnt <= 0) continue;         // the same for the whole warp
                    float s = (half ? s1[r] : s0[r]) * p.scale;
                    if (p.bias.mul) s -= mul * log1pf(rate * (float)(n_keys[r] - 1 - i));
                    if (i >= n_keys[r]) s = -INFINITY;
                    const float m_new = fmaxf(m[r], warp_max(s));
                    const float e = (i < n_keys[r]) ? expf(s - m_new) : 0.f;
                    const float corr = (m[r] == -INFINITY) ? 0.f : expf(m[r] - m_new);
                    l[r] = l[r] * corr + warp_sum(e);
                    m[r] = m_new;
#pragma unroll
                    for (int x = 0; x < DPL; ++x) acc[r][x] *= corr;
                    ps[(warp * RPW + r) * 32 + lane] = e;
                }
                __syncwarp();
                const float* vrow = vs + 32 * half * d + lane;
                if (whole && c0 < warp_keys) {
                    for (int jj = 0; jj < 32; jj += 4) {
                        float v[4][DPL];
#pragma unroll
                        for (int u = 0; u < 4; ++u)
#pragma unroll
                            for (int x = 0; x < DPL; ++x) v[u][x] = lane + 32 * x < d ? vrow[(jj + u) * d + 32 * x] : 0.f;
#pragma unroll
                        for (int r = 0; r < RPW; ++r) {
                            if (n_keys[r] == 0) continue;
                            const float4 e = *(const float4*)(ps + (warp * RPW + r) * 32 + jj);
#pragma unroll
                            for (int x = 0; x < DPL; ++x) {
                                acc[r][x] = fmaf(e.x, v[0][x], acc[r][x]); acc[r][x] = fmaf(e.y, v[1][x], acc[r][x]);
                                acc[r][x] = fmaf(e.z, v[2][x], acc[r][x]); acc[r][x] = fmaf(e.w, v[3][x], acc[r][x]);
                            }
                        }
                    }
                } else {
#pragma unroll
                    for (int r = 0; r < RPW; ++r) {
                        const int cnt = min(32, n_keys[r] - c0);
                        for (int jj = 0; jj < cnt; ++jj) {
                            const float e = ps[(warp * RPW + r) * 32 + jj];
#pragma unroll
                            for (int x = 0; x < DPL; ++x)
                                if (lane + 32 * x < d) acc[r][x] = fmaf(e, vrow[jj * d + 32 * x], acc[r][x]);
                        }
                    }
                }
                __syncwarp();
            }
        }
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
            if (n_keys[r] == 0) continue;
            const float inv = 1.0f / l[r];
            T* orow = p.out + (size_t)(row0 + warp * RPW + r) * p.out_stride + (size_t)h * d;
#pragma unroll
            for (int x = 0; x < DPL; ++x)
                if (lane + 32 * x < d) orow[lane + 32 * x] = from_float<T>(acc[r][x] * inv);
        }
    }
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

template <typename K>
int allow_smem(K kernel, size_t smem) {
    if (smem <= 48 * 1024) return 0;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) cudaGetLastError();
    return (int)e;
}

template <typename T, int KEYS>
int launch_rows(const SimtParams<T>& p, cudaStream_t stream) {
    const size_t smem = sizeof(float) * (KEYS * (2 * p.head_dim + 4) + p.head_dim + KEYS);
    if (const int rc = allow_smem(attention_simt_rows_kernel<T, KEYS>, smem)) return rc;
    const int blocks = p.tiled ? (p.n_tokens + TILE_ROWS - 1) / TILE_ROWS * SLOTS : p.n_tokens;
    return tnx_launch_in_order(attention_simt_rows_kernel<T, KEYS>, dim3(blocks, p.n_heads), dim3(128), smem, stream, p);
}

template <typename T, int DPL>
int launch_tiles(const SimtParams<T>& p, cudaStream_t stream) {
    const size_t smem = sizeof(float) * (TILE_ROWS * p.head_dim + 64 * (2 * p.head_dim + 4) + TILE_ROWS * 32);
    if (const int rc = allow_smem(attention_simt_tiles_kernel<T, DPL>, smem)) return rc;
    return tnx_launch_in_order(attention_simt_tiles_kernel<T, DPL>, dim3((p.n_tokens + TILE_ROWS - 1) / TILE_ROWS, p.n_heads), dim3(128), smem, stream, p);
}

// portions: some request may have several rows.  The tiles take them where no mask shifts the 32-key steps of neighbouring
// rows against one another and the rows are enough to give the SMs tiles (64 rows of 16 heads: 24 us row by row, 33 in
// tiles; 140 rows of 2 heads: 19 and 53); the rows kernel follows for those that are alone in their tile.
template <typename T>
int launch_all(SimtParams<T> p, int portions, cudaStream_t stream) {
    const bool staged = p.head_dim % 4 == 0 && p.head_dim <= 128 && (uintptr_t)p.cache % (4 * sizeof(T)) == 0 && p.n_heads <= 65535;
    if (!staged) return launch_wide<T>(p, stream);
    p.tiled = portions && p.window == 0 && (long long)p.n_tokens * p.n_heads >= 2048;
    if (p.tiled) {
        const int rc = p.head_dim <= 32 ? launch_tiles<T, 1>(p, stream) : p.head_dim <= 64 ? launch_tiles<T, 2>(p, stream)
                                                                        : launch_tiles<T, 4>(p, stream);
        if (rc) return rc;
    }
    return p.head_dim <= 64 ? launch_rows<T, 128>(p, stream) : launch_rows<T, 64>(p, stream);
}
}  // namespace

// portions: 0 where every request of the batch has one row (the rows kernel alone), else 1.
TNX_EXPORT int tnx_attention_simt(const void* q, int q_stride, const void* cache, const int* block_tables,
                                  int bt_stride, const int* token_request, const int* positions, void* out,
                                  int out_stride, int n_tokens, int n_heads, int n_kv_heads, int head_dim,
                                  int page_size, int window, float scale, int keep_first, const float* bias_mul,
                                  const float* bias_rate, int has_sink, float sink_score, int is_h16, int portions,
                                  cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (head_dim <= 0 || head_dim > 32 * WIDE_DIMS_PER_LANE || n_kv_heads <= 0 || n_heads % n_kv_heads)
        return TNX_ERR_UNSUPPORTED;
    if (keep_first < 0 || (bias_mul && !bias_rate)) return TNX_ERR_BAD_ARG;
    const DistanceBias bias{bias_mul, bias_rate};
    const SoftmaxSink sink{has_sink, sink_score};
#define ASIMT(T)                                                                                                        \
    return launch_all<T>(SimtParams<T>{(const T*)q, q_stride, (const T*)cache, block_tables, bt_stride, token_request,  \
                                       positions, (T*)out, out_stride, n_tokens, n_heads, n_kv_heads, head_dim,         \
                                       page_size, window, scale, keep_first, bias, sink, 0}, portions, stream)
    if (is_h16) ASIMT(h16);
    ASIMT(float);
#undef ASIMT
}
