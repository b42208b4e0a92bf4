// Matrix product on CUDA cores with 32-bit FMA accumulation: the true 32-bit path (no tensor
// cores, no reduced-precision mode), and the path for sizes that the tensor-core kernel refuses.
//
//   C[m, n] = epilogue( sum_k A[m, k] * W[n, k] )           A: [M, K], W: [N, K] (both row-major)
//   epilogue: + bias[n]; activation (by code, common.cuh); + residual[m, n] (32-bit); stored as float or in the 16-bit type.
//
// Every output element adds its products in ascending k with one accumulator, so a row's result
// does not depend on which other rows are in the call.
#include "common.cuh"

namespace {

// Every thread owns a patch of TM x TN outputs; a K block of BK is staged k-major in shared memory, double-buffered, the
// next block's 16- or 8-byte loads in flight (in registers) while the current one is used, and neighbouring outputs of a
// row are multiplied two at a time (fma.rn.f32x2: two ordinary 32-bit FMAs in one instruction; 2,048 tokens by
// [8192 x 2048] 1,470 us with it, 1,780 without).
// What bounds it: with patches of 8 x 8 a warp's reads of shared memory (16 bytes a thread take it four cycles) last as long
// as its multiplications, so 48 TFLOP/s is what large products reach of 74; with few tiles it is the latency of one block's
// K loop.  Patches of 16 x 8 (252 registers, four warps an SM) reached 43; every element of A twice in shared memory, to
// spare the register moves that pair it, 39: the reads are the bound.
// Measured at 502 tokens, 16-bit weights, against tiles of 64 x 64 with patches of 4 x 4, scalar loads and one buffer:
// [6144 x 2048] 582 -> 339 us, [2048 x 2048] 245 -> 145, [8192 x 2048] 827 -> 422, [2048 x 8192] 953 -> 556; one token by
// [2048 x 2048] 156 -> 60.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d)
        : "l"(*(const unsigned long long*)&a), "l"(*(const unsigned long long*)&b), "l"(*(const unsigned long long*)&c));
    return *(float2*)&d;
}

// Four neighbouring elements of a row as floats; zeros beyond the row's K elements.  vec: rows start on 4-element boundaries.
template <typename T> __device__ __forceinline__ float4 load4(const T* row, int k, int K, bool vec);
template <> __device__ __forceinline__ float4 load4<float>(const float* row, int k, int K, bool vec) {
    if (vec && k + 4 <= K) return __ldg((const float4*)(row + k));
    float4 v;
    v.x = k < K ? row[k] : 0.f; v.y = k + 1 < K ? row[k + 1] : 0.f;
    v.z = k + 2 < K ? row[k + 2] : 0.f; v.w = k + 3 < K ? row[k + 3] : 0.f;
    return v;
}
template <> __device__ __forceinline__ float4 load4<h16>(const h16* row, int k, int K, bool vec) {
    float4 v;
    if (vec && k + 4 <= K) {
        const uint2 raw = __ldg((const uint2*)(row + k));
        const float2 a = h16x2_to_float2(*(const h16x2*)&raw.x), b = h16x2_to_float2(*(const h16x2*)&raw.y);
        return make_float4(a.x, a.y, b.x, b.y);
    }
    v.x = k < K ? to_float(row[k]) : 0.f; v.y = k + 1 < K ? to_float(row[k + 1]) : 0.f;
    v.z = k + 2 < K ? to_float(row[k + 2]) : 0.f; v.w = k + 3 < K ? to_float(row[k + 3]) : 0.f;
    return v;
}

// A thread's patch: rows in groups of GM = min(TM, 4) neighbours every BM / (TM / GM) rows, columns likewise.
template <typename TA, typename TW, typename TO, int BM, int BN, int BK, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), TM * TN == 64 ? 3 : 4)
gemm_simt_kernel(const TA* __restrict__ A, const TW* __restrict__ W, const float* __restrict__ bias,
                 const float* residual, TO* C, int M, int N, int K, int lda, int ldw, int ldc,
                 int act, int vec_a, int vec_w) {
    constexpr int THREADS = (BM / TM) * (BN / TN);
    constexpr int GM = TM < 4 ? TM : 4, GN = TN < 4 ? TN : 4;
    constexpr int CPR = BK / 4;                              // 4-element pieces of a row's K block
    constexpr int LA = BM * CPR / THREADS, LW = BN * CPR / THREADS;
    static_assert(LA * THREADS == BM * CPR && LW * THREADS == BN * CPR, "the loaders share the K block evenly");
    __shared__ __align__(16) float As[2][BK][BM + 4];
    __shared__ __align__(16) float Ws[2][BK][BN + 4];
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tx = tid % (BN / TN), ty = tid / (BN / TN);
    float2 acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = make_float2(0.f, 0.f);

    float4 ra[LA], rw[LW];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < LA; ++i) {
            const int c = tid + i * THREADS, row = m0 + c / CPR, k = k0 + (c % CPR) * 4;
            ra[i] = row < M ? load4<TA>(A + (size_t)row * lda, k, K, vec_a) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < LW; ++i) {
            const int c = tid + i * THREADS, row = n0 + c / CPR, k = k0 + (c % CPR) * 4;
            rw[i] = row < N ? load4<TW>(W + (size_t)row * ldw, k, K, vec_w) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    auto put = [&](int b) {
#pragma unroll
        for (int i = 0; i < LA; ++i) {
            const int c = tid + i * THREADS, row = c / CPR, k = (c % CPR) * 4;
            As[b][k][row] = ra[i].x; As[b][k + 1][row] = ra[i].y; As[b][k + 2][row] = ra[i].z; As[b][k + 3][row] = ra[i].w;
        }
#pragma unroll
        for (int i = 0; i < LW; ++i) {
            const int c = tid + i * THREADS, row = c / CPR, k = (c % CPR) * 4;
            Ws[b][k][row] = rw[i].x; Ws[b][k + 1][row] = rw[i].y; Ws[b][k + 2][row] = rw[i].z; Ws[b][k + 3][row] = rw[i].w;
        }
    };
    fetch(0);
    put(0);
    __syncthreads();
    int b = 0;
    for (int k0 = 0; k0 < K; k0 += BK, b ^= 1) {
        const bool more = k0 + BK < K;
        if (more) fetch(k0 + BK);
#pragma unroll 16
        for (int kk = 0; kk < BK; ++kk) {
            float a[TM];
            float2 w[TN / 2];
#pragma unroll
            for (int g = 0; g < TM / GM; ++g) {
                const float* src = &As[b][kk][g * (BM / (TM / GM)) + ty * GM];
                if constexpr (GM == 4) {
                    const float4 v = *(const float4*)src;
                    a[g * 4] = v.x; a[g * 4 + 1] = v.y; a[g * 4 + 2] = v.z; a[g * 4 + 3] = v.w;
                } else {
#pragma unroll
                    for (int e = 0; e < GM; ++e) a[g * GM + e] = src[e];
                }
            }
#pragma unroll
            for (int g = 0; g < TN / GN; ++g) {
                const float* src = &Ws[b][kk][g * (BN / (TN / GN)) + tx * GN];
                if constexpr (GN == 4) {
                    const float4 v = *(const float4*)src;
                    w[g * 2] = make_float2(v.x, v.y); w[g * 2 + 1] = make_float2(v.z, v.w);
                } else {
                    w[g] = *(const float2*)src;
                }
            }
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) acc[i][j] = fma2(make_float2(a[i], a[i]), w[j], acc[i][j]);
        }
        if (more) {
            put(b ^ 1);                                      // its last readers passed the barrier of the block before
            __syncthreads();
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + (i / GM) * (BM / (TM / GM)) + ty * GM + i % GM;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + (j / GN) * (BN / (TN / GN)) + tx * GN + j % GN;
            if (n >= N) continue;
            float v = j % 2 ? acc[i][j / 2].y : acc[i][j / 2].x;
            if (bias) v += bias[n];
            v = apply_activation(v, act);
            if (residual) v += residual[(size_t)m * ldc + n];
            C[(size_t)m * ldc + n] = from_float<TO>(v);
        }
    }
}

template <typename T> bool rows_on_4_elements(const void* p, int ld) {
    return ld % 4 == 0 && (uintptr_t)p % (4 * sizeof(T)) == 0;
}

template <typename TA, typename TW, typename TO, int BM, int BN, int BK, int TM, int TN>
int launch_tile(const void* A, const void* W, const float* bias, const float* residual, void* C, int M,
                int N, int K, int lda, int ldw, int ldc, int act, cudaStream_t stream) {
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    return tnx_launch_in_order(gemm_simt_kernel<TA, TW, TO, BM, BN, BK, TM, TN>, grid, dim3((BM / TM) * (BN / TN)), 0, stream,
                               (const TA*)A, (const TW*)W, bias, residual, (TO*)C, M, N, K, lda, ldw, ldc, act,
                               (int)rows_on_4_elements<TA>(A, lda), (int)rows_on_4_elements<TW>(W, ldw));
}

// The tile.  Up to 16 tokens: 16 x 32 with a deep K block (its blocks are the most, and the time is the weights').
// Otherwise the one that the busiest SM is estimated to be done with first.  The estimates are for K = 2,048 (all are
// proportional to K), fitted to 8 .. 2,048 tokens by 2,048 .. 8,192 features: n tiles an SM take no less than the latency of
// one K loop and a little more for each further tile, and no less than the SM's rate allows.
//   128 x 64, patches of 8 x 8:  n = 1, 2, 3, 4, 14 measured 178, 248, 339, 450, 1437 us
//   64 x 64,  patches of 8 x 4:  n = 1, 2, 3, 6, 28 measured 126, 144, 201, 363, 1568 us
//   64 x 32,  patches of 4 x 4:  n = 1, 2, 3, 4     measured  82, 104, 142, 185 us
template <typename TA, typename TW, typename TO>
int launch(const void* A, const void* W, const float* bias, const float* residual, void* C, int M,
           int N, int K, int lda, int ldw, int ldc, int act, cudaStream_t stream) {
    constexpr int SMS = 148;
    auto tiles = [&](int bm, int bn) { return (int)((((long long)N + bn - 1) / bn * (((long long)M + bm - 1) / bm) + SMS - 1) / SMS); };
    auto most = [](double a, double b) { return a > b ? a : b; };
    const int n1 = tiles(128, 64), n2 = tiles(64, 64), n3 = tiles(64, 32);
    const double t1 = most(178. + 70. * (n1 - 1), 105. * n1), t2 = most(126. + 18. * (n2 - 1), 20. + 57. * n2),
                 t3 = most(82. + 22. * (n3 - 1), 5. + 45. * n3);
    if (M <= 16) return launch_tile<TA, TW, TO, 16, 32, 64, 2, 2>(A, W, bias, residual, C, M, N, K, lda, ldw, ldc, act, stream);
    if (t3 <= t1 && t3 <= t2)
        return launch_tile<TA, TW, TO, 64, 32, 32, 4, 4>(A, W, bias, residual, C, M, N, K, lda, ldw, ldc, act, stream);
    if (t2 <= t1)
        return launch_tile<TA, TW, TO, 64, 64, 16, 8, 4>(A, W, bias, residual, C, M, N, K, lda, ldw, ldc, act, stream);
    return launch_tile<TA, TW, TO, 128, 64, 16, 8, 8>(A, W, bias, residual, C, M, N, K, lda, ldw, ldc, act, stream);
}

}  // namespace

// a_h16 / w_h16 / c_h16: element types (1 = bfloat16, 0 = float).  residual (32-bit, same
// leading dimension as C) may alias C when C is float.
TNX_EXPORT int tnx_gemm_simt(const void* A, const void* W, const float* bias, const float* residual,
                             void* C, int M, int N, int K, int lda, int ldw, int ldc, int act,
                             int a_h16, int w_h16, int c_h16, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || lda < K || ldw < K || ldc < N) return TNX_ERR_BAD_ARG;
    if (residual && c_h16) return TNX_ERR_BAD_ARG;
    if (act < 0 || act >= TNX_ACT_COUNT) return TNX_ERR_BAD_ARG;
    const int code = (a_h16 ? 4 : 0) | (w_h16 ? 2 : 0) | (c_h16 ? 1 : 0);
    switch (code) {
        case 0: return launch<float, float, float>(A, W, bias, residual, C, M, N, K, lda, ldw, ldc, act, stream);
        case 2: return launch<float, h16, float>(A, W, bias, residual, C, M, N, K, lda, ldw, ldc, act, stream);
        case 4: return launch<h16, float, float>(A, W, bias, residual, C, M, N, K, lda, ldw, ldc, act, stream);
        case 5: return launch<h16, float, h16>(A, W, bias, residual, C, M, N, K, lda, ldw, ldc, act, stream);
        case 6: return launch<h16, h16, float>(A, W, bias, residual, C, M, N, K, lda, ldw, ldc, act, stream);
        case 7: return launch<h16, h16, h16>(A, W, bias, residual, C, M, N, K, lda, ldw, ldc, act, stream);
        default: return TNX_ERR_UNSUPPORTED;
    }
}
