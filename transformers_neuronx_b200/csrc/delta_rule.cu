// A recurrence with an error-correcting write ("delta rule") and a decay per head and key channel.  Per head, with
// q_t, k_t of k_dim numbers, v_t of v_dim numbers and a state S of k_dim x v_dim (32-bit, kept per request):
//     S <- diag(g_t) S;   u = beta_t (v_t - S^T k_t);   S <- S + k_t u^T;   o_t = S^T q_t
// so the read-out sees the current token's write.  Query/key heads may be shared by groups of heads (G of them for H
// heads: head h uses q/k head h / (H / G)).
//
// tnx_delta_prep, per token (one thread block for a prompt's tokens; several for the few tokens of a decode step, which
//   share the token's heads and channels, so that eight tokens still fill the device): from the projections' output
//   (queries, keys and values side by side from column col0 on: G*dk, G*dk, H*dv channels)
//     y_t[c] = act(sum_j w[j, c] u_(t - taps + 1 + j)[c])        the short causal convolution (zeros before position 0;
//                                                                 the past comes from this step's rows or from the
//                                                                 request's state [slots, taps - 1, channels])
//     q, k per head: y / sqrt(sum(y^2) + unit_eps), q times q_scale;  v = y
//     beta[h] = sigmoid(proj[b_off + h]);   g[h, i] = exp(-exp(a_log[h]) * softplus(a[h * dk + i] + dt_bias[h * dk + i]))
//   Everything after the loads is 32-bit and stays 32-bit: q, k, v, beta and g are written as floats.  A request with
//   one row shifts its convolution state here; requests with several rows are brought up to date by the convolution
//   library's state kernel afterwards.
// tnx_delta_scan: a thread block owns C columns (value dims) of one head of one request and walks the request's tokens
//   of this step in order, the state's columns in registers: a column's k_dim rows are spread over R adjacent lanes,
//   which add their partial sums of S^T k, S^T q and q.k with shuffles (o = (gS)^T q + (q.k) u).
//   The tokens' inputs reach shared memory by asynchronous copies, a stage ahead of the walk.
//   The state is stored [slot, head, v_dim, k_dim] (a column's rows side by side).
#include "common.cuh"

namespace {

constexpr int PREP_MAX_TAPS = 8;
constexpr int PREP_FILL_BLOCKS = 2 * 148;   // blocks that fill the device: two an SM

__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(expf(x)); }

template <typename T>
__global__ void __launch_bounds__(256)
delta_prep_kernel(const T* __restrict__ proj, int ld, int col0, int b_off, const float* __restrict__ a, int a_ld,
                  const float* __restrict__ conv_w, int taps, T* state, const int* __restrict__ token_request,
                  const int* __restrict__ positions, const int* __restrict__ q_start, const int* __restrict__ q_len,
                  const int* __restrict__ state_slots, const float* __restrict__ a_log, const float* __restrict__ dt_bias,
                  float unit_eps, float q_scale, int act, float* __restrict__ q_out, float* __restrict__ k_out,
                  float* __restrict__ v_out, float* __restrict__ beta_out, float* __restrict__ g_out, int H, int G, int dk,
                  int dv) {
    extern __shared__ float y[];                      // a query or key head's convolved channels, per warp
    pdl_launch_dependents();
    pdl_wait();
    const int n = blockIdx.x;
    const int req = token_request[n];
    if (req < 0) return;                              // a padded row of a captured step
    const int pos = positions[n], idx = n - q_start[req], slot = state_slots[req];
    const bool alone = q_len[req] == 1;
    const int keep = taps - 1, nqk = 2 * G * dk, C = nqk + H * dv;
    const T* row = proj + (size_t)n * ld + col0;
    T* st = (keep > 0 && slot >= 0) ? state + (size_t)slot * keep * C : nullptr;
    auto conv = [&](int c) -> float {                 // channel c of this token: convolution, state shift, activation
        float past[PREP_MAX_TAPS];                    // past[b]: the projected value b positions back
        past[0] = to_float(row[c]);
        for (int b = 1; b < taps; ++b) {
            float v = 0.f;
            if (pos - b >= 0) {
                if (idx - b >= 0) v = to_float(row[c - (ptrdiff_t)b * ld]);
                else if (st) v = to_float(st[(size_t)(keep + idx - b) * C + c]);
            }
            past[b] = v;
        }
        float s = 0.f;
        for (int j = 0; j < taps; ++j) s = fmaf(conv_w[(size_t)j * C + c], past[taps - 1 - j], s);
        if (alone && st)                              // oldest first: what was one back is now two back
            for (int q = 0; q < keep; ++q) st[(size_t)q * C + c] = from_float<T>(past[keep - 1 - q]);
        return apply_activation(s, act);
    };
    // The token's work is spread over gridDim.y blocks: heads of q and k a warp each (unit vectors), the rest a thread
    // per channel.
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    float* mine = y + warp * dk;
    for (int u = blockIdx.y * warps + warp; u < 2 * G; u += gridDim.y * warps) {      // the heads of q, then those of k
        float ss = 0.f;
        for (int i = lane; i < dk; i += 32) {
            const float x = conv(u * dk + i);
            mine[i] = x;
            ss = fmaf(x, x, ss);
        }
        const float rinv = (u < G ? q_scale : 1.f) / sqrtf(warp_sum(ss) + unit_eps);
        float* dst = (u < G ? q_out + (size_t)n * G * dk + u * dk : k_out + (size_t)n * G * dk + (u - G) * dk);
        for (int i = lane; i < dk; i += 32) dst[i] = mine[i] * rinv;      // a lane reads back what it wrote itself
    }
    const int first = blockIdx.y * blockDim.x + threadIdx.x, stride = gridDim.y * blockDim.x;
    for (int c = first; c < H * dv; c += stride) v_out[(size_t)n * H * dv + c] = conv(nqk + c);
    for (int h = first; h < H; h += stride)
        beta_out[(size_t)n * H + h] = 1.f / (1.f + expf(-to_float(proj[(size_t)n * ld + b_off + h])));
    for (int c = first; c < H * dk; c += stride) {
        const float rate = expf(a_log[c / dk]);
        g_out[(size_t)n * H * dk + c] = expf(-rate * softplus_f(a[(size_t)n * a_ld + c] + dt_bias[c]));
    }
}

// The same with eight channels a thread (16-byte loads of the projections and the state, the taps' loads independent of
// one another): sizes and addresses in multiples of eight channels.
// TAPS: the number of taps where it is the usual four (a thread then has all its rows' loads in flight; one after the other a
// token's three rounds of four loads are what its block waits for), 0: any.  1,536 tokens, 16 heads
// of 128 on 4: 34.2 -> 29.0 us; about half of that is exponentials, logarithms and divisions in full 32-bit precision.
template <typename T, int TAPS>
__global__ void __launch_bounds__(256)
delta_prep_vec_kernel(const T* __restrict__ proj, int ld, int col0, int b_off, const float* __restrict__ a, int a_ld,
                  const float* __restrict__ conv_w, int taps, T* state, const int* __restrict__ token_request,
                  const int* __restrict__ positions, const int* __restrict__ q_start, const int* __restrict__ q_len,
                  const int* __restrict__ state_slots, const float* __restrict__ a_log, const float* __restrict__ dt_bias,
                  float unit_eps, float q_scale, int act, float* __restrict__ q_out, float* __restrict__ k_out,
                  float* __restrict__ v_out, float* __restrict__ beta_out, float* __restrict__ g_out, int H, int G, int dk,
                  int dv) {
    extern __shared__ float y[];                      // a query or key head's convolved channels, per warp
    pdl_launch_dependents();
    pdl_wait();
    const int n = blockIdx.x;
    const int req = token_request[n];
    if (req < 0) return;                              // a padded row of a captured step
    const int pos = positions[n], idx = n - q_start[req], slot = state_slots[req];
    const bool alone = q_len[req] == 1;
    const int keep = taps - 1, nqk = 2 * G * dk, C = nqk + H * dv;
    const T* row = proj + (size_t)n * ld + col0;
    T* st = (keep > 0 && slot >= 0) ? state + (size_t)slot * keep * C : nullptr;
    auto conv8 = [&](int c, float (&s)[8]) {          // channels c .. c + 7: convolution, state shift, activation
#pragma unroll
        for (int i = 0; i < 8; ++i) s[i] = 0.f;
        auto source = [&](int b) -> const T* {        // the value b positions back: this step's rows, the state, or zero
            if (b == 0) return row + c;
            if (pos - b < 0) return nullptr;
            if (idx - b >= 0) return row + c - (ptrdiff_t)b * ld;
            return st ? st + (size_t)(keep + idx - b) * C + c : nullptr;
        };
        auto tap = [&](int b, const Vec8<T>& x) {
            const float* w = conv_w + (size_t)(keep - b) * C + c;
            const float4 w0 = *(const float4*)w, w1 = *(const float4*)(w + 4);
            float xv[8];
            x.get(xv);
            s[0] = fmaf(w0.x, xv[0], s[0]); s[1] = fmaf(w0.y, xv[1], s[1]); s[2] = fmaf(w0.z, xv[2], s[2]);
            s[3] = fmaf(w0.w, xv[3], s[3]); s[4] = fmaf(w1.x, xv[4], s[4]); s[5] = fmaf(w1.y, xv[5], s[5]);
            s[6] = fmaf(w1.z, xv[6], s[6]); s[7] = fmaf(w1.w, xv[7], s[7]);
        };
        // oldest first, as the one-channel form adds them; a request's single row moves its past on: what is b back now is
        // b + 1 back for the next token
        if constexpr (TAPS > 0) {
            Vec8<T> x[TAPS];
#pragma unroll
            for (int b = TAPS - 1; b >= 0; --b) {
                const T* src = source(b);
                if (src) x[b].load(src); else x[b].zero();
            }
#pragma unroll
            for (int b = TAPS - 1; b >= 0; --b) {
                tap(b, x[b]);
                if (alone && st && b < TAPS - 1) x[b].store(st + (size_t)(TAPS - 2 - b) * C + c);
            }
        } else {
            for (int b = keep; b >= 0; --b) {         // the slot written here was read one round ago
                const T* src = source(b);
                Vec8<T> x;
                if (src) x.load(src); else x.zero();
                tap(b, x);
                if (alone && st && b < keep) x.store(st + (size_t)(keep - 1 - b) * C + c);
            }
        }
        if (act == TNX_ACT_SILU) {                    // inline: the usual one
#pragma unroll
            for (int i = 0; i < 8; ++i) s[i] = s[i] / (1.f + expf(-s[i]));
            return;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) s[i] = apply_activation(s[i], act);
    };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    float* mine = y + warp * dk;
    for (int u = blockIdx.y * warps + warp; u < 2 * G; u += gridDim.y * warps) {      // the heads of q, then those of k
        float ss = 0.f;
        for (int i = 8 * lane; i < dk; i += 256) {
            float s[8];
            conv8(u * dk + i, s);
#pragma unroll
            for (int e = 0; e < 8; ++e) ss = fmaf(s[e], s[e], ss);
            *(float4*)(mine + i) = make_float4(s[0], s[1], s[2], s[3]);
            *(float4*)(mine + i + 4) = make_float4(s[4], s[5], s[6], s[7]);
        }
        const float rinv = (u < G ? q_scale : 1.f) / sqrtf(warp_sum(ss) + unit_eps);
        float* dst = (u < G ? q_out + (size_t)n * G * dk + u * dk : k_out + (size_t)n * G * dk + (u - G) * dk);
        for (int i = 8 * lane; i < dk; i += 256) {    // a lane reads back what it wrote itself
            float4 a0 = *(const float4*)(mine + i), a1 = *(const float4*)(mine + i + 4);
            a0.x *= rinv; a0.y *= rinv; a0.z *= rinv; a0.w *= rinv; a1.x *= rinv; a1.y *= rinv; a1.z *= rinv; a1.w *= rinv;
            *(float4*)(dst + i) = a0;
            *(float4*)(dst + i + 4) = a1;
        }
    }
    const int first = blockIdx.y * blockDim.x + threadIdx.x, stride = gridDim.y * blockDim.x;
    for (int c = 8 * first; c < H * dv; c += 8 * stride) {
        float s[8];
        conv8(nqk + c, s);
        float* dst = v_out + (size_t)n * H * dv + c;
        *(float4*)dst = make_float4(s[0], s[1], s[2], s[3]);
        *(float4*)(dst + 4) = make_float4(s[4], s[5], s[6], s[7]);
    }
    for (int h = first; h < H; h += stride)
        beta_out[(size_t)n * H + h] = 1.f / (1.f + expf(-to_float(proj[(size_t)n * ld + b_off + h])));
    for (int c = 4 * first; c < H * dk; c += 4 * stride) {          // four channels of one head (dk is a multiple of 8)
        const float rate = expf(a_log[c / dk]);
        const float4 x = *(const float4*)(a + (size_t)n * a_ld + c), bias = *(const float4*)(dt_bias + c);
        *(float4*)(g_out + (size_t)n * H * dk + c) =
            make_float4(expf(-rate * softplus_f(x.x + bias.x)), expf(-rate * softplus_f(x.y + bias.y)),
                        expf(-rate * softplus_f(x.z + bias.z)), expf(-rate * softplus_f(x.w + bias.w)));
    }
}

// tokens whose inputs are staged in shared memory at a time, in each of two buffers (24 KB of keys, queries and decays)
__host__ __device__ constexpr int scan_stage(int dkp) { return dkp > 128 ? 4 : dkp > 64 ? 8 : 16; }

// Asynchronous copies global -> shared; `bytes_src` 0 fills the destination with zeros and reads nothing.
__device__ __forceinline__ void cp_async4(float* dst, const float* src, bool take) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(take ? 4u : 0u) : "memory");
}
__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool take) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(take ? 16u : 0u) : "memory");
}

// One form for every token, so that the state after a token has the same bits however the prompt was cut.  KPT: rows of a
// column one thread keeps; R: lanes a column's rows are spread over (KPT * R >= k_dim); a block of 128
// threads owns 128 / R columns.  The tokens' inputs come in stages through two buffers: while one stage is walked, the
// next one's copies are in flight, so the walk waits for memory once, at the first stage.  VEC: k_dim is a multiple
// of 4 and the rows are 16-byte aligned (16-byte copies).
template <int KPT, int R, bool VEC>
__global__ void __launch_bounds__(128)
delta_scan_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
                  const float* __restrict__ beta, const float* __restrict__ g, float* __restrict__ state,
                  const int* __restrict__ q_start, const int* __restrict__ q_len, const int* __restrict__ state_slots,
                  float* __restrict__ out, int H, int G, int dk, int dv) {
    constexpr int DKP = KPT * R, C = 128 / R, ST = scan_stage(KPT * R);
    __shared__ __align__(16) float qs[2][ST][DKP], ks[2][ST][DKP], gs[2][ST][DKP];
    __shared__ float vs[2][ST][C], bs[2][ST];
    pdl_launch_dependents();
    pdl_wait();
    const int req = blockIdx.z, h = blockIdx.y;
    const int len = q_len[req];
    if (len <= 0) return;                             // a padded request of a captured batch
    const int slot = state_slots[req];
    if (slot < 0) return;
    const int t_first = q_start[req], kvh = h / (H / G);
    const int jl = threadIdx.x / R, r = threadIdx.x % R;
    const int j = blockIdx.x * C + jl;
    const bool col = j < dv;

    auto fetch = [&](int t0, int buf) {               // the inputs of tokens t0 .. t0 + ST - 1 of this request's rows
        const int nt = min(ST, len - t0);
        if (VEC) {
            for (int e = threadIdx.x; e < nt * (DKP / 4); e += 128) {
                const int tt = e / (DKP / 4), i = (e % (DKP / 4)) * 4;
                const size_t t = (size_t)(t_first + t0 + tt);
                const bool in = i < dk;
                cp_async16(&qs[buf][tt][i], in ? q + (t * G + kvh) * dk + i : q, in);
                cp_async16(&ks[buf][tt][i], in ? k + (t * G + kvh) * dk + i : k, in);
                cp_async16(&gs[buf][tt][i], in ? g + (t * H + h) * dk + i : g, in);
            }
        } else {
            for (int e = threadIdx.x; e < nt * DKP; e += 128) {
                const int tt = e / DKP, i = e % DKP;
                const size_t t = (size_t)(t_first + t0 + tt);
                const bool in = i < dk;
                cp_async4(&qs[buf][tt][i], in ? q + (t * G + kvh) * dk + i : q, in);
                cp_async4(&ks[buf][tt][i], in ? k + (t * G + kvh) * dk + i : k, in);
                cp_async4(&gs[buf][tt][i], in ? g + (t * H + h) * dk + i : g, in);
            }
        }
        for (int e = threadIdx.x; e < nt * C; e += 128) {
            const int tt = e / C, c = blockIdx.x * C + e % C;
            cp_async4(&vs[buf][tt][e % C], c < dv ? v + ((size_t)(t_first + t0 + tt) * H + h) * dv + c : v, c < dv);
        }
        if (threadIdx.x < nt) cp_async4(&bs[buf][threadIdx.x], beta + (size_t)(t_first + t0 + threadIdx.x) * H + h, true);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    fetch(0, 0);
    float* st = state + (((size_t)slot * H + h) * dv + (col ? j : 0)) * dk;
    float S[KPT];
#pragma unroll
    for (int m = 0; m < KPT; ++m) S[m] = (col && r + R * m < dk) ? st[r + R * m] : 0.f;
    int buf = 0;
    for (int t0 = 0; t0 < len; t0 += ST, buf ^= 1) {
        const int nt = min(ST, len - t0);
        if (t0 + ST < len) {
            fetch(t0 + ST, buf ^ 1);                  // the buffer that the stage before this one used: all have left it
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();                              // every thread's copies of this stage have landed
        for (int tt = 0; tt < nt; ++tt) {
            float sk0 = 0.f, sk1 = 0.f, sq0 = 0.f, sq1 = 0.f, qk = 0.f;
            float Sg[KPT];
            // the decayed state first, then its products with k and q, in two chains each (half the dependent adds)
#pragma unroll
            for (int m = 0; m < KPT; ++m) {
                const int i = r + R * m;
                const float kk = ks[buf][tt][i], qq = qs[buf][tt][i], gg = gs[buf][tt][i];
                Sg[m] = S[m] * gg;
                if (m & 1) { sk1 = fmaf(kk, Sg[m], sk1); sq1 = fmaf(qq, Sg[m], sq1); }
                else { sk0 = fmaf(kk, Sg[m], sk0); sq0 = fmaf(qq, Sg[m], sq0); }
                qk = fmaf(qq, kk, qk);
            }
            float sk = sk0 + sk1, sq = sq0 + sq1;
#pragma unroll
            for (int o = R >> 1; o > 0; o >>= 1) {    // the R lanes of a column are neighbours in one warp
                sk += __shfl_xor_sync(0xffffffffu, sk, o);
                sq += __shfl_xor_sync(0xffffffffu, sq, o);
                qk += __shfl_xor_sync(0xffffffffu, qk, o);
            }
            const float u = bs[buf][tt] * (vs[buf][tt][jl] - sk);
#pragma unroll
            for (int m = 0; m < KPT; ++m) S[m] = fmaf(ks[buf][tt][r + R * m], u, Sg[m]);
            if (r == 0 && col) out[((size_t)(t_first + t0 + tt) * H + h) * dv + j] = fmaf(qk, u, sq);
        }
        __syncthreads();                              // the stage is no longer read: the next fetch may overwrite it
    }
    if (col) {
#pragma unroll
        for (int m = 0; m < KPT; ++m)
            if (r + R * m < dk) st[r + R * m] = S[m];
    }
}

// Two 32-bit numbers at once: an ordinary multiplication, or multiply-add, of each in one instruction.
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(*(const unsigned long long*)&a), "l"(*(const unsigned long long*)&b));
    return *(float2*)&d;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d)
        : "l"(*(const unsigned long long*)&a), "l"(*(const unsigned long long*)&b), "l"(*(const unsigned long long*)&c));
    return *(float2*)&d;
}
__device__ __forceinline__ float2 low(const float4& x) { return make_float2(x.x, x.y); }
__device__ __forceinline__ float2 high(const float4& x) { return make_float2(x.z, x.w); }

// Where the caller allows it (`ahead`): the first token of a call has no token before it whose write could be corrected for, so
// where a prompt was cut shows in the last bits.  A thread keeps KPT rows, in runs of four neighbours, of two neighbouring columns (what it reads from
// shared memory feeds both), and multiplies them in pairs; R lanes share the columns.
// A token's write waits for the sum u = beta (v - S^T k), and that sum over R lanes is most of a token's chain.  So the walk
// forms it a token ahead, from the state before the write that comes between, and corrects it by one number:
//     S_t^T k_(t+1) after its decay  =  (g_t S_(t-1))^T (g_(t+1) k_(t+1))  +  (k_t . g_(t+1) k_(t+1)) u_t
// One chain of a sum and a write then serves two tokens.  The four sums of a lane (the next token's S^T k and this one's
// S^T q, two columns) are added over the lanes by halving what a lane keeps in the first two rounds; the two numbers that
// the columns share (q.k and k.gk) likewise.  The lanes whose top bit is clear end up with S^T k and k.gk and form u, the
// others with S^T q and q.k and form the output.
// Measured, 16 heads of 128 x 128 on 4 key heads, against a column a lane and the sum inside the token's chain: three
// requests of 512 tokens 360 -> 198 us, one of 2,048 650 -> 406 (32 heads 969 -> 557), one of 64 26 -> 19, 64 single tokens 39 -> 35; four columns a
// lane without the sum ahead 251, 799 (799); two 209, 527 (650); eight lanes a column 228, 656.  Errors against 64-bit are equal.
// What bounds it: one warp a scheduler, about 150 instructions a token and the chain of two tokens in turn.
// Inputs come in stages through three buffers: one is walked, the next one has landed (the token ahead may be its first), the
// third one's copies are in flight.
constexpr int WIDE_THREADS = 128;
template <int KPT, int R>
__global__ void __launch_bounds__(WIDE_THREADS)
delta_scan_ahead_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
                        const float* __restrict__ beta, const float* __restrict__ g, float* __restrict__ state,
                        const int* __restrict__ q_start, const int* __restrict__ q_len, const int* __restrict__ state_slots,
                        float* __restrict__ out, int H, int G, int dk, int dv) {
    constexpr int DKP = KPT * R, C = WIDE_THREADS / R * 2, ST = scan_stage(DKP), RUNS = KPT / 4;
    __shared__ __align__(16) float qs[3 * ST][DKP], ks[3 * ST][DKP], gs[3 * ST][DKP];
    __shared__ __align__(16) float vs[3 * ST][C], bs[3 * ST];
    pdl_launch_dependents();
    pdl_wait();
    const int req = blockIdx.z, h = blockIdx.y;
    const int len = q_len[req];
    if (len <= 0) return;                             // a padded request of a captured batch
    const int slot = state_slots[req];
    if (slot < 0) return;
    const int t_first = q_start[req], kvh = h / (H / G);
    const int jl = threadIdx.x / R * 2, r = threadIdx.x % R;     // the thread's first column in the block, its place among the R lanes
    const int j0 = blockIdx.x * C + jl;

    auto fetch = [&](int t0, int at) {                // the inputs of tokens t0 .. t0 + ST - 1 of this request into rows `at` on
        const int nt = min(ST, len - t0);
        for (int e = threadIdx.x; e < nt * (DKP / 4); e += WIDE_THREADS) {
            const int tt = e / (DKP / 4), i = (e % (DKP / 4)) * 4;
            const size_t t = (size_t)(t_first + t0 + tt);
            const bool in = i < dk;
            cp_async16(&qs[at + tt][i], in ? q + (t * G + kvh) * dk + i : q, in);
            cp_async16(&ks[at + tt][i], in ? k + (t * G + kvh) * dk + i : k, in);
            cp_async16(&gs[at + tt][i], in ? g + (t * H + h) * dk + i : g, in);
        }
        for (int e = threadIdx.x; e < nt * C; e += WIDE_THREADS) {
            const int tt = e / C, c = blockIdx.x * C + e % C;
            cp_async4(&vs[at + tt][e % C], c < dv ? v + ((size_t)(t_first + t0 + tt) * H + h) * dv + c : v, c < dv);
        }
        for (int e = threadIdx.x; e < nt; e += WIDE_THREADS) cp_async4(&bs[at + e], beta + (size_t)(t_first + t0 + e) * H + h, true);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0, 0);
    fetch(ST, ST);                                    // an empty group where the request has one stage

    float2 S[2][KPT / 2];                             // rows 4 (r + R m) .. + 3 of the two columns, in pairs
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const float* st = state + (((size_t)slot * H + h) * dv + min(j0 + c, dv - 1)) * dk;
#pragma unroll
        for (int m = 0; m < RUNS; ++m) {
            const int i = 4 * (r + R * m);
            const float4 x = j0 + c < dv && i < dk ? *(const float4*)(st + i) : make_float4(0.f, 0.f, 0.f, 0.f);
            S[c][2 * m] = low(x); S[c][2 * m + 1] = high(x);
        }
    }
    const unsigned FULL = 0xffffffffu;
    const bool top = r & (R / 2);
    const int mine = r / (R / 4) & 1;                 // the column whose sum the lane ends up with
    float* o = out + ((size_t)t_first * H + h) * dv + j0 + mine;
    const bool stores = top && r % (R / 4) == 0 && j0 + mine < dv;
    // The sums a[0], a[1] (to the lanes with the top bit clear) and b[0], b[1] (to the others) over the R lanes.
    auto sum_columns = [&](float2 (&a)[2], float2 (&b)[2]) {
        const float a0 = a[0].x + a[0].y, a1 = a[1].x + a[1].y, b0 = b[0].x + b[0].y, b1 = b[1].x + b[1].y;
        const float w0 = (top ? b0 : a0) + __shfl_xor_sync(FULL, top ? a0 : b0, R / 2);
        const float w1 = (top ? b1 : a1) + __shfl_xor_sync(FULL, top ? a1 : b1, R / 2);
        float w = (mine ? w1 : w0) + __shfl_xor_sync(FULL, mine ? w0 : w1, R / 4);
#pragma unroll
        for (int x = R / 8; x > 0; x >>= 1) w += __shfl_xor_sync(FULL, w, x);
        return w;
    };
    auto sum_shared = [&](float a, float b) {
        float w = (top ? b : a) + __shfl_xor_sync(FULL, top ? a : b, R / 2);
#pragma unroll
        for (int x = R / 4; x > 0; x >>= 1) w += __shfl_xor_sync(FULL, w, x);
        return w;
    };

    float4 k4[RUNS], q4[RUNS], g4[RUNS];              // of the token that is walked
    float ahead = 0.f, shared = 0.f, u_before = 0.f;  // its S^T k but for the write before it; (k.gk | q.k); that write's u
    int at = 0;
    for (int t0 = 0; t0 < len; t0 += ST) {
        const int nt = min(ST, len - t0);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                              // this stage and the next one are there; the one before is no longer read
        if (t0 + 2 * ST < len) fetch(t0 + 2 * ST, at >= ST ? at - ST : 2 * ST);
        if (t0 == 0) {                                // the first token's sum has no write before it
            float2 sk[2], none[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
            for (int m = 0; m < RUNS; ++m) {
                const int i = 4 * (r + R * m);
                k4[m] = *(const float4*)&ks[0][i]; q4[m] = *(const float4*)&qs[0][i]; g4[m] = *(const float4*)&gs[0][i];
                const float2 kl = mul2(low(k4[m]), low(g4[m])), kh = mul2(high(k4[m]), high(g4[m]));
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    sk[c] = m ? fma2(kl, S[c][2 * m], sk[c]) : mul2(kl, S[c][2 * m]);
                    sk[c] = fma2(kh, S[c][2 * m + 1], sk[c]);
                }
            }
            ahead = sum_columns(sk, none);
        }
#pragma unroll 2
        for (int tt = 0; tt < nt; ++tt) {
            const int row = at + tt, next = t0 + tt + 1 < len ? (row + 1 < 3 * ST ? row + 1 : 0) : row;
            const float vb = vs[row][jl + mine], b = bs[row];
            float4 kn[RUNS], gn[RUNS], qn[RUNS];
            float2 sk[2], sq[2], qk, kgk;
#pragma unroll
            for (int m = 0; m < RUNS; ++m) {
                const int i = 4 * (r + R * m);
                kn[m] = *(const float4*)&ks[next][i]; gn[m] = *(const float4*)&gs[next][i]; qn[m] = *(const float4*)&qs[next][i];
            }
            // u of this token: the sum formed a token ago and the write since
            const float u_mine = b * (vb - fmaf(shared, u_before, ahead));       // in the lanes whose top bit is clear
            const float u0 = __shfl_sync(FULL, u_mine, 0, R), u1 = __shfl_sync(FULL, u_mine, R / 4, R);
#pragma unroll
            for (int m = 0; m < KPT / 2; ++m) {
                const float2 kp = m & 1 ? high(k4[m / 2]) : low(k4[m / 2]), qp = m & 1 ? high(q4[m / 2]) : low(q4[m / 2]);
                const float2 gp = m & 1 ? high(g4[m / 2]) : low(g4[m / 2]);
                const float2 kg = m & 1 ? mul2(high(kn[m / 2]), high(gn[m / 2])) : mul2(low(kn[m / 2]), low(gn[m / 2]));
                qk = m ? fma2(qp, kp, qk) : mul2(qp, kp);
                kgk = m ? fma2(kp, kg, kgk) : mul2(kp, kg);
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    S[c][m] = mul2(S[c][m], gp);
                    sk[c] = m ? fma2(kg, S[c][m], sk[c]) : mul2(kg, S[c][m]);
                    sq[c] = m ? fma2(qp, S[c][m], sq[c]) : mul2(qp, S[c][m]);
                }
            }
            const float both = sum_shared(kgk.x + kgk.y, qk.x + qk.y);
            const float sums = sum_columns(sk, sq);
#pragma unroll
            for (int m = 0; m < KPT / 2; ++m) {
                const float2 kp = m & 1 ? high(k4[m / 2]) : low(k4[m / 2]);
                S[0][m] = fma2(kp, make_float2(u0, u0), S[0][m]);
                S[1][m] = fma2(kp, make_float2(u1, u1), S[1][m]);
            }
            if (stores) *o = fmaf(both, mine ? u1 : u0, sums);
            o += (size_t)H * dv;
            ahead = sums; shared = both; u_before = u_mine;
#pragma unroll
            for (int m = 0; m < RUNS; ++m) { k4[m] = kn[m]; g4[m] = gn[m]; q4[m] = qn[m]; }
        }
        at = at + ST < 3 * ST ? at + ST : 0;
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        float* st = state + (((size_t)slot * H + h) * dv + j0 + c) * dk;
#pragma unroll
        for (int m = 0; m < RUNS; ++m) {
            const int i = 4 * (r + R * m);
            if (j0 + c < dv && i < dk) *(float4*)(st + i) = make_float4(S[c][2 * m].x, S[c][2 * m].y, S[c][2 * m + 1].x, S[c][2 * m + 1].y);
        }
    }
}

}  // namespace

TNX_EXPORT int tnx_delta_prep(const void* proj, int ld, int col0, int b_off, const float* a, int a_ld, const float* conv_w,
                              int taps, void* state, const int* token_request, const int* positions, const int* q_start,
                              const int* q_len, const int* state_slots, const float* a_log, const float* dt_bias,
                              float unit_eps, float q_scale, int act, float* q_out, float* k_out, float* v_out,
                              float* beta_out, float* g_out, int n_tokens, int H, int G, int dk, int dv, int is_h16,
                              cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G || dk <= 0 || dv <= 0 || taps < 1 || taps > PREP_MAX_TAPS || !conv_w ||
        (taps > 1 && !state) || act < 0 || act >= TNX_ACT_COUNT)
        return TNX_ERR_BAD_ARG;
    const size_t smem = (size_t)8 * dk * sizeof(float);
    if (smem > 200 * 1024) return TNX_ERR_UNSUPPORTED;
    // few tokens: a token's channels over several blocks, so that a step of single tokens fills the device
    const int most = max(1, max((2 * G + 7) / 8, (H * max(dk, dv) + 255) / 256));
    const int parts = min(most, max(1, (PREP_FILL_BLOCKS + n_tokens - 1) / n_tokens));
    const bool vec = dk % 8 == 0 && dv % 8 == 0 && ld % 8 == 0 && col0 % 8 == 0 && a_ld % 4 == 0 &&
                     !(((uintptr_t)proj | (uintptr_t)state | (uintptr_t)conv_w | (uintptr_t)a | (uintptr_t)dt_bias |
                        (uintptr_t)q_out | (uintptr_t)k_out | (uintptr_t)v_out | (uintptr_t)g_out) & 15);
#define DPREP(T)                                                                                                        \
    do {                                                                                                                \
        auto kernel = !vec ? delta_prep_kernel<T> : taps == 4 ? delta_prep_vec_kernel<T, 4> : delta_prep_vec_kernel<T, 0>;                                            \
        if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);     \
        return tnx_launch_in_order(kernel, dim3(n_tokens, parts), dim3(256), smem, stream, (const T*)proj, ld, col0,    \
                                   b_off, a, a_ld, conv_w, taps, (T*)state, token_request, positions, q_start, q_len,   \
                                   state_slots, a_log, dt_bias, unit_eps, q_scale, act, q_out, k_out, v_out, beta_out,  \
                                   g_out, H, G, dk, dv);                                                                \
    } while (0)
    if (is_h16) DPREP(h16);
    DPREP(float);
#undef DPREP
}

TNX_EXPORT int tnx_delta_scan(const float* q, const float* k, const float* v, const float* beta, const float* g,
                              float* state, const int* q_start, const int* q_len, const int* state_slots, float* out,
                              int n_requests, int H, int G, int dk, int dv, int ahead, cudaStream_t stream) {
    if (n_requests <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G || dk <= 0 || dv <= 0) return TNX_ERR_BAD_ARG;
    const bool vec = dk % 4 == 0 && !(((uintptr_t)q | (uintptr_t)k | (uintptr_t)g) & 15);
    const bool wide = ahead && vec && !((uintptr_t)state & 15);
#define DSCAN(KPT, R)                                                                                                   \
    do {                                                                                                                \
        const int C = wide ? 2 * (WIDE_THREADS / (R)) : 128 / (R);                                                      \
        const dim3 grid((dv + C - 1) / C, H, n_requests);                                                               \
        if (wide)                                                                                                       \
            return tnx_launch_in_order(delta_scan_ahead_kernel<KPT, R>, grid, dim3(WIDE_THREADS), 0, stream, q, k, v,   \
                                       beta, g, state, q_start, q_len, state_slots, out, H, G, dk, dv);                 \
        if (vec)                                                                                                        \
            return tnx_launch_in_order(delta_scan_kernel<KPT, R, true>, grid, dim3(128), 0, stream, q, k, v, beta, g,   \
                                       state, q_start, q_len, state_slots, out, H, G, dk, dv);                          \
        return tnx_launch_in_order(delta_scan_kernel<KPT, R, false>, grid, dim3(128), 0, stream, q, k, v, beta, g,      \
                                   state, q_start, q_len, state_slots, out, H, G, dk, dv);                              \
    } while (0)
    if (dk <= 16) DSCAN(4, 4);
    if (dk <= 32) DSCAN(4, 8);
    if (dk <= 64) DSCAN(8, 8);
    if (dk <= 128) DSCAN(8, 16);
    if (dk <= 256) DSCAN(16, 16);
    return TNX_ERR_UNSUPPORTED;
#undef DSCAN
}
