// The state-space recurrence and the gated delta rules over prompt portions, in chunks (chunk_walk.cuh says how): what the
// walk needs of each chunk, and the launches.
#include "chunk_walk.cuh"

namespace se {
namespace walk {

// State space: one block per (chunk, group of heads that share B and C).  step = softplus(raw + bias), the log decay is
// -exp(A_log) step; P[t][s] = e^(B_t - B_s) C_t . B_s; the step sizes become the factor on the value rows.
template <int DP, typename T_>
__global__ void __launch_bounds__(kThreads, 3)
ssm_prepare_kernel(const float* __restrict__ xbc, const T_* __restrict__ proj, int pitch, int dt_off, const float* __restrict__ dt_bias,
                   const float* __restrict__ a_log, const int* __restrict__ cu_q, int entries, float* __restrict__ p,
                   float* __restrict__ rs, float* __restrict__ ts, float* __restrict__ steps, int H, int P, int N, int G) {
    constexpr int T = 64, QP = DP + 4;
    extern __shared__ __align__(16) float sm[];
    float* qs = sm;                                  // C
    float* ks = qs + T * QP;                         // B
    __shared__ double sums[8][T];                    // B_t of eight heads at a time
    int first, n;
    chunk_of<T>(blockIdx.x, cu_q, entries, first, n);
    if (n <= 0) return;
    const int g = blockIdx.y, rep = H / G, width = H * P + 2 * G * N;
    load_tile<T, DP>(ks, xbc + H * P + (size_t)g * N, width, first, n, N);
    load_tile<T, DP>(qs, xbc + H * P + (size_t)(G + g) * N, width, first, n, N);
    cp_commit();
    cp_wait<0>();
    __syncthreads();
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float acc[4][4] = {};
    row_products<DP, 4>(qs, ks, ty, tx, acc);
    for (int h0 = 0; h0 < rep; h0 += 8) {
        __syncthreads();                             // the sums of the eight heads before have been read
        if (h0 + warp < rep) {                       // a warp per head, two neighbouring tokens per lane
            const int h = g * rep + h0 + warp;
            const float rate = expf(a_log[h]), bias = dt_bias[h];
            float step[2];
            double sum[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int t = 2 * lane + j;
                step[j] = t < n ? softplus32(to_float(proj[(size_t)(first + t) * pitch + dt_off + h]) + bias) : 0.f;
                sum[j] = -(double)rate * (double)step[j] + (j ? sum[0] : 0.0);
            }
            double before = sum[1];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double v = __shfl_up_sync(0xffffffffu, before, o);
                if (lane >= o) before += v;
            }
            const double last = __shfl_sync(0xffffffffu, before, 31);
            before -= sum[1];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int t = 2 * lane + j;
                const double b = before + sum[j];
                sums[warp][t] = b;
                if (t < n) {
                    const size_t at = (size_t)(first + t) * H + h;
                    rs[at] = expf((float)b);
                    ts[at] = expf((float)(last - b));
                    steps[at] = step[j];
                }
            }
        }
        __syncthreads();
        for (int hh = 0; hh < min(8, rep - h0); ++hh) {
            const int h = g * rep + h0 + hh;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int t = ty + 16 * i;
                if (t >= n) continue;
                const double bt = sums[hh][t];
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const int s = tx + 16 * b;
                    p[((size_t)(first + t) * H + h) * T + s] = s <= t ? acc[i][b] * expf((float)(bt - sums[hh][s])) : 0.f;
                }
            }
        }
    }
}

// x[t] -= sum_{s < t} A[t][s] x[s]: forward substitution, one column per thread; at [s][t] transposed, pitch T + 4
template <int T>
__device__ __forceinline__ void solve_column(float (&x)[T], const float* at) {
#pragma unroll
    for (int s = 0; s < T - 1; ++s) {
        const float xs = x[s];
#pragma unroll
        for (int t4 = (s + 1) / 4 * 4; t4 < T; t4 += 4) {
            const float4 v = ld4(at + s * (T + 4) + t4);
            const float v4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (t4 + j > s) x[t4 + j] = fmaf(-v4[j], xs, x[t4 + j]);
        }
    }
}

// Delta rule, one decay per head.  qkv: unit q | unit k | v rows; w [tokens][H][d], u [tokens][H][dv].
template <int DP>
__global__ void __launch_bounds__(kThreads, 2)
delta_head_prepare_kernel(const float* __restrict__ qkv, const float* __restrict__ log_dec, const float* __restrict__ beta,
                          const int* __restrict__ cu_q, int entries, float* __restrict__ p, float* __restrict__ w,
                          float* __restrict__ u, float* __restrict__ rs, float* __restrict__ ts, int H, int G, int d, int dv) {
    constexpr int T = 64, QP = DP + 4;
    extern __shared__ __align__(16) float sm[];
    float* qs = sm;
    float* ks = qs + T * QP;
    float* at = ks + T * QP;                         // [s][T + 4]: A[t][s]
    __shared__ double sums[T];
    __shared__ float bt[T], eb[T];
    int first, n;
    chunk_of<T>(blockIdx.x, cu_q, entries, first, n);
    if (n <= 0) return;
    const int h = blockIdx.y, g = h / (H / G), width = 2 * G * d + H * dv;
    load_tile<T, DP>(qs, qkv + (size_t)g * d, width, first, n, d);
    load_tile<T, DP>(ks, qkv + (size_t)(G + g) * d, width, first, n, d);
    cp_commit();
    if (threadIdx.x < 32) {                          // two neighbouring tokens per lane
        const int lane = threadIdx.x;
        double sum[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int t = 2 * lane + j;
            sum[j] = (t < n ? (double)log_dec[(size_t)(first + t) * H + h] : 0.0) + (j ? sum[0] : 0.0);
            bt[t] = t < n ? beta[(size_t)(first + t) * H + h] : 0.f;
        }
        double before = sum[1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double v = __shfl_up_sync(0xffffffffu, before, o);
            if (lane >= o) before += v;
        }
        const double last = __shfl_sync(0xffffffffu, before, 31);
        before -= sum[1];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int t = 2 * lane + j;
            const double b = before + sum[j];
            sums[t] = b;
            eb[t] = expf((float)b);
            if (t < n) {
                rs[(size_t)(first + t) * H + h] = eb[t];
                ts[(size_t)(first + t) * H + h] = expf((float)(last - b));
            }
        }
    }
    cp_wait<0>();
    __syncthreads();
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
    float kk[4][4] = {}, qk[4][4] = {};
    row_products<DP, 4>(ks, ks, ty, tx, kk);
    row_products<DP, 4>(qs, ks, ty, tx, qk);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int t = ty + 16 * i;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int s = tx + 16 * b;
            const float f = s <= t ? expf((float)(sums[t] - sums[s])) : 0.f;
            at[s * (T + 4) + t] = s < t ? bt[t] * f * kk[i][b] : 0.f;
            if (t < n) p[((size_t)(first + t) * H + h) * T + s] = s <= t ? qk[i][b] * f : 0.f;
        }
    }
    __syncthreads();
    for (int c = threadIdx.x; c < d + dv; c += kThreads) {
        float x[T];
        const float* vb = qkv + (size_t)first * width + 2 * G * d + (size_t)h * dv + (c - d);
#pragma unroll
        for (int t = 0; t < T; ++t)
            x[t] = c < d ? bt[t] * eb[t] * ks[t * QP + c] : t < n ? bt[t] * vb[(size_t)t * width] : 0.f;
        solve_column<T>(x, at);
        float* dst = c < d ? w + ((size_t)first * H + h) * d + c : u + ((size_t)first * H + h) * dv + (c - d);
        const size_t step = (size_t)H * (c < d ? d : dv);
#pragma unroll
        for (int t = 0; t < T; ++t)
            if (t < n) dst[t * step] = x[t];
    }
}

// Delta rule, one decay per head and key channel, chunks of 32 tokens in two blocks of 16.  Products of decays take the
// place of exponents: within a block P and A are summed with the decays multiplied up token by token, between the blocks
// k_t e^(B_t - B_15) and e^(B_15 - B_s) k_s are formed first.  Every factor is at most 1.  qt, kt [tokens][H][d]: e^(B_t) q_t and
// e^(B_n - B_t) k_t; tot [places][H][d]: e^(B_n).
template <int DP>
__global__ void __launch_bounds__(kThreads, 2)
delta_channel_prepare_kernel(const float* __restrict__ qkv, const float* __restrict__ dec, const float* __restrict__ beta,
                             const int* __restrict__ cu_q, int entries, float* __restrict__ p, float* __restrict__ w,
                             float* __restrict__ u, float* __restrict__ qt, float* __restrict__ kt, float* __restrict__ tot,
                             int H, int G, int d, int dv) {
    constexpr int T = 32, QP = DP + 4, HB = 16;
    extern __shared__ __align__(16) float sm[];
    float* qs = sm;                                  // [T][QP]
    float* ks = qs + T * QP;
    float* gs = ks + T * QP;                         // the decays; later e^(B_t) k_t
    float* ka = gs + T * QP;                         // [HB][QP]: the second block's k_t e^(B_t - B_15)
    float* qa = ka + HB * QP;                        // [HB][QP]: and its q_t e^(B_t - B_15)
    float* kb = qa + HB * QP;                        // [HB][QP]: the first block's e^(B_15 - B_s) k_s
    float* at = kb + HB * QP;                        // [T][T + 4]: A[t][s] at [s][t]
    float* pt = at + T * (T + 4);                    // [T][T + 4]: P[t][s]
    __shared__ float bt[T];
    int first, n;
    const int e = chunk_of<T>(blockIdx.x, cu_q, entries, first, n);
    if (n <= 0) return;
    (void)e;
    const int h = blockIdx.y, g = h / (H / G), width = 2 * G * d + H * dv;
    load_tile<T, DP>(qs, qkv + (size_t)g * d, width, first, n, d);
    load_tile<T, DP>(ks, qkv + (size_t)(G + g) * d, width, first, n, d);
    load_tile<T, DP>(gs, dec + (size_t)h * d, H * d, first, n, d);
    cp_commit();
    if (threadIdx.x < T) bt[threadIdx.x] = threadIdx.x < n ? beta[(size_t)(first + threadIdx.x) * H + h] : 0.f;
    for (int i = threadIdx.x; i < 2 * T * (T + 4); i += kThreads) at[i] = 0.f;
    cp_wait<0>();
    __syncthreads();
    // within the blocks: eight threads per (block, token s) walk t = s, s + 1, ... with e^(B_t - B_s) k_s of DP / 8 channels each
    {
        constexpr int W = DP / 8;
        const int part = threadIdx.x & 7, pair = threadIdx.x >> 3, b0 = (pair >> 4) * HB, sl = pair & 15, s = b0 + sl;
        float ex[W];
#pragma unroll
        for (int c = 0; c < W; c += 4) st4(ex + c, ld4(ks + s * QP + (c / 4 * 8 + part) * 4));
        for (int tl = 0; tl < HB; ++tl) {            // every thread takes every step: the sums below are over neighbouring lanes
            const int t = b0 + tl;
            float ak = 0.f, aq = 0.f;
#pragma unroll
            for (int c = 0; c < W; c += 4) {
                const int at4 = t * QP + (c / 4 * 8 + part) * 4;
                if (tl > sl) {
                    const float4 gv = ld4(gs + at4);
                    ex[c] *= gv.x; ex[c + 1] *= gv.y; ex[c + 2] *= gv.z; ex[c + 3] *= gv.w;
                }
                const float4 ev = ld4(ex + c);
                ak = fma4(ld4(ks + at4), ev, ak);
                aq = fma4(ld4(qs + at4), ev, aq);
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) {
                ak += __shfl_xor_sync(0xffffffffu, ak, o);
                aq += __shfl_xor_sync(0xffffffffu, aq, o);
            }
            if (part == 0 && tl >= sl) {
                pt[t * (T + 4) + s] = aq;
                if (tl > sl) at[s * (T + 4) + t] = bt[t] * ak;
            }
        }
    }
    __syncthreads();
    // the products of decays, a channel per thread
    if (threadIdx.x < DP) {
        const int c = threadIdx.x;
        float run = 1.f;                             // first block: e^(B_15 - B_s), backwards
#pragma unroll
        for (int s = HB - 1; s >= 0; --s) {
            kb[s * QP + c] = run * ks[s * QP + c];
            run *= gs[s * QP + c];
        }
        run = 1.f;                                   // second block: e^(B_t - B_15)
#pragma unroll
        for (int t = 0; t < HB; ++t) {
            run *= gs[(HB + t) * QP + c];
            ka[t * QP + c] = run * ks[(HB + t) * QP + c];
            qa[t * QP + c] = run * qs[(HB + t) * QP + c];
        }
        if (c < d) {
            run = 1.f;                               // to the chunk's end: e^(B_n - B_t), backwards
            for (int t = n - 1; t >= 0; --t) {
                kt[((size_t)(first + t) * H + h) * d + c] = run * ks[t * QP + c];
                run *= gs[t * QP + c];
            }
            tot[((size_t)blockIdx.x * H + h) * d + c] = run;
        }
        run = 1.f;                                   // from its start: e^(B_t)
        for (int t = 0; t < n; ++t) {
            run *= gs[t * QP + c];
            if (c < d) qt[((size_t)(first + t) * H + h) * d + c] = run * qs[t * QP + c];
            gs[t * QP + c] = run * ks[t * QP + c];
        }
    }
    __syncthreads();
    {                                                // between the blocks: 16 x 16 products, one of each kind per thread
        const int tl = threadIdx.x >> 4, s = threadIdx.x & 15, t = HB + tl;
        float ak = 0.f, aq = 0.f;
#pragma unroll 4
        for (int k = 0; k < DP; k += 4) {
            const float4 v = ld4(kb + s * QP + k);
            ak = fma4(ld4(ka + tl * QP + k), v, ak);
            aq = fma4(ld4(qa + tl * QP + k), v, aq);
        }
        at[s * (T + 4) + t] = bt[t] * ak;
        pt[t * (T + 4) + s] = aq;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < T * (T / 4); i += kThreads) {
        const int t = i / (T / 4), c = (i - t * (T / 4)) * 4;
        if (t < n) st4(p + ((size_t)(first + t) * H + h) * T + c, ld4(pt + t * (T + 4) + c));
    }
    for (int c = threadIdx.x; c < d + dv; c += kThreads) {
        float x[T];
        const float* vb = qkv + (size_t)first * width + 2 * G * d + (size_t)h * dv + (c - d);
#pragma unroll
        for (int t = 0; t < T; ++t) x[t] = t >= n ? 0.f : bt[t] * (c < d ? gs[t * QP + c] : vb[(size_t)t * width]);
        solve_column<T>(x, at);
        float* dst = c < d ? w + ((size_t)first * H + h) * d + c : u + ((size_t)first * H + h) * dv + (c - d);
        const size_t step = (size_t)H * (c < d ? d : dv);
#pragma unroll
        for (int t = 0; t < T; ++t)
            if (t < n) dst[t * step] = x[t];
    }
}

}  // namespace walk
}  // namespace se

// Sizes the chunked recurrences of this file take: rows and columns of a head's state.
extern "C" int se_chunk_walk_supported(int d, int dv) { return se::walk::takes(d, dv); }

// State space (arguments as se_ssm_scan's).  work: float [tokens * H * (64 + 3)].
extern "C" int se_ssm_walk(const float* xbc, const void* proj, int pitch, int dt_off, const float* dt_bias, const float* a_log,
                           const float* d_skip, float* state, long long state_stride, const int* cu_q, const int* seq_rows,
                           float* y, float* work, int tokens, int entries, int H, int P, int N, int G, int sms, int dtype,
                           cudaStream_t stream) {
    using namespace se::walk;
    if (entries <= 0 || tokens <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G) return SE_ERR_ARGUMENT;
    if (!takes(N, P) || H > 65535 || P / 16 >= 65535 || !aligned(xbc) || !aligned(y) || !aligned(work)) return SE_ERR_UNSUPPORTED;
    float* p = work;
    float* rs = p + (size_t)tokens * H * 64;
    float* ts = rs + (size_t)tokens * H;
    float* steps = ts + (size_t)tokens * H;
    SE_WALK_DIMS(N, {
        int rc = 0;
        SE_DISPATCH_DTYPE(dtype, T_, {
            rc = launch(ssm_prepare_kernel<DP, T_>, dim3(tokens / 64 + entries, G), 2 * 64 * (DP + 4) * sizeof(float), stream, xbc,
                        (const T_*)proj, pitch, dt_off, dt_bias, a_log, cu_q, entries, p, rs, ts, steps, H, P, N, G);
        });
        if (rc != 0) return rc;
        WalkArgs a = {};
        a.q = xbc + H * P + G * N; a.k = xbc + H * P; a.qk_stride = H * P + 2 * G * N; a.rep = H / G;
        a.v = xbc; a.v_stride = a.qk_stride; a.v_scale = steps; a.skip = d_skip;
        a.p = p; a.rs = rs; a.ts = ts; a.state = state; a.state_stride = state_stride; a.s_row = 1; a.s_col = N; a.o = y;
        a.cu_q = cu_q; a.seq_rows = seq_rows; a.H = H; a.d = N; a.dv = P;
        return launch_walk<64, DP, false, false, float>(a, entries, walk_columns(entries, H, P, sms), stream);
    });
}

// Delta rule with one decay per head (log_dec [tokens, H], dec null) or per head and key channel (dec [tokens, H * d], log_dec
// null); the other arguments as se_delta_scan's.  work: float [tokens * H * (64 + 2 + d + dv)], or
// [tokens * H * (32 + 3 * d + dv) + (tokens / 32 + entries) * H * d].
extern "C" int se_delta_walk(const float* qkv, const float* dec, const float* log_dec, const float* beta, float* state,
                             long long state_stride, const int* cu_q, const int* seq_rows, float* o, float* work, int tokens,
                             int entries, int H, int G, int d, int dv, int sms, cudaStream_t stream) {
    using namespace se::walk;
    if (entries <= 0 || tokens <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G || (dec == nullptr) == (log_dec == nullptr)) return SE_ERR_ARGUMENT;
    if (!takes(d, dv) || H > 65535 || dv / 16 >= 65535 || !aligned(qkv) || !aligned(o) || !aligned(work)) return SE_ERR_UNSUPPORTED;
    if (dec != nullptr && !aligned(dec)) return SE_ERR_UNSUPPORTED;
    const size_t rows = (size_t)tokens * H;
    WalkArgs a = {};
    a.state = state; a.state_stride = state_stride; a.s_row = 1; a.s_col = d; a.o = o; a.cu_q = cu_q; a.seq_rows = seq_rows;
    a.H = H; a.d = d; a.dv = dv;
    const int cols = walk_columns(entries, H, dv, sms);
    float* w = work;
    float* u = w + rows * d;
    a.w = w; a.v = u; a.v_stride = H * dv;
    SE_WALK_DIMS(d, {
        if (dec == nullptr) {
            float* p = u + rows * dv;
            float* rs = p + rows * 64;
            float* ts = rs + rows;
            const int rc = launch(delta_head_prepare_kernel<DP>, dim3(tokens / 64 + entries, H),
                                  (2 * 64 * (DP + 4) + 64 * 68) * sizeof(float), stream, qkv, log_dec, beta, cu_q, entries, p, w, u,
                                  rs, ts, H, G, d, dv);
            if (rc != 0) return rc;
            a.q = qkv; a.k = qkv + G * d; a.qk_stride = 2 * G * d + H * dv; a.rep = H / G; a.p = p; a.rs = rs; a.ts = ts;
            return launch_walk<64, DP, true, false, float>(a, entries, cols, stream);
        }
        float* qt = u + rows * dv;
        float* kt = qt + rows * d;
        float* p = kt + rows * d;
        float* tot = p + rows * 32;
        const int rc = launch(delta_channel_prepare_kernel<DP>, dim3(tokens / 32 + entries, H),
                              ((3 * 32 + 3 * 16) * (DP + 4) + 2 * 32 * 36) * sizeof(float), stream, qkv, dec, beta, cu_q, entries,
                              p, w, u, qt, kt, tot, H, G, d, dv);
        if (rc != 0) return rc;
        a.q = qt; a.k = kt; a.qk_stride = H * d; a.rep = 1; a.p = p; a.tot = tot;
        return launch_walk<32, DP, true, true, float>(a, entries, cols, stream);
    });
}
