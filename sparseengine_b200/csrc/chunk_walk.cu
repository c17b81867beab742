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
    constexpr int T = 64, QP = DP + 8;
    extern __shared__ __align__(16) float sm[];
    float* qs = sm;                                  // C
    float* ks = qs + T * QP;                         // B
    __shared__ double sums[8][T];                    // B_t of eight heads at a time
    int first, n;
    chunk_of<T>(blockIdx.x, cu_q, entries, first, n);
    if (n <= 0) return;
    const int g = blockIdx.y, rep = H / G, width = H * P + 2 * G * N;
    load_tile<T, DP, 8>(ks, xbc + H * P + (size_t)g * N, width, first, n, N);
    load_tile<T, DP, 8>(qs, xbc + H * P + (size_t)(G + g) * N, width, first, n, N);
    cp_commit();
    cp_wait<0>();
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float* const x[1] = {qs};
    triangle_products<DP, 1>(x, ks, warp, lane, [&](const auto& acc, int r0, int n0, int zeros) {
        constexpr int NT = sizeof(acc[0]) / sizeof(acc[0][0]);
        for (int h0 = 0; h0 < rep; h0 += 8) {
            roles_sync<kThreads>();                  // the sums of the eight heads before have been read
            if (h0 + warp < rep) {                   // a warp per head, two neighbouring tokens per lane
                const int h = g * rep + h0 + warp;
                const float rate = expf(a_log[h]), bias = dt_bias[h];
                float step[2];
                double sum[2];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int t = 2 * lane + j;
                    step[j] = t < n ? softplus32(to_float(proj[(size_t)(first + t) * pitch + dt_off + h]) + bias) : 0.f;
                    sum[j] = (t < n ? log_decay(rate, step[j]) : 0.0) + (j ? sum[0] : 0.0);
                }
                double before;
                const double last = sum_before(sum[1], lane, before);
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
            roles_sync<kThreads>();
            for (int hh = 0; hh < min(8, rep - h0); ++hh) {
                const int h = g * rep + h0 + hh;
#pragma unroll
                for (int j = 0; j < 4; j += 2) {
                    const int t = r0 + 4 * j;
                    if (t >= n) continue;
                    const double bt = sums[hh][t];
                    float* row = p + ((size_t)(first + t) * H + h) * T;
#pragma unroll
                    for (int x = 0; x < NT; ++x) {
                        const int s = n0 + 8 * x;
                        *reinterpret_cast<float2*>(row + s) = make_float2(s <= t ? acc[0][x][j] * expf((float)(bt - sums[hh][s])) : 0.f,
                                                                          s < t ? acc[0][x][j + 1] * expf((float)(bt - sums[hh][s + 1])) : 0.f);
                    }
                    for (int s = zeros; s < T; s += 16) *reinterpret_cast<float2*>(row + s) = make_float2(0.f, 0.f);
                }
            }
        }
    });
}

// x[t] -= sum_{s < t} A[t][s] x[s]: forward substitution, one column per thread; at [s][t] transposed
template <int T, int PITCH>
__device__ __forceinline__ void solve_column(float (&x)[T], const float* at) {
#pragma unroll
    for (int s = 0; s < T - 1; ++s) {
        const float xs = x[s];
#pragma unroll
        for (int t4 = (s + 1) / 4 * 4; t4 < T; t4 += 4) {
            const float4 v = ld4(at + s * PITCH + t4);
            const float v4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (t4 + j > s) x[t4 + j] = fmaf(-v4[j], xs, x[t4 + j]);
        }
    }
}

// The delta rules' inputs as the convolution and the projections leave them: qkv rows q | k | v; a head's decay (or its
// channels') is exp(-exp(A_log) softplus(a + dt_bias)), its beta a sigmoid of a projection's column; q and k become unit
// vectors, q also times q_scale.
template <typename T_>
struct DeltaInputs {
    const float* qkv;
    const T_* a;                   // [tokens][H] or [tokens][H * d], rows a_pitch apart
    int a_pitch;
    const T_* b;                   // beta's columns, rows b_pitch apart
    int b_pitch;
    const float* dt_bias;
    const float* a_log;
    float unit_eps, q_scale;
    const int* cu_q;
    int entries, H, G, d, dv;
};

__device__ __forceinline__ float sigmoid32(float v) { return 1.f / (1.f + expf(-v)); }

// One decay per head, chunks of 64 tokens.  q and k stay as they are: their lengths go into the factors of rows and columns (of
// P and A here, rs and ts in the walk).  eb: e^(B_t); w [tokens][H][d], u [tokens][H][dv].  The system is solved in two halves of
// 32 rows, a column per thread: the second half's right side takes the first half's solution in between (a straight-line solution
// of 64 rows is 2,600 instructions that every warp fetches).  Measured over 2,048 tokens of 16 heads of 128: 68 us, with unit
// vectors, decays and beta; 146 with those in a kernel ahead, the rows solved at once and the values asked for row by row.
template <int DP, typename T_>
__global__ void __launch_bounds__(kThreads, 2)
delta_head_prepare_kernel(const DeltaInputs<T_> in, float* __restrict__ p, float* __restrict__ w, float* __restrict__ u,
                          float* __restrict__ rs, float* __restrict__ ts, float* __restrict__ eb_out) {
    constexpr int T = 64, QP = DP + 8, HB = 32;
    const int H = in.H, G = in.G, d = in.d, dv = in.dv;
    extern __shared__ __align__(16) float sm[];
    float* ks = sm;
    float* at = ks + T * QP;                         // [s][T + 4]: A[t][s]
    float* qs = at + T * (T + 4);                    // q, later [HB][kThreads]: right sides of the second half
    __shared__ double sums[T];
    __shared__ float bt[T], eb[T], fq[T], fk[T];
    int first, n;
    chunk_of<T>(blockIdx.x, in.cu_q, in.entries, first, n);
    if (n <= 0) return;
    const int h = blockIdx.y, g = h / (H / G), width = 2 * G * d + H * dv, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    load_tile<T, DP, 8>(qs, in.qkv + (size_t)g * d, width, first, n, d);
    load_tile<T, DP, 8>(ks, in.qkv + (size_t)(G + g) * d, width, first, n, d);
    cp_commit();
    float after[2] = {};
    if (warp == 0) {                                 // two neighbouring tokens per lane
        const float rate = expf(in.a_log[h]);
        const float bias = in.dt_bias[h];
        double sum[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int t = 2 * lane + j;
            const size_t row = (size_t)(first + t);
            sum[j] = (t < n ? log_decay(rate, softplus32(to_float(in.a[row * in.a_pitch + h]) + bias)) : 0.0) + (j ? sum[0] : 0.0);
            bt[t] = t < n ? sigmoid32(to_float(in.b[row * in.b_pitch + h])) : 0.f;
        }
        double before;
        const double last = sum_before(sum[1], lane, before);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int t = 2 * lane + j;
            const double b = before + sum[j];
            sums[t] = b;
            eb[t] = expf((float)b);
            after[j] = expf((float)(last - b));
        }
    }
    cp_wait<0>();
    __syncthreads();
    for (int r = warp; r < 2 * T; r += kThreads / 32) {          // lengths of q's rows, then of k's
        const float* row = (r < T ? qs : ks - T * QP) + r * QP;
        float ss = 0.f;
        for (int c = lane * 4; c < DP; c += 128) ss = fma4(ld4(row + c), ld4(row + c), ss);
        ss = warp_sum(ss);
        if (lane == 0) (r < T ? fq : fk - T)[r] = (r < T ? in.q_scale : 1.f) / sqrtf(ss + in.unit_eps);
    }
    __syncthreads();
    if (warp == 0)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int t = 2 * lane + j;
            if (t < n) {
                const size_t at_ = (size_t)(first + t) * H + h;
                rs[at_] = fq[t] * eb[t];
                ts[at_] = fk[t] * after[j];
                eb_out[at_] = eb[t];
            }
        }
    const float* const x[2] = {ks, qs};
    triangle_products<DP, 2>(x, ks, warp, lane, [&](const auto& acc, int r0, int n0, int zeros) {
        constexpr int NT = sizeof(acc[0]) / sizeof(acc[0][0]);
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
            const int t = r0 + 4 * j;
            const float ft = bt[t] * fk[t];
            float* row = p + ((size_t)(first + t) * H + h) * T;
#pragma unroll
            for (int x = 0; x < NT; ++x) {
                const int s0 = n0 + 8 * x;
                float2 pv;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int s = s0 + i;
                    const float f = s <= t ? expf((float)(sums[t] - sums[s])) * fk[s] : 0.f;
                    at[s * (T + 4) + t] = s < t ? ft * f * acc[0][x][j + i] : 0.f;
                    (i ? pv.y : pv.x) = s <= t ? fq[t] * f * acc[1][x][j + i] : 0.f;
                }
                if (t < n) *reinterpret_cast<float2*>(row + s0) = pv;
            }
            for (int s = zeros; s < T; s += 16) {
                at[s * (T + 4) + t] = 0.f;
                at[(s + 1) * (T + 4) + t] = 0.f;
                if (t < n) *reinterpret_cast<float2*>(row + s) = make_float2(0.f, 0.f);
            }
        }
    });
    __syncthreads();                                 // A is there, q has been read
    for (int c = tid; c < d + dv; c += kThreads) {
        float* dst = c < d ? w + ((size_t)first * H + h) * d + c : u + ((size_t)first * H + h) * dv + (c - d);
        const size_t step = (size_t)H * (c < d ? d : dv);
        float* mine = qs + tid;                      // this thread's column of the second half's right sides
        float x[HB];
        if (c < d) {                                 // right sides: the second half's wait in shared memory
#pragma unroll 4
            for (int t = 0; t < HB; ++t) mine[t * kThreads] = bt[HB + t] * eb[HB + t] * fk[HB + t] * ks[(HB + t) * QP + c];
#pragma unroll
            for (int t = 0; t < HB; ++t) x[t] = bt[t] * eb[t] * fk[t] * ks[t * QP + c];
        } else {
            const float* vb = in.qkv + (size_t)first * width + 2 * G * d + (size_t)h * dv + (c - d);
#pragma unroll
            for (int t = 0; t < HB; ++t) x[t] = HB + t < n ? vb[(size_t)(HB + t) * width] : 0.f;       // asked for together
#pragma unroll
            for (int t = 0; t < HB; ++t) mine[t * kThreads] = bt[HB + t] * x[t];
#pragma unroll
            for (int t = 0; t < HB; ++t) x[t] = t < n ? vb[(size_t)t * width] : 0.f;
#pragma unroll
            for (int t = 0; t < HB; ++t) x[t] *= bt[t];
        }
#pragma unroll 1
        for (int half = 0;; ++half) {
            solve_column<HB, T + 4>(x, at + half * HB * (T + 4) + half * HB);
#pragma unroll
            for (int t = 0; t < HB; ++t)
                if (half * HB + t < n) dst[(half * HB + t) * step] = x[t];
            if (half == 1 || n <= HB) break;
#pragma unroll 1
            for (int t = 0; t < HB; t += 4) {        // four rows at a time take the first half's solution in
                float r[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) r[j] = mine[(t + j) * kThreads];
#pragma unroll
                for (int s = 0; s < HB; ++s) {
                    const float4 v = ld4(at + s * (T + 4) + HB + t);
                    r[0] = fmaf(-v.x, x[s], r[0]);
                    r[1] = fmaf(-v.y, x[s], r[1]);
                    r[2] = fmaf(-v.z, x[s], r[2]);
                    r[3] = fmaf(-v.w, x[s], r[3]);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) mine[(t + j) * kThreads] = r[j];
            }
#pragma unroll
            for (int t = 0; t < HB; ++t) x[t] = mine[t * kThreads];
        }
    }
}

// v[0..7] per lane -> the sum over the warp of the value numbered 4 (lane's bit 4) + 2 (bit 3) + (bit 2)
__device__ __forceinline__ float warp_sum8(float (&v)[8], int lane) {
#pragma unroll
    for (int o = 16, m = 4; o >= 4; o >>= 1, m >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < m; ++i) {
            const float give = up ? v[i] : v[i + m], keep = up ? v[i + m] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// One decay per head and key channel, chunks of 32 tokens in two blocks of 16.  Products of decays take the place of exponents:
// within a block P and A are summed with the decays multiplied up token by token (a warp takes four tokens s, a lane four
// channels: a token t's q, k and decays are read once for the four), between the blocks k_t e^(B_t - B_15) and e^(B_15 - B_s) k_s
// are formed first.  Every factor is at most 1.  Measured over 4,670 tokens of 16 heads of 128: 188 us (three blocks per SM; 207
// with two and fewer spills), 377 with a lane group per token s that read q, k and decays for itself and the inputs in a kernel
// ahead.  qt, kt [tokens][H][d]: e^(B_t) q_t and e^(B_n - B_t) k_t; tot [places][H][d]: e^(B_n).
template <int DP, typename T_>
__global__ void __launch_bounds__(kThreads, 3)
delta_channel_prepare_kernel(const DeltaInputs<T_> in, float* __restrict__ p, float* __restrict__ w, float* __restrict__ u,
                             float* __restrict__ qt, float* __restrict__ kt, float* __restrict__ tot) {
    constexpr int T = 32, QP = DP + 4, HB = 16;
    const int H = in.H, G = in.G, d = in.d, dv = in.dv;
    extern __shared__ __align__(16) float sm[];
    float* qs = sm;                                  // [T][QP]; rows of the second block later e^(B_t - B_15) q_t
    float* ks = qs + T * QP;                         // later e^(B_15 - B_s) k_s, then e^(B_t - B_15) k_t
    float* gs = ks + T * QP;                         // the decays; later e^(B_t) k_t
    float* at = gs + T * QP;                         // [T][T + 4]: A[t][s] at [s][t]
    float* pt = at + T * (T + 4);                    // [T][T + 4]: P[t][s]
    float* ends = pt + T * (T + 4);                  // [2][DP]: the blocks' products of decays
    __shared__ float bt[T];
    int first, n;
    chunk_of<T>(blockIdx.x, in.cu_q, in.entries, first, n);
    if (n <= 0) return;
    const int h = blockIdx.y, g = h / (H / G), width = 2 * G * d + H * dv, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    load_tile<T, DP, 4>(qs, in.qkv + (size_t)g * d, width, first, n, d);
    load_tile<T, DP, 4>(ks, in.qkv + (size_t)(G + g) * d, width, first, n, d);
    cp_commit();
    const float rate = expf(in.a_log[h]);
#pragma unroll 4
    for (int i = tid; i < T * (DP / 4); i += kThreads) {         // decays; 1 where there is no token or channel
        const int t = i / (DP / 4), c = (i % (DP / 4)) * 4;
        float4 v = make_float4(1.f, 1.f, 1.f, 1.f);
        if (t < n && c < d) {
            const float4 x = load4(in.a + (size_t)(first + t) * in.a_pitch + h * d + c), b = ld4(in.dt_bias + h * d + c);
            v = make_float4(expf(-rate * softplus32(x.x + b.x)), expf(-rate * softplus32(x.y + b.y)),
                            expf(-rate * softplus32(x.z + b.z)), expf(-rate * softplus32(x.w + b.w)));
        }
        st4(gs + t * QP + c, v);
    }
    if (tid < T) bt[tid] = tid < n ? sigmoid32(to_float(in.b[(size_t)(first + tid) * in.b_pitch + h])) : 0.f;
    for (int i = tid; i < 2 * T * (T + 4); i += kThreads) at[i] = 0.f;
    cp_wait<0>();
    __syncthreads();
    for (int r = warp; r < 2 * T; r += kThreads / 32) {          // unit vectors: q's rows, then k's (which follow them)
        float* row = qs + r * QP;
        float ss = 0.f;
        for (int c = lane * 4; c < DP; c += 128) ss = fma4(ld4(row + c), ld4(row + c), ss);
        const float f = (r < T ? in.q_scale : 1.f) / sqrtf(warp_sum(ss) + in.unit_eps);
        for (int c = lane * 4; c < DP; c += 128) {
            const float4 v = ld4(row + c);
            st4(row + c, make_float4(v.x * f, v.y * f, v.z * f, v.w * f));
        }
    }
    __syncthreads();
    // within the blocks
    {
        const int b0 = (warp >> 2) * HB, s0 = b0 + (warp & 3) * 4, c = lane * 4;
        const bool mine = c < DP;
        float ex[4][4] = {};
        if (mine)
#pragma unroll
            for (int j = 0; j < 4; ++j) st4(ex[j], ld4(ks + (s0 + j) * QP + c));
        for (int t = s0; t < b0 + HB; ++t) {
            float4 gv = make_float4(0.f, 0.f, 0.f, 0.f), kv = gv, qv = gv;
            if (mine) {
                gv = ld4(gs + t * QP + c);
                kv = ld4(ks + t * QP + c);
                qv = ld4(qs + t * QP + c);
            }
            float v[8];                              // A's four, P's four
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (t > s0 + j) { ex[j][0] *= gv.x; ex[j][1] *= gv.y; ex[j][2] *= gv.z; ex[j][3] *= gv.w; }
                const float4 x = make_float4(ex[j][0], ex[j][1], ex[j][2], ex[j][3]);
                v[j] = fma4(kv, x, 0.f);
                v[4 + j] = fma4(qv, x, 0.f);
            }
            const float sum = warp_sum8(v, lane);
            const int which = lane >> 2, s = s0 + (which & 3);
            if ((lane & 3) == 0) {
                if (which < 4 && t > s) at[s * (T + 4) + t] = bt[t] * sum;
                if (which >= 4 && t >= s) pt[t * (T + 4) + s] = sum;
            }
        }
    }
    __syncthreads();
    // the products of decays: a channel of a block per thread
    {
        const int c = tid % DP, half = tid / DP, r0 = half * HB * QP + c;
        float gv[HB], run = 1.f;
        if (half < 2) {
#pragma unroll
            for (int i = 0; i < HB; ++i) {
                gv[i] = gs[r0 + i * QP];
                run *= gv[i];
            }
            ends[half * DP + c] = run;
        }
        __syncthreads();
        const float start = half == 1 ? ends[c] : 1.f, rest = half == 0 ? ends[DP + c] : 1.f;
        const size_t at_ = ((size_t)(first + half * HB) * H + h) * d + c, step = (size_t)H * d;
        auto forward = [&]() {                       // from the block's start; e^(B_t) k_t takes the decays' place
            float f = 1.f;
#pragma unroll
            for (int i = 0; i < HB; ++i) {
                const int r = r0 + i * QP;
                f *= gv[i];
                const float kf = f * ks[r], qf = f * qs[r];
                gs[r] = start * kf;
                if (half) {
                    ks[r] = kf;
                    qs[r] = qf;
                }
                if (half * HB + i < n && c < d) qt[at_ + i * step] = start * qf;
            }
        };
        auto backward = [&]() {                      // to the block's end
            float f = 1.f;
#pragma unroll
            for (int i = HB - 1; i >= 0; --i) {
                const int r = r0 + i * QP;
                const float kr = f * ks[r];
                f *= gv[i];
                if (!half) ks[r] = kr;
                if (half * HB + i < n && c < d) kt[at_ + i * step] = rest * kr;
            }
        };
        if (half == 0) {
            forward();
            backward();
            if (c < d) tot[((size_t)blockIdx.x * H + h) * d + c] = ends[c] * ends[DP + c];
        } else if (half == 1) {
            backward();
            forward();
        }
    }
    __syncthreads();
    // between the blocks: 16 x 16 products of both kinds, 2 x 2 per thread, four neighbouring lanes share out the channels
    {
        const int part = tid & 3, tile = tid >> 2, t0 = tile >> 3, s0 = (tile & 1) * 4 + ((tile >> 1) & 3);
        float ak[2][2] = {}, aq[2][2] = {};
#pragma unroll 2
        for (int k = part * 4; k < DP; k += 16) {
            const float4 ya = ld4(ks + s0 * QP + k), yb = ld4(ks + (s0 + 8) * QP + k);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float4 kv = ld4(ks + (HB + t0 + 8 * i) * QP + k), qv = ld4(qs + (HB + t0 + 8 * i) * QP + k);
                ak[i][0] = fma4(kv, ya, ak[i][0]);
                ak[i][1] = fma4(kv, yb, ak[i][1]);
                aq[i][0] = fma4(qv, ya, aq[i][0]);
                aq[i][1] = fma4(qv, yb, aq[i][1]);
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
#pragma unroll
                for (int o = 1; o < 4; o <<= 1) {
                    ak[i][j] += __shfl_xor_sync(0xffffffffu, ak[i][j], o);
                    aq[i][j] += __shfl_xor_sync(0xffffffffu, aq[i][j], o);
                }
                const int t = HB + t0 + 8 * i, s = s0 + 8 * j;
                if (part == 0) at[s * (T + 4) + t] = bt[t] * ak[i][j];
                if (part == 1) pt[t * (T + 4) + s] = aq[i][j];
            }
    }
    __syncthreads();
    for (int i = tid; i < T * (T / 4); i += kThreads) {
        const int t = i / (T / 4), c = (i % (T / 4)) * 4;
        if (t < n) st4(p + ((size_t)(first + t) * H + h) * T + c, ld4(pt + t * (T + 4) + c));
    }
    for (int c = tid; c < d + dv; c += kThreads) {
        float x[T];
        if (c < d) {
#pragma unroll
            for (int t = 0; t < T; ++t) x[t] = bt[t] * gs[t * QP + c];
        } else {
            const float* vp = in.qkv + (size_t)first * width + 2 * G * d + (size_t)h * dv + (c - d);
#pragma unroll
            for (int t = 0; t < T; ++t, vp += width) x[t] = t < n ? *vp : 0.f;
#pragma unroll
            for (int t = 0; t < T; ++t) x[t] *= bt[t];
        }
        solve_column<T, T + 4>(x, at);
        float* dst = c < d ? w + ((size_t)first * H + h) * d + c : u + ((size_t)first * H + h) * dv + (c - d);
        const size_t step = (size_t)H * (c < d ? d : dv);
#pragma unroll
        for (int t = 0; t < T; ++t, dst += step)
            if (t < n) *dst = x[t];
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
            rc = launch(ssm_prepare_kernel<DP, T_>, dim3(tokens / 64 + entries, G), 2 * 64 * (DP + 8) * sizeof(float), stream, xbc,
                        (const T_*)proj, pitch, dt_off, dt_bias, a_log, cu_q, entries, p, rs, ts, steps, H, P, N, G);
        });
        if (rc != 0) return rc;
        WalkArgs a = {};
        a.q = xbc + H * P + G * N; a.k = xbc + H * P; a.qk_stride = H * P + 2 * G * N; a.rep = H / G;
        a.v = xbc; a.v_stride = a.qk_stride; a.v_scale = steps; a.skip = d_skip;
        a.p = p; a.rs = rs; a.ts = ts; a.eb = rs; a.state = state; a.state_stride = state_stride; a.s_row = 1; a.s_col = N; a.o = y;
        a.cu_q = cu_q; a.seq_rows = seq_rows; a.H = H; a.d = N; a.dv = P;
        return launch_walk<64, DP, false, false, false, false, float>(a, entries, walk_columns(entries, H, P, sms), stream);
    });
}

// Delta rule with one decay per head (`per_head`) or per head and key channel, from what the convolution and the projections
// leave: qkv [tokens][2 G d + H dv], a [tokens][H] or [tokens][H d] (rows a_pitch apart), beta's columns of `proj` from b_off on.
// work: float [tokens * H * (64 + 3 + d + dv)], or [tokens * H * (32 + 3 * d + dv) + (tokens / 32 + entries) * H * d].
extern "C" int se_delta_walk(const float* qkv, const void* in_a, int a_pitch, const void* proj, int pitch, int b_off,
                             const float* dt_bias, const float* a_log, float* state, long long state_stride, const int* cu_q,
                             const int* seq_rows, float* o, float* work, int tokens, int entries, int H, int G, int d, int dv,
                             float unit_eps, float q_scale, int per_head, int sms, int dtype, cudaStream_t stream) {
    using namespace se::walk;
    if (entries <= 0 || tokens <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G || a_pitch < (per_head ? H : H * d)) return SE_ERR_ARGUMENT;
    if (!takes(d, dv) || H > 65535 || dv / 16 >= 65535 || !aligned(qkv) || !aligned(o) || !aligned(work)) return SE_ERR_UNSUPPORTED;
    if (!per_head && (a_pitch % 4 || !aligned(in_a) || !aligned(dt_bias))) return SE_ERR_UNSUPPORTED;
    const size_t rows = (size_t)tokens * H;
    WalkArgs a = {};
    a.state = state; a.state_stride = state_stride; a.s_row = 1; a.s_col = d; a.o = o; a.cu_q = cu_q; a.seq_rows = seq_rows;
    a.H = H; a.d = d; a.dv = dv;
    float* w = work;
    float* u = w + rows * d;
    a.w = w; a.v = u; a.v_stride = H * dv;
    SE_DISPATCH_DTYPE(dtype, T_, {
        const DeltaInputs<T_> in{qkv, (const T_*)in_a, a_pitch, (const T_*)proj + b_off, pitch, dt_bias, a_log, unit_eps, q_scale,
                                 cu_q, entries, H, G, d, dv};
        SE_WALK_DIMS(d, {
            if (per_head) {
                float* p = u + rows * dv;
                float* rs = p + rows * 64;
                float* ts = rs + rows;
                float* eb = ts + rows;
                const int tile = 64 * (DP + 8) > 32 * kThreads ? 64 * (DP + 8) : 32 * kThreads;
                const int rc = launch(delta_head_prepare_kernel<DP, T_>, dim3(tokens / 64 + entries, H),
                                      (64 * (DP + 8) + 64 * 68 + tile) * sizeof(float), stream, in, p, w, u, rs, ts, eb);
                if (rc != 0) return rc;
                a.q = qkv; a.k = qkv + G * d; a.qk_stride = 2 * G * d + H * dv; a.rep = H / G; a.p = p; a.rs = rs; a.ts = ts; a.eb = eb;
                return launch_walk<64, DP, true, false, false, false, float>(a, entries, walk_columns(entries, H, dv, sms), stream);
            }
            float* qt = u + rows * dv;
            float* kt = qt + rows * d;
            float* p = kt + rows * d;
            float* tot = p + rows * 32;
            const int rc = launch(delta_channel_prepare_kernel<DP, T_>, dim3(tokens / 32 + entries, H),
                                  (3 * 32 * (DP + 4) + 2 * 32 * 36 + 2 * DP) * sizeof(float), stream, in, p, w, u, qt, kt, tot);
            if (rc != 0) return rc;
            a.q = qt; a.k = kt; a.qk_stride = H * d; a.rep = 1; a.p = p; a.tot = tot;
            // Chunks of 32 tokens leave two blocks an SM: 16 columns are ahead also where there are many (16 heads, walk alone in us by columns,
            // 16 / 32: two entries of 1,558 tokens 201 / 248, three of 1,500 311 / 331, four of 1,500 320 / 335; eight of 700 the same).
            return launch_walk_columns<32, DP, 16, true, true, true, false, float>(a, entries, stream);
        });
    });
}
