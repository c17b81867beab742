// Linear recurrences over prompt portions in chunks of T tokens, all in 32-bit: the state-space recurrence, retention and
// both gated delta rules.  Within a chunk (local index t, s; S_0 the state at its start; B_t the sum of the log decays up to
// and with token t, a number per head or one per key channel) every one of them is
//
//     u   = U - W S_0                                   (delta rules; else u is the value row)
//     o_t = e^(B_t) q_t . S_0 + sum_{s <= t} P[t][s] u_s,         P[t][s] = q_t . e^(B_t - B_s) k_s
//     S   = e^(B_n) S_0 + sum_s (e^(B_n - B_s) k_s) u_s^T
//
// and, for the delta rules, [W | U] solves (I + A) X = [beta e^(B) K | beta V] with A[t][s] = beta_t k_t . e^(B_t - B_s) k_s for
// s < t.  So the work splits in two kernels: a `prepare` kernel per (chunk, head), parallel over all chunks of the step, which
// makes P and where needed W and U (and per-channel decays' scaled q and k); and a `walk` kernel per (request, head, tile of
// value columns) that takes the chunks in turn with its slice of the state in shared memory: two or three small matrix
// products per chunk instead of a chain of T dependent steps.
// (State spaces and retention beside bfloat16 activations have a form whose outputs are no part of the chain: chunk_tiles.cuh.)
//
// What bounds the walk is the chain of a chunk: products, the split of their operands, barriers, the state through shared memory.  The tensor pipe is busy
// 43 % of the time (state space), instructions issue in 49 % of the cycles; 16-bit operands would
// lose what the recurrence has to keep.  With multiply-adds it stood at half their rate, its other half shared-memory reads (8 x 8 outputs
// a thread, an LDS.128 each four multiply-adds); products in tf32 terms by mma.sync read less.  Measured, multiply-adds / now: state space,
// 2,048 tokens of 64 heads of 64 columns, 204 / 151 us; retention, 8,192 tokens of 32 heads of 128, 752 / 456; delta rule per channel, 4,670 tokens of
// 16 heads of 128, 418 / 322; per head, 2,048 tokens, 176 / 122.  Sixteen warps at the products instead of eight, all loading for themselves: 168, 616, -, 148
// (eight: 152, 563, 333 with 32 value columns, 134).  Every exponent is a
// difference of sums of logarithms that is at most 0 up to the 64-bit sums' rounding
// (no token's logarithm lies below -1e4) or, for decays per channel, a product of decays of at most T tokens: no term overflows.
//
// A step's batch is ragged: entry e owns tokens cu_q[e] .. cu_q[e+1]-1 and state row seq_rows[e].  Chunk c of entry e has the
// place cu_q[e] / T + e + c among the step's chunks (the places of different entries never meet), so that a block finds its
// chunk from the device's arrays alone.
#pragma once
#include "common.cuh"
#include "split_mma.cuh"

namespace se {
namespace walk {

constexpr int kThreads = 256;

__device__ __forceinline__ void cp16(float* dst, const float* src, bool fill) {      // 16 bytes, or zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(fill ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ float fma4(float4 a, float4 b, float c) { return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, c)))); }

__device__ __forceinline__ float softplus32(float v) { return v > 20.f ? v : log1pf(expf(v)); }
template <typename T> __device__ __forceinline__ float value_silu(float v) {
    return sizeof(T) == 2 ? __fdividef(v, 1.f + __expf(-v)) : v / (1.f + expf(-v));
}

// four neighbouring elements as 32-bit values
__device__ __forceinline__ float4 load4(const float* p) { return ld4(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    return make_float4(a.x, a.y, b.x, b.y);
}

// two of them
__device__ __forceinline__ float2 load2(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 load2(const __nv_bfloat16* p) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p)); }

__device__ __forceinline__ void group_sync(int group) { asm volatile("bar.sync %0, 128;" ::"r"(group + 1) : "memory"); }

// A meeting of `THREADS` threads whose warps come from different places in the code (roles, branches that a whole warp takes): the numbered barrier counts
// arrivals from wherever they come, which __syncthreads() does not promise.
template <int THREADS> __device__ __forceinline__ void roles_sync() { asm volatile("bar.sync 5, %0;" ::"n"(THREADS) : "memory"); }

// the entry that owns place `slot` among the step's chunks, and the chunk's first token and length (0: nobody's place)
template <int T>
__device__ __forceinline__ int chunk_of(int slot, const int* cu_q, int entries, int& first, int& n) {
    int lo = 0, hi = entries - 1;
    while (lo < hi) {                                  // the last entry whose first place is at most `slot`
        const int mid = (lo + hi + 1) >> 1;
        if (cu_q[mid] / T + mid <= slot) lo = mid; else hi = mid - 1;
    }
    first = cu_q[lo] + (slot - cu_q[lo] / T - lo) * T;
    n = min(T, cu_q[lo + 1] - first);
    return lo;
}

// A token's log decay, -rate * step, no further down than -1e4: a decay below e^-104 is 0 in 32-bit, and with an infinite rate or step
// the sums would be infinite and their differences NaN.  Sums of 128 such terms differ by less than 2e-9 from what they should.  NaN
// stays NaN.
__device__ __forceinline__ double log_decay(float rate, float step) {
    const double v = -(double)rate * (double)step;
    return v < -1e4 ? -1e4 : v;
}

// The sum of the lanes' `own` (returned) and, in `before`, that of the lanes below: shifted, not the sum less `own`, so that a
// lane's infinity or NaN reaches no prefix but those of the lanes above.
__device__ __forceinline__ double sum_before(double own, int lane, double& before) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double v = __shfl_up_sync(0xffffffffu, own, o);
        if (lane >= o) own += v;
    }
    before = __shfl_up_sync(0xffffffffu, own, 1);
    if (lane == 0) before = 0.0;
    return __shfl_sync(0xffffffffu, own, 31);
}

// ---- the walk ------------------------------------------------------------------------------------
struct WalkArgs {
    const float* q;                // q and k rows: element t * qk_stride + (h / rep) * d (+ k_off)
    const float* k;
    int qk_stride, rep;
    const float* w;                // [tokens][H][d]: solved keys (delta rules)
    const void* v;                 // value rows: element t * v_stride + h * dv, of the kernel's value type
    int v_stride, silu;
    const float* v_scale;          // [tokens][H] a factor on the value rows, or null
    const float* skip;             // per head: o_t += skip * (unscaled) value row, or null
    const float* p;                // [tokens][H][T]
    const float* rs;               // [tokens][H]: factor on q's products with S_0, e^(B_t) (decays per head)
    const float* ts;               // [tokens][H]: factor on u where k takes it into the state, e^(B_n - B_t); not where k comes scaled
    const float* eb;               // [tokens][H]: e^(B_t)
    const float* tot;              // [places][H][d]: e^(B_n)       (decays per channel: q and k come scaled)
    float* state;
    long long state_stride;
    int s_row, s_col;              // state element (row i, column c) of a head at i * s_row + c * s_col
    float* o;                      // [tokens][H][dv]
    const int* cu_q;
    const int* seq_rows;
    int H, d, dv;
};

// Two groups of four warps share a chunk's products, all of them on the tensor cores in tf32 terms (split_mma.cuh).  Without a
// system to solve, group 0 makes the outputs (q S_0, then P u) while group 1 updates the state, which it keeps in registers and
// hands over through a second buffer, and brings the next values: one barrier per chunk.  With one, group 0 makes
// u = U - W S_0 and then the state's update while group 1 makes q S_0 and then the outputs: two barriers.  With chunks of 64 tokens
// and 128 state rows (one block per SM) a third group brings tiles and values, a chunk ahead where there is room for two: the copies, a cp.async
// per 16 bytes, took the other two 1,400 to 2,300 of a chunk's 8,000 to 9,000 cycles.  Elsewhere (two blocks per SM) tiles are copied by the
// warps that read them, as soon as they have read the last chunk's.  Row pitches are such that no fragment read
// meets a bank twice: 8 more than a multiple of 32 where rows lie along k (two neighbours per lane), 4 more than a
// multiple of 16 where columns do.
template <int T, int DP, int C, bool SOLVE, bool SCALED>
struct WalkShape {
    static constexpr int kQP = DP + 8, kKP = DP + 4, kPP = T + 8, kCP = C + 4;
    static constexpr int kBuffers = SOLVE ? 1 : 2;                    // of k, u and the state
    static constexpr bool kLoader = T == 64 && DP == 128;             // a group that only loads
    static constexpr int kThreads = kLoader ? 384 : 256;
    static constexpr int kAhead = kLoader ? 2 : 1;                    // buffers of q and W
    static constexpr int kFloats = (SOLVE ? 2 : 1) * kAhead * T * kQP + kBuffers * T * kKP + T * kPP +
                                   kBuffers * (SCALED ? 1 : 2) * T * kCP + kBuffers * DP * kCP + 2 * T;
    static constexpr int kBlocks = kFloats * 4 <= 112 * 1024 ? 2 : 1;            // per SM
};

// CHANNEL: a decay per key channel; SCALED: k comes as e^(B_n - B_t) k; EXACT: the value rows are 16-bit numbers and nothing else, so
// that products with them need two terms (retention of 8,192 tokens of 32 heads: 541 and 456 us).
template <int T, int DP, int C, bool SOLVE, bool CHANNEL, bool SCALED, bool EXACT, typename TV>
__global__ void __launch_bounds__(WalkShape<T, DP, C, SOLVE, SCALED>::kThreads, WalkShape<T, DP, C, SOLVE, SCALED>::kBlocks)
chunk_walk_kernel(const WalkArgs a) {
    using Shape = WalkShape<T, DP, C, SOLVE, SCALED>;
    constexpr int QP = Shape::kQP, KP = Shape::kKP, PP = Shape::kPP, CP = Shape::kCP, NB = Shape::kBuffers;
    constexpr int QB = Shape::kAhead * T * QP, kThreads = Shape::kThreads;
    constexpr bool LOADER = Shape::kLoader;
    constexpr int WR = T / 16, WC = 4 / WR, NT = C / 8 / WC;          // a warp's outputs: 16 rows, NT tiles of eight columns
    constexpr int MT = DP / 64, NS = C / 8;                           // a warp's state: MT tiles of 16 rows, all columns
    constexpr int NQ = T * C / 4 / 128;                               // quads of the chunk's value columns per thread of a group
    static_assert(SOLVE || T == 64, "without a system a warp has its rows of q and P for itself");
    extern __shared__ __align__(16) float sm[];
    float* qs = sm;                                  // [T][QP], twice with a loading group
    float* ws = qs + QB;                             // W: the same
    float* ks = ws + (SOLVE ? QB : 0);               // [NB][T][KP]
    float* ps = ks + NB * T * KP;                    // [T][PP]
    float* us = ps + T * PP;                         // [NB][T][CP]: u
    float* u2 = SCALED ? us : us + NB * T * CP;      // [NB][T][CP]: e^(B_n - B_t) u, where k does not come with that factor
    float* Ss = u2 + NB * T * CP;                    // [NB][DP][CP]
    float* rss = Ss + NB * DP * CP;                  // [2][T]
    const int e = blockIdx.x, h = blockIdx.y, c0 = blockIdx.z * C;
    const int t_first = a.cu_q[e], t_last = a.cu_q[e + 1];
    if (t_last <= t_first) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lr = lane >> 2, lc = lane & 3;
    const int group = warp >> 2, gw = warp & 3, gt = tid & 127;          // the group, and this thread's place in it
    const int d = a.d, dv = a.dv;
    const int r0 = (gw % WR) * 16 + lr, col0 = (gw / WR) * NT * 8;       // this lane's first row and its warp's first column of outputs
    const int m0 = gw * MT * 16;                                         // the warp's first row of the state

    float* S0 = a.state + (size_t)a.seq_rows[e] * a.state_stride + (size_t)h * d * dv;
    for (int i = tid; i < DP * C; i += kThreads) {   // the faster index in memory runs over neighbouring threads
        const int row = a.s_row == 1 ? i % DP : i / C, c = a.s_row == 1 ? i / DP : i % C;
        Ss[row * CP + c] = row < d && c0 + c < dv ? S0[(size_t)row * a.s_row + (size_t)(c0 + c) * a.s_col] : 0.f;
    }

    // ROWS x COLS floats from (row0, col0) of a chunk's rows to shared memory by `threads` threads, this one being number `who`; rows
    // from n on and columns from `most` on are zeros
    auto load = [&](float* tile, int pitch, const float* src, size_t stride, int t0, int n, int rows, int row0, int cols, int col, int most, int who, int threads) {
#pragma unroll 4
        for (int i = who; i < rows * (cols / 4); i += threads) {
            const int t = row0 + i / (cols / 4), c = col + (i % (cols / 4)) * 4;
            const bool in = t < n && c < most;
            cp16(tile + t * pitch + c, src + (size_t)(t0 + (in ? t : 0)) * stride + (in ? c : 0), in);
        }
    };
    const float* qb = a.q + (size_t)(h / a.rep) * d;
    const float* kb = a.k + (size_t)(h / a.rep) * d;
    const float* wb = SOLVE ? a.w + (size_t)h * d : nullptr;
    const float* pb = a.p + (size_t)h * T;
    const TV* vb = static_cast<const TV*>(a.v) + (size_t)h * dv + c0;
    auto load_k = [&](float* to, int t0, int n) { load(to, KP, kb, a.qk_stride, t0, n, T, 0, DP, 0, d, gt, 128); };
    auto load_p = [&](int t0, int n) {
        if (SOLVE || LOADER) load(ps, PP, pb, (size_t)a.H * T, t0, n, T, 0, T, 0, T, gt, 128);
        else load(ps, PP, pb, (size_t)a.H * T, t0, n, 16, gw * 16, T, 0, T, lane, 32);
    };
    auto load_q = [&](int t0, int n, int buffer = 0) {
        if (SOLVE || LOADER) load(qs + buffer * T * QP, QP, qb, a.qk_stride, t0, n, T, 0, DP, 0, d, gt, 128);
        else load(qs, QP, qb, a.qk_stride, t0, n, 16, gw * 16, DP, 0, d, lane, 32);
    };
    auto load_w = [&](int t0, int n, int buffer = 0) { load(ws + buffer * T * QP, QP, wb, (size_t)a.H * d, t0, n, T, 0, DP, 0, d, gt, 128); };

    // rows of x . S
    auto state_product = [&](const float* x, const float* S, float (&acc)[1][NT][4]) {
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[0][n][j] = 0.f;
        const float* xr = x + r0 * QP + 2 * lc;
        const float* sr = S + 2 * lc * CP + col0 + lr;
        split::products<1, NT, 4>(acc, DP / 8,
            [&](int, int s, float (&v)[4]) {
                const float2 top = *reinterpret_cast<const float2*>(xr + 8 * s), low = *reinterpret_cast<const float2*>(xr + 8 * QP + 8 * s);
                v[0] = top.x; v[1] = low.x; v[2] = top.y; v[3] = low.y;
            },
            [&](int n, int s, float (&v)[2]) { v[0] = sr[8 * s * CP + 8 * n]; v[1] = sr[(8 * s + 1) * CP + 8 * n]; });
        if (split::odd(acc))
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (isfinite(acc[0][n][j])) continue;
                    const float* row = x + (r0 + (j >> 1) * 8) * QP;
                    const float* column = S + col0 + 8 * n + 2 * lc + (j & 1);
                    float sum = 0.f;
#pragma unroll 1
                    for (int k = 0; k < DP; ++k) sum = fmaf(row[k], column[k * CP], sum);
                    acc[0][n][j] = sum;
                }
    };
    // P u; P is zero for s > t
    auto token_product = [&](const float* u, float (&acc)[1][NT][4]) {
        const float* pr = ps + r0 * PP + 2 * lc;
        const float* ur = u + 2 * lc * CP + col0 + lr;
        auto run = [&](bool finite_only, float (&to)[1][NT][4]) {
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int j = 0; j < 4; ++j) to[0][n][j] = 0.f;
            split::products<1, NT, 2, EXACT>(to, 2 * (gw % WR) + 2,
                [&](int, int s, float (&v)[4]) {
                    const float2 top = *reinterpret_cast<const float2*>(pr + 8 * s), low = *reinterpret_cast<const float2*>(pr + 8 * PP + 8 * s);
                    v[0] = top.x; v[1] = low.x; v[2] = top.y; v[3] = low.y;
                },
                [&](int n, int s, float (&v)[2]) {
                    v[0] = ur[8 * s * CP + 8 * n];
                    v[1] = ur[(8 * s + 1) * CP + 8 * n];
                    if (finite_only) {
                        if (!isfinite(v[0])) v[0] = 0.f;
                        if (!isfinite(v[1])) v[1] = 0.f;
                    }
                });
        };
        run(false, acc);
        if (split::odd(acc)) {                       // a token that a row does not see does not touch it, whatever it holds
            float rest[1][NT][4];
            run(true, rest);
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (isfinite(acc[0][n][j])) continue;
                    const int t = r0 + (j >> 1) * 8;
                    const float* column = u + col0 + 8 * n + 2 * lc + (j & 1);
                    float sum = 0.f;
#pragma unroll 1
                    for (int s = 0; s <= t; ++s) sum = fmaf(ps[t * PP + s], column[s * CP], sum);
                    acc[0][n][j] = isfinite(sum) && isfinite(rest[0][n][j]) ? rest[0][n][j] : sum;
                }
        }
    };
    // st = e^(B_n) st + sum_s k_s u_s^T over the warp's rows, and the copy that the other products read
    float st[MT][NS][4];
    auto get_state = [&](const float* from) {
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int n = 0; n < NS; ++n)
#pragma unroll
                for (int j = 0; j < 4; ++j) st[i][n][j] = from[(m0 + 16 * i + lr + (j >> 1) * 8) * CP + 8 * n + 2 * lc + (j & 1)];
    };
    auto put_state = [&](float* to) {
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int n = 0; n < NS; ++n)
#pragma unroll
                for (int j = 0; j < 4; j += 2)
                    *reinterpret_cast<float2*>(to + (m0 + 16 * i + lr + j * 4) * CP + 8 * n + 2 * lc) = make_float2(st[i][n][j], st[i][n][j + 1]);
    };
    auto update_state = [&](const float* k, const float* u, const float (&total)[MT][2]) {
        float sum[MT][NS][4] = {};
        const float* kr = k + 2 * lc * KP + m0 + lr;
        const float* ur = u + 2 * lc * CP + lr;
        split::products<MT, NS, 2, EXACT>(sum, T / 8,
            [&](int i, int s, float (&v)[4]) {
                const float* at = kr + 8 * s * KP + 16 * i;
                v[0] = at[0]; v[1] = at[8]; v[2] = at[KP]; v[3] = at[KP + 8];
            },
            [&](int n, int s, float (&v)[2]) { v[0] = ur[8 * s * CP + 8 * n]; v[1] = ur[(8 * s + 1) * CP + 8 * n]; });
        if (split::odd(sum))
#pragma unroll
            for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int n = 0; n < NS; ++n)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (isfinite(sum[i][n][j])) continue;
                        const float* kc = k + m0 + 16 * i + lr + (j >> 1) * 8;
                        const float* uc = u + 8 * n + 2 * lc + (j & 1);
                        float x = 0.f;
#pragma unroll 1
                        for (int s = 0; s < T; ++s) x = fmaf(kc[s * KP], uc[s * CP], x);
                        sum[i][n][j] = x;
                    }
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int n = 0; n < NS; ++n)
#pragma unroll
                for (int j = 0; j < 4; ++j) st[i][n][j] = fmaf(total[i][j >> 1], st[i][n][j], sum[i][n][j]);
    };
    auto put_outputs = [&](int t0, int n, const float (&acc)[1][NT][4]) {
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
            const int t = r0 + 4 * j;
            if (t >= n) continue;
#pragma unroll
            for (int x = 0; x < NT; ++x) {
                const int c = col0 + 8 * x + 2 * lc;
                if (c0 + c >= dv) continue;
                *reinterpret_cast<float2*>(a.o + ((size_t)(t0 + t) * a.H + h) * dv + c0 + c) = make_float2(acc[0][x][j], acc[0][x][j + 1]);
            }
        }
    };

    const int first_n = min(T, t_last - t_first);
    float* last_state = Ss;
    if constexpr (!SOLVE) {
        // value rows of a chunk, quad by quad, with the factors that go with their tokens
        float4 vreg[NQ];
        float vfac[NQ], tfac[NQ], rfac = 0.f, total = 0.f;
        auto load_v = [&](int t0, int n) {
#pragma unroll
            for (int x = 0; x < NQ; ++x) {
                const int i = x * 128 + gt, t = i / (C / 4), c = (i % (C / 4)) * 4;
                const bool in = t < n && c0 + c < dv;
                const size_t at = (size_t)(t0 + t) * a.H + h;
                vreg[x] = in ? load4(vb + (size_t)(t0 + t) * a.v_stride + c) : make_float4(0.f, 0.f, 0.f, 0.f);
                vfac[x] = in && a.v_scale != nullptr ? a.v_scale[at] : 1.f;
                tfac[x] = !SCALED && in ? a.ts[at] : 1.f;
            }
            if (gt < T) rfac = gt < n ? a.rs[(size_t)(t0 + gt) * a.H + h] : 0.f;
        };
        auto put_values = [&](int buffer) {
#pragma unroll
            for (int x = 0; x < NQ; ++x) {
                const int i = x * 128 + gt, at = (buffer * T + i / (C / 4)) * CP + (i % (C / 4)) * 4;
                float4 v = vreg[x];
                if (a.silu) v = make_float4(value_silu<TV>(v.x), value_silu<TV>(v.y), value_silu<TV>(v.z), value_silu<TV>(v.w));
                v = make_float4(v.x * vfac[x], v.y * vfac[x], v.z * vfac[x], v.w * vfac[x]);
                st4(us + at, v);
                if (!SCALED) st4(u2 + at, make_float4(v.x * tfac[x], v.y * tfac[x], v.z * tfac[x], v.w * tfac[x]));
            }
            if (gt < T) rss[buffer * T + gt] = rfac;
        };
        if (group == (LOADER ? 2 : 0)) {
            load_q(t_first, first_n);
            cp_commit();
            load_p(t_first, first_n);
            cp_commit();
        }
        if (group == (LOADER ? 2 : 1)) {
            load_k(ks, t_first, first_n);
            cp_commit();
            load_v(t_first, first_n);
            put_values(0);
            cp_wait<0>();                            // k (and, with a loading group, q and P)
        }
        if (group == 1) total = a.eb[(size_t)(t_first + first_n - 1) * a.H + h];
        __syncthreads();                             // state, u and factors of the first chunk
        if (group == 1) get_state(Ss);
        const float skip = a.skip != nullptr ? a.skip[h] : 0.f;
        int cur = 0;
        if (LOADER && group == 2) {
            asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
            for (int t0 = t_first; t0 < t_last; t0 += T, cur ^= 1) {
                const int next = t0 + T, next_n = min(T, t_last - next);
                if (t0 > t_first) {
                    cp_wait<0>();
                    asm volatile("bar.arrive 4, 256;" ::: "memory");         // this chunk's P is there
                }
                if (next < t_last) {
                    load_q(next, next_n, cur ^ 1);
                    load_k(ks + (cur ^ 1) * T * KP, next, next_n);
                    cp_commit();
                    load_v(next, next_n);
                    put_values(cur ^ 1);
                    asm volatile("bar.sync 3, 256;" ::: "memory");           // this chunk's P has been read
                    load_p(next, next_n);
                    cp_commit();
                    cp_wait<1>();                    // the next q and k
                }
                roles_sync<kThreads>();
            }
        } else {
        if (LOADER) asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");        // 128 x (2 x 208 + 88): what 384 threads of 168 have
        for (int t0 = t_first; t0 < t_last; t0 += T, cur ^= 1) {
            const int n = min(T, t_last - t0), next = t0 + T, next_n = min(T, t_last - next);
            if (group == 0) {
                float acc[1][NT][4], sum[1][NT][4];
                float2 raw[2][NT];                   // the outputs' own values, where they are added
                if (a.skip != nullptr)
#pragma unroll
                    for (int j = 0; j < 2; ++j)
#pragma unroll
                        for (int x = 0; x < NT; ++x) {
                            const int t = r0 + 8 * j, c = col0 + 8 * x + 2 * lc;
                            raw[j][x] = t < n && c0 + c < dv ? load2(vb + (size_t)(t0 + t) * a.v_stride + c) : make_float2(0.f, 0.f);
                        }
                if constexpr (LOADER) {
                    state_product(qs + cur * T * QP, Ss + cur * DP * CP, acc);
                    if (t0 > t_first) asm volatile("bar.sync 4, 256;" ::: "memory");
                    token_product(us + cur * T * CP, sum);
                    if (next < t_last) asm volatile("bar.arrive 3, 256;" ::: "memory");
                } else {
                    cp_wait<1>();                    // q
                    __syncwarp();
                    state_product(qs, Ss + cur * DP * CP, acc);
                    __syncwarp();
                    if (next < t_last) load_q(next, next_n);
                    cp_commit();
                    cp_wait<1>();                    // P
                    __syncwarp();
                    token_product(us + cur * T * CP, sum);
                    __syncwarp();
                    if (next < t_last) load_p(next, next_n);
                    cp_commit();
                }
#pragma unroll
                for (int x = 0; x < NT; ++x)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[0][x][j] = fmaf(rss[cur * T + r0 + (j >> 1) * 8], acc[0][x][j], sum[0][x][j]);
                if (a.skip != nullptr)
#pragma unroll
                    for (int x = 0; x < NT; ++x)
#pragma unroll
                        for (int j = 0; j < 4; ++j) acc[0][x][j] = fmaf(skip, (j & 1) ? raw[j >> 1][x].y : raw[j >> 1][x].x, acc[0][x][j]);
                put_outputs(t0, n, acc);
            } else {
                const float now = total;
                float totals[MT][2];
#pragma unroll
                for (int i = 0; i < MT; ++i) totals[i][0] = totals[i][1] = now;
                if (next < t_last) {
                    if (!LOADER) {
                        load_k(ks + (cur ^ 1) * T * KP, next, next_n);
                        load_v(next, next_n);
                    }
                    total = a.eb[(size_t)(next + next_n - 1) * a.H + h];
                }
                cp_commit();
                update_state(ks + cur * T * KP, u2 + cur * T * CP, totals);
                put_state(Ss + (cur ^ 1) * DP * CP);
                if (!LOADER && next < t_last) put_values(cur ^ 1);
                cp_wait<0>();                        // the next k
            }
            roles_sync<kThreads>();
        }
        }
        last_state = Ss + cur * DP * CP;
    } else {
        const float* ub = reinterpret_cast<const float*>(vb);
        float ureg[NT][4], fac[2] = {}, totals[MT][2];
        auto load_u = [&](int t0, int n) {           // U where the products' sums lie, and the tokens' factors
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
                const int t = r0 + 4 * j;
#pragma unroll
                for (int x = 0; x < NT; ++x) {
                    const int c = col0 + 8 * x + 2 * lc;
                    const float2 v = t < n && c0 + c < dv ? load2(ub + (size_t)(t0 + t) * a.v_stride + c) : make_float2(0.f, 0.f);
                    ureg[x][j] = v.x;
                    ureg[x][j + 1] = v.y;
                }
            }
        };
        auto load_factors = [&](const float* from, int t0, int n) {
            if (!CHANNEL)
#pragma unroll
                for (int j = 0; j < 2; ++j) fac[j] = r0 + 8 * j < n ? from[(size_t)(t0 + r0 + 8 * j) * a.H + h] : 0.f;
        };
        auto load_totals = [&](int t0, int n) {
#pragma unroll
            for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int row = m0 + 16 * i + lr + 8 * j;
                    totals[i][j] = !CHANNEL ? a.eb[(size_t)(t0 + n - 1) * a.H + h]
                                   : row < d ? a.tot[((size_t)(t_first / T + e + (t0 - t_first) / T) * a.H + h) * d + row] : 0.f;
                }
        };
        if (LOADER ? group == 2 : group == 0) {
            load_w(t_first, first_n);
            if (LOADER) load_q(t_first, first_n);
            cp_commit();
            load_k(ks, t_first, first_n);
            if (LOADER) load_p(t_first, first_n);
        } else if (!LOADER) {
            load_q(t_first, first_n);
            cp_commit();
            load_p(t_first, first_n);
        }
        cp_commit();
        if (group == 0) {
            load_u(t_first, first_n);
            if (!SCALED) load_factors(a.ts, t_first, first_n);
            load_totals(t_first, first_n);
        } else if (group == 1) {
            load_factors(a.rs, t_first, first_n);
        }
        __syncthreads();
        if (group == 0) get_state(Ss);
        int cur = 0;
        if (LOADER && group == 2) {
            asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
            for (int t0 = t_first; t0 < t_last; t0 += T, cur ^= 1) {
                const int n = min(T, t_last - t0), next = t0 + T, next_n = min(T, t_last - next);
                cp_wait<0>();                        // W and q
                roles_sync<kThreads>();              // k and P of the chunk before have been read
                if (t0 > t_first) {
                    load_k(ks, t0, n);
                    load_p(t0, n);
                }
                cp_commit();
                if (next < t_last) {
                    load_w(next, next_n, cur ^ 1);
                    load_q(next, next_n, cur ^ 1);
                }
                cp_commit();
                cp_wait<1>();
                roles_sync<kThreads>();
            }
        } else {
        if (LOADER) asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");        // 128 x (2 x 208 + 88): what 384 threads of 168 have
        for (int t0 = t_first; t0 < t_last; t0 += T, cur ^= LOADER) {
            const int n = min(T, t_last - t0), next = t0 + T, next_n = min(T, t_last - next);
            cp_wait<1>();                            // W or q (k and P may still be on their way)
            roles_sync<kThreads>();                  // and the state is up to date
            float acc[1][NT][4];
            state_product((group == 0 ? ws : qs) + cur * T * QP, Ss, acc);
            if (group == 0) {
#pragma unroll
                for (int x = 0; x < NT; ++x)
#pragma unroll
                    for (int j = 0; j < 4; j += 2) {
                        const float2 u = make_float2(ureg[x][j] - acc[0][x][j], ureg[x][j + 1] - acc[0][x][j + 1]);
                        const int at = (r0 + 4 * j) * CP + col0 + 8 * x + 2 * lc;
                        *reinterpret_cast<float2*>(us + at) = u;
                        if (!SCALED) *reinterpret_cast<float2*>(u2 + at) = make_float2(u.x * fac[j >> 1], u.y * fac[j >> 1]);
                    }
            }
            cp_wait<0>();
            roles_sync<kThreads>();                  // u, k and P are there, W, q and the state have been read
            if (group == 0) {
                if (next < t_last) {
                    if (!LOADER) load_w(next, next_n);
                    load_u(next, next_n);
                    if (!SCALED) load_factors(a.ts, next, next_n);
                }
                cp_commit();
                update_state(ks, u2, totals);
                put_state(Ss);
                if (!LOADER) group_sync(0);
                if (next < t_last) {
                    if (!LOADER) load_k(ks, next, next_n);
                    load_totals(next, next_n);
                }
                cp_commit();
            } else {
                float sum[1][NT][4];
                if (!LOADER && next < t_last) load_q(next, next_n);
                cp_commit();
                token_product(us, sum);
                if (!LOADER) group_sync(1);
                if (!LOADER && next < t_last) load_p(next, next_n);
                cp_commit();
#pragma unroll
                for (int x = 0; x < NT; ++x)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[0][x][j] = CHANNEL ? acc[0][x][j] + sum[0][x][j] : fmaf(fac[j >> 1], acc[0][x][j], sum[0][x][j]);
                if (next < t_last) load_factors(a.rs, next, next_n);
                put_outputs(t0, n, acc);
            }
        }
        }
    }
    cp_wait<0>();
    __syncthreads();
    for (int i = tid; i < DP * C; i += kThreads) {
        const int row = a.s_row == 1 ? i % DP : i / C, c = a.s_row == 1 ? i / DP : i % C;
        if (row < d && c0 + c < dv) S0[(size_t)row * a.s_row + (size_t)(c0 + c) * a.s_col] = last_state[row * CP + c];
    }
}

// ---- what the walk needs, per chunk ---------------------------------------------------------------
// rows r of `src` (element (first + r) * stride + c) into tile [T][DP + PAD]; rows from n on and columns from d to DP are zeros
template <int T, int DP, int PAD>
__device__ __forceinline__ void load_tile(float* tile, const float* src, int stride, int first, int n, int d) {
    constexpr int QP = DP + PAD;
    for (int i = threadIdx.x; i < T * (DP / 4); i += kThreads) {
        const int t = i / (DP / 4), c = (i - t * (DP / 4)) * 4;
        const bool in = t < n && c < d;
        cp16(tile + t * QP + c, src + (size_t)(first + (in ? t : 0)) * stride + (in ? c : 0), in);
    }
}

// Products of 64 rows x[i] (MT matrices) with 64 rows y over DP columns, rows DP + 8 floats apart, where the row of y is not after the
// row of x: eight warps share out the tiles of 16 x 8 on and below the diagonal, ten to each scheduler's two.  use(acc, r0, n0,
// first zero column): acc[i][n] holds (row r0, columns n0 + 8 n and the one after it), then the same of row r0 + 8.  Multiply-adds on
// 4 x 4 outputs a thread were bound by their reads from shared memory.
template <int DP, int MT, int NT, typename Use>
__device__ __forceinline__ void triangle_tiles(const float* const (&x)[MT], const float* y, int block, int half, int lane, Use use) {
    constexpr int QP = DP + 8;
    const int lr = lane >> 2, lc = lane & 3, r0 = block * 16 + lr, n0 = half * NT * 8;
    const float* yr = y + (n0 + lr) * QP + 2 * lc;
    float acc[MT][NT][4] = {};
    split::products<MT, NT, 2>(acc, DP / 8,
        [&](int i, int s, float (&v)[4]) {
            const float* at = x[i] + r0 * QP + 2 * lc + 8 * s;
            const float2 top = *reinterpret_cast<const float2*>(at), low = *reinterpret_cast<const float2*>(at + 8 * QP);
            v[0] = top.x; v[1] = low.x; v[2] = top.y; v[3] = low.y;
        },
        [&](int n, int s, float (&v)[2]) {
            const float2 w = *reinterpret_cast<const float2*>(yr + 8 * n * QP + 8 * s);
            v[0] = w.x; v[1] = w.y;
        });
    if (split::odd(acc))
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (isfinite(acc[i][n][j])) continue;
                    const float* row = x[i] + (r0 + (j >> 1) * 8) * QP;
                    const float* other = y + (n0 + 8 * n + 2 * lc + (j & 1)) * QP;
                    float sum = 0.f;
#pragma unroll 1
                    for (int k = 0; k < DP; ++k) sum = fmaf(row[k], other[k], sum);
                    acc[i][n][j] = sum;
                }
    use(acc, r0, n0 + 2 * lc, (block + 1) * 16 + half * 8 + 2 * lc);
}
template <int DP, int MT, typename Use>
__device__ __forceinline__ void triangle_products(const float* const (&x)[MT], const float* y, int warp, int lane, Use use) {
    const int half = warp & 1;
    switch (warp >> 1) {
        case 0: triangle_tiles<DP, MT, 4>(x, y, 3, half, lane, use); break;
        case 1: triangle_tiles<DP, MT, 3>(x, y, 2, half, lane, use); break;
        case 2: triangle_tiles<DP, MT, 1>(x, y, 0, half, lane, use); break;
        default: triangle_tiles<DP, MT, 2>(x, y, 1, half, lane, use);
    }
}

// ---- launches ------------------------------------------------------------------------------------
template <typename... KArgs, typename... Args>
int launch_threads(void (*kernel)(KArgs...), dim3 grid, int threads, size_t smem, cudaStream_t stream, Args... args) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    kernel<<<grid, threads, smem, stream>>>(KArgs(args)...);
    return (int)cudaGetLastError();
}
template <typename... KArgs, typename... Args>
int launch(void (*kernel)(KArgs...), dim3 grid, size_t smem, cudaStream_t stream, Args... args) {
    return launch_threads(kernel, grid, kThreads, smem, stream, args...);
}
template <int T, int DP, int C, bool SOLVE, bool CHANNEL, bool SCALED, bool EXACT, typename TV>
int launch_walk_columns(const WalkArgs& a, int entries, cudaStream_t stream) {
    using Shape = WalkShape<T, DP, C, SOLVE, SCALED>;
    return launch_threads(chunk_walk_kernel<T, DP, C, SOLVE, CHANNEL, SCALED, EXACT, TV>, dim3(entries, a.H, ceil_div(a.dv, C)), Shape::kThreads,
                          Shape::kFloats * sizeof(float), stream, a);
}
template <int T, int DP, bool SOLVE, bool CHANNEL, bool SCALED, bool EXACT, typename TV>
int launch_walk(const WalkArgs& a, int entries, int cols, cudaStream_t stream) {
    if (cols == 16) return launch_walk_columns<T, DP, 16, SOLVE, CHANNEL, SCALED, EXACT, TV>(a, entries, stream);
    return launch_walk_columns<T, DP, 32, SOLVE, CHANNEL, SCALED, EXACT, TV>(a, entries, stream);
}

// Value columns per block: 32 while the blocks then fill the device, 16 (twice the blocks, which each read q and k) else.
inline int walk_columns(long long entries, int H, int dv, int sms) { return entries * H * ((dv + 31) / 32) >= sms * 4 / 5 ? 32 : 16; }

inline bool takes(int d, int dv) { return d >= 8 && d <= 128 && d % 4 == 0 && dv >= 4 && dv % 4 == 0; }
inline bool aligned(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

#define SE_WALK_DIMS(d, ...)                                 \
    if ((d) <= 64) { constexpr int DP = 64; __VA_ARGS__; }   \
    else { constexpr int DP = 128; __VA_ARGS__; }

}  // namespace walk
}  // namespace se

