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
//
// What bounds them is the FMA rate (3 to 5 multiply-adds per state element and token); a tensor-core form would need
// 16-bit or split operands.  Every exponent is a difference of sums of logarithms that is at most 0 (sums in 64-bit) or, for
// decays per channel, a product of decays of at most T tokens: no term overflows.
//
// A step's batch is ragged: entry e owns tokens cu_q[e] .. cu_q[e+1]-1 and state row seq_rows[e].  Chunk c of entry e has the
// place cu_q[e] / T + e + c among the step's chunks (the places of different entries never meet), so that a block finds its
// chunk from the device's arrays alone.
#pragma once
#include "common.cuh"

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
    const float* rs;               // [tokens][H]: e^(B_t)          (decays per head)
    const float* ts;               // [tokens][H]: e^(B_n - B_t)
    const float* tot;              // [places][H][d]: e^(B_n)       (decays per channel: q and k come scaled)
    float* state;
    long long state_stride;
    int s_row, s_col;              // state element (row i, column c) of a head at i * s_row + c * s_col
    float* o;                      // [tokens][H][dv]
    const int* cu_q;
    const int* seq_rows;
    int H, d, dv;
};

template <int T, int DP, int C, bool SOLVE, bool CHANNEL>
struct WalkShape {
    static constexpr int kRowSplit = T == 64 && C == 32 ? 2 : 1;      // row halves of the products with the state ...
    static constexpr int kSlices = 8 / kRowSplit;                     // ... and slices of their inner dimension, per warp
    static constexpr int kTimeSplit = 8 / (DP / 32);                  // slices of the tokens in the state's update
    static constexpr int kQP = DP + 4, kPP = T + 4;
    static constexpr int kFloats = (SOLVE ? 3 : 2) * T * kQP + T * kPP + 2 * T * C + DP * C + kSlices * T * C +
                                   (kTimeSplit - 1) * DP * C + 2 * T + (CHANNEL ? DP : 0);
};

template <int T, int DP, int C, bool SOLVE, bool CHANNEL, typename TV>
__global__ void __launch_bounds__(kThreads, 1)
chunk_walk_kernel(const WalkArgs a) {
    using Shape = WalkShape<T, DP, C, SOLVE, CHANNEL>;
    constexpr int QP = Shape::kQP, PP = Shape::kPP, KS = Shape::kSlices, TS = Shape::kTimeSplit;
    constexpr int RM = T / 8 / Shape::kRowSplit, RC = C / 4;           // rows and columns of a thread's output tile
    constexpr int NV = (T * C / 4 + kThreads - 1) / kThreads;          // value quads per thread
    extern __shared__ __align__(16) float sm[];
    float* qs = sm;                                  // [T][QP]
    float* ks = qs + T * QP;                         // [T][QP]
    float* ws = ks + T * QP;                         // [T][QP]
    float* ps = ws + (SOLVE ? T * QP : 0);           // [T][PP]
    float* us = ps + T * PP;                         // [T][C]: u
    float* u2 = us + T * C;                          // [T][C]: e^(B_n - B_t) u (decays per head)
    float* Ss = u2 + T * C;                          // [DP][C]
    float* part = Ss + DP * C;                       // [KS][T][C]
    float* part2 = part + KS * T * C;                // [TS - 1][DP][C]
    float* rss = part2 + (TS - 1) * DP * C;          // [T]
    float* tss = rss + T;                            // [T]
    float* tots = tss + T;                           // [DP]
    const int e = blockIdx.x, h = blockIdx.y, c0 = blockIdx.z * C;
    const int t_first = a.cu_q[e], t_last = a.cu_q[e + 1];
    if (t_last <= t_first) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lr = lane >> 2, lc = lane & 3;
    const int d = a.d, dv = a.dv;
    const int d4 = d / 4;

    // columns of q, k and w beyond d, once; the loads below never touch them
    if (d < DP)
        for (int i = tid; i < (SOLVE ? 3 : 2) * T * (DP - d); i += kThreads) {
            const int r = i / (DP - d);
            qs[r * QP + d + i - r * (DP - d)] = 0.f;
        }
    float* S0 = a.state + (size_t)a.seq_rows[e] * a.state_stride + (size_t)h * d * dv;
    for (int i = tid; i < DP * C; i += kThreads) {   // the faster index in memory runs over neighbouring threads
        const int row = a.s_row == 1 ? i % DP : i / C, c = a.s_row == 1 ? i / DP : i % C;
        Ss[row * C + c] = row < d && c0 + c < dv ? S0[(size_t)row * a.s_row + (size_t)(c0 + c) * a.s_col] : 0.f;
    }

    const float* qb = a.q + (size_t)(h / a.rep) * d;
    const float* kb = a.k + (size_t)(h / a.rep) * d;
    auto load_qw = [&](int t0, int n) {
        for (int i = tid; i < T * d4; i += kThreads) {
            const int t = i / d4, c = (i - t * d4) * 4;
            const size_t row = (size_t)(t0 + (t < n ? t : 0));
            cp16(qs + t * QP + c, qb + row * a.qk_stride + c, t < n);
            if (SOLVE) cp16(ws + t * QP + c, a.w + (row * a.H + h) * d + c, t < n);
        }
        cp_commit();
    };
    auto load_kp = [&](int t0, int n) {
        for (int i = tid; i < T * d4; i += kThreads) {
            const int t = i / d4, c = (i - t * d4) * 4;
            cp16(ks + t * QP + c, kb + (size_t)(t0 + (t < n ? t : 0)) * a.qk_stride + c, t < n);
        }
        for (int i = tid; i < T * (T / 4); i += kThreads) {
            const int t = i / (T / 4), c = (i - t * (T / 4)) * 4;
            cp16(ps + t * PP + c, a.p + ((size_t)(t0 + (t < n ? t : 0)) * a.H + h) * T + c, t < n);
        }
        cp_commit();
    };
    // values (a quad per place i * kThreads + tid) and per-token factors of a chunk, in registers until they are wanted
    const TV* vb = static_cast<const TV*>(a.v) + (size_t)h * dv + c0;
    float4 vreg[NV];
    float fac = 0.f, vfac[NV];
    auto load_v = [&](int t0, int n) {
#pragma unroll
        for (int x = 0; x < NV; ++x) {
            const int i = x * kThreads + tid, t = i / (C / 4), c = (i - t * (C / 4)) * 4;
            const bool in = i < T * C / 4 && t < n && c0 + c < dv;
            vreg[x] = in ? load4(vb + (size_t)(t0 + t) * a.v_stride + c) : make_float4(0.f, 0.f, 0.f, 0.f);
            vfac[x] = in && a.v_scale != nullptr ? a.v_scale[(size_t)(t0 + t) * a.H + h] : 1.f;
        }
        if (!CHANNEL && tid < 2 * T) {
            const int t = tid < T ? tid : tid - T;
            fac = t < n ? (tid < T ? a.rs : a.ts)[(size_t)(t0 + t) * a.H + h] : 0.f;
        }
        if (CHANNEL && tid < d) fac = a.tot[((size_t)(t_first / T + e + (t0 - t_first) / T) * a.H + h) * d + tid];
    };
    const float skip = a.skip != nullptr ? a.skip[h] : 0.f;

    const int first_n = min(T, t_last - t_first);
    load_qw(t_first, first_n);
    load_kp(t_first, first_n);
    load_v(t_first, first_n);
    const int slice = warp / Shape::kRowSplit, r0 = (warp % Shape::kRowSplit) * (T / Shape::kRowSplit);
    for (int t0 = t_first; t0 < t_last; t0 += T) {
        const int n = min(T, t_last - t0), next = t0 + T, next_n = min(T, t_last - next);
        float4 raw[NV];                              // the value rows as they are (or the solved U)
#pragma unroll
        for (int x = 0; x < NV; ++x) {
            raw[x] = vreg[x];
            if (a.silu) raw[x] = make_float4(value_silu<TV>(raw[x].x), value_silu<TV>(raw[x].y), value_silu<TV>(raw[x].z), value_silu<TV>(raw[x].w));
        }
        int odd = 0;                                 // a value that is not finite
        if (!CHANNEL && tid < 2 * T) (tid < T ? rss : tss - T)[tid] = fac;
        if (CHANNEL && tid < DP) tots[tid] = tid < d ? fac : 0.f;
        auto put_u = [&](int x, float4 u, float after) {     // u and e^(B_n - B_t) u of one quad
            const int i = x * kThreads + tid;
            if (i >= T * C / 4) return;
            odd |= !(isfinite(u.x) && isfinite(u.y) && isfinite(u.z) && isfinite(u.w));
            st4(us + i * 4, u);
            if (!CHANNEL) st4(u2 + i * 4, make_float4(u.x * after, u.y * after, u.z * after, u.w * after));
        };
        cp_wait<1>();                                // this chunk's q and w
        __syncthreads();                             // (and the state is up to date)
        if (!SOLVE)
#pragma unroll
            for (int x = 0; x < NV; ++x) {
                const int t = (x * kThreads + tid) / (C / 4);
                put_u(x, make_float4(raw[x].x * vfac[x], raw[x].y * vfac[x], raw[x].z * vfac[x], raw[x].w * vfac[x]), CHANNEL || t >= T ? 1.f : tss[t]);
            }
        // products with the state: a warp takes T (or T/2) rows, all columns and a slice of the inner dimension
        float acc[RM][RC] = {}, accw[SOLVE ? RM : 1][RC] = {};
#pragma unroll 2
        for (int k = slice * (DP / KS); k < (slice + 1) * (DP / KS); k += 4) {
            float sv[4][RC];
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int g = 0; g < RC / 4; ++g) *reinterpret_cast<float4*>(&sv[j][4 * g]) = ld4(Ss + (k + j) * C + 16 * g + lc * 4);
#pragma unroll
            for (int i = 0; i < RM; ++i) {
                const float4 qv = ld4(qs + (r0 + lr + 8 * i) * QP + k);
#pragma unroll
                for (int c = 0; c < RC; ++c) acc[i][c] = fmaf(qv.w, sv[3][c], fmaf(qv.z, sv[2][c], fmaf(qv.y, sv[1][c], fmaf(qv.x, sv[0][c], acc[i][c]))));
                if (SOLVE) {
                    const float4 wv = ld4(ws + (r0 + lr + 8 * i) * QP + k);
#pragma unroll
                    for (int c = 0; c < RC; ++c) accw[i][c] = fmaf(wv.w, sv[3][c], fmaf(wv.z, sv[2][c], fmaf(wv.y, sv[1][c], fmaf(wv.x, sv[0][c], accw[i][c]))));
                }
            }
        }
        auto put_part = [&](const float (*v)[RC]) {
#pragma unroll
            for (int i = 0; i < RM; ++i)
#pragma unroll
                for (int g = 0; g < RC / 4; ++g)
                    st4(part + (slice * T + r0 + lr + 8 * i) * C + 16 * g + lc * 4, make_float4(v[i][4 * g], v[i][4 * g + 1], v[i][4 * g + 2], v[i][4 * g + 3]));
        };
        auto sum_part = [&](int x) {                 // the sum over the slices of one quad
            const int i = x * kThreads + tid;
            float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
            if (i < T * C / 4)
#pragma unroll
                for (int z = 0; z < KS; ++z) {
                    const float4 v = ld4(part + z * T * C + i * 4);
                    s = make_float4(s.x + v.x, s.y + v.y, s.z + v.z, s.w + v.w);
                }
            return s;
        };
        if (SOLVE) put_part(accw);
        cp_wait<0>();                                // this chunk's k and P
        if (SOLVE) {
            __syncthreads();
#pragma unroll
            for (int x = 0; x < NV; ++x) {
                const int t = (x * kThreads + tid) / (C / 4);
                const float4 s = sum_part(x);
                put_u(x, make_float4(raw[x].x - s.x, raw[x].y - s.y, raw[x].z - s.z, raw[x].w - s.w), CHANNEL || t >= T ? 1.f : tss[t]);
            }
        }
        odd = __syncthreads_or(odd);
        if (next < t_last) {                         // q and w have been read: the next chunk's follow
            load_qw(next, next_n);
            load_v(next, next_n);
        } else {
            cp_commit();
        }
        // what the chunk's own tokens add: P u, a slice of the tokens s per warp; P is zero for s > t
        if (!CHANNEL)
#pragma unroll
            for (int i = 0; i < RM; ++i) {
                const float f = rss[r0 + lr + 8 * i];
#pragma unroll
                for (int c = 0; c < RC; ++c) acc[i][c] *= f;
            }
        auto add_tokens = [&](bool guarded) {
#pragma unroll
            for (int sq = 0; sq < T / KS; sq += 4) {
                const int s = slice * (T / KS) + sq;
                float uv[4][RC];
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int g = 0; g < RC / 4; ++g) *reinterpret_cast<float4*>(&uv[j][4 * g]) = ld4(us + (s + j) * C + 16 * g + lc * 4);
#pragma unroll
                for (int i = 0; i < RM; ++i) {
                    if (r0 + 8 * i + 7 < s) continue;        // rows before these tokens
                    const int t = r0 + lr + 8 * i;
                    const float4 pv = ld4(ps + t * PP + s);
                    const float p4[4] = {pv.x, pv.y, pv.z, pv.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j)
#pragma unroll
                        for (int c = 0; c < RC; ++c)
                            if (!guarded || s + j <= t) acc[i][c] = fmaf(p4[j], uv[j][c], acc[i][c]);
                }
            }
        };
        if (odd) add_tokens(true);                   // a token that a row does not see does not touch it, whatever it holds
        else add_tokens(false);
        put_part(acc);
        // the state's update: a warp takes 32 rows, all columns and a slice of the tokens
        const int dg = warp % (DP / 32), tsl = warp / (DP / 32), row0 = dg * 32 + lr * 4;
        const float* uu = CHANNEL ? us : u2;
        float st[4][RC] = {};
#pragma unroll 4
        for (int s = tsl * (T / TS); s < (tsl + 1) * (T / TS); ++s) {
            const float4 kv = ld4(ks + s * QP + row0);
            const float k4[4] = {kv.x, kv.y, kv.z, kv.w};
            float uv[RC];
#pragma unroll
            for (int g = 0; g < RC / 4; ++g) *reinterpret_cast<float4*>(&uv[4 * g]) = ld4(uu + s * C + 16 * g + lc * 4);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int c = 0; c < RC; ++c) st[i][c] = fmaf(k4[i], uv[c], st[i][c]);
        }
        if (tsl > 0)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int g = 0; g < RC / 4; ++g)
                    st4(part2 + ((tsl - 1) * DP + row0 + i) * C + 16 * g + lc * 4, make_float4(st[i][4 * g], st[i][4 * g + 1], st[i][4 * g + 2], st[i][4 * g + 3]));
        const float total = CHANNEL ? 0.f : rss[n - 1];
        __syncthreads();                             // k, P, u and the old state have been read; the partial sums are there
        if (next < t_last) load_kp(next, next_n);
        else cp_commit();
#pragma unroll
        for (int x = 0; x < NV; ++x) {
            const int i = x * kThreads + tid, t = i / (C / 4), c = (i - t * (C / 4)) * 4;
            if (i < T * C / 4 && t < n && c0 + c < dv) {
                const float4 s = sum_part(x);
                st4(a.o + ((size_t)(t0 + t) * a.H + h) * dv + c0 + c,
                    make_float4(s.x + skip * raw[x].x, s.y + skip * raw[x].y, s.z + skip * raw[x].z, s.w + skip * raw[x].w));
            }
        }
        if (tsl == 0)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int g = 0; g < RC / 4; ++g) {
                    const int at = (row0 + i) * C + 16 * g + lc * 4;
                    const float f = CHANNEL ? tots[row0 + i] : total;
                    float4 s = ld4(Ss + at);
                    s = make_float4(fmaf(f, s.x, st[i][4 * g]), fmaf(f, s.y, st[i][4 * g + 1]), fmaf(f, s.z, st[i][4 * g + 2]), fmaf(f, s.w, st[i][4 * g + 3]));
#pragma unroll
                    for (int z = 0; z < TS - 1; ++z) {
                        const float4 v = ld4(part2 + z * DP * C + at);
                        s = make_float4(s.x + v.x, s.y + v.y, s.z + v.z, s.w + v.w);
                    }
                    st4(Ss + at, s);
                }
    }
    __syncthreads();
    for (int i = tid; i < DP * C; i += kThreads) {
        const int row = a.s_row == 1 ? i % DP : i / C, c = a.s_row == 1 ? i / DP : i % C;
        if (row < d && c0 + c < dv) S0[(size_t)row * a.s_row + (size_t)(c0 + c) * a.s_col] = Ss[row * C + c];
    }
}

// ---- what the walk needs, per chunk ---------------------------------------------------------------
// rows r of `src` (element (first + r) * stride + c) into tile [T][QP]; rows from n on and columns from d to DP are zeros
template <int T, int DP>
__device__ __forceinline__ void load_tile(float* tile, const float* src, int stride, int first, int n, int d) {
    constexpr int QP = DP + 4;
    for (int i = threadIdx.x; i < T * (DP / 4); i += kThreads) {
        const int t = i / (DP / 4), c = (i - t * (DP / 4)) * 4;
        const bool in = t < n && c < d;
        cp16(tile + t * QP + c, src + (size_t)(first + (in ? t : 0)) * stride + (in ? c : 0), in);
    }
}

// acc[a][b] += rows (ty * M + a) of x . rows (tx * M + b) of y, over DP columns
template <int DP, int M>
__device__ __forceinline__ void row_products(const float* x, const float* y, int ty, int tx, float (*acc)[M]) {
    constexpr int QP = DP + 4;
#pragma unroll 4
    for (int k = 0; k < DP; k += 4) {
        float4 yv[M];
#pragma unroll
        for (int b = 0; b < M; ++b) yv[b] = ld4(y + (tx + 16 * b) * QP + k);
#pragma unroll
        for (int i = 0; i < M; ++i) {
            const float4 xv = ld4(x + (ty + 16 * i) * QP + k);
#pragma unroll
            for (int b = 0; b < M; ++b) acc[i][b] = fma4(xv, yv[b], acc[i][b]);
        }
    }
}

// ---- launches ------------------------------------------------------------------------------------
template <typename... KArgs, typename... Args>
int launch(void (*kernel)(KArgs...), dim3 grid, size_t smem, cudaStream_t stream, Args... args) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    kernel<<<grid, kThreads, smem, stream>>>(KArgs(args)...);
    return (int)cudaGetLastError();
}

template <int T, int DP, bool SOLVE, bool CHANNEL, typename TV>
int launch_walk(const WalkArgs& a, int entries, int cols, cudaStream_t stream) {
    const dim3 grid(entries, a.H, ceil_div(a.dv, cols));
    if (cols == 16)
        return launch(chunk_walk_kernel<T, DP, 16, SOLVE, CHANNEL, TV>, grid, WalkShape<T, DP, 16, SOLVE, CHANNEL>::kFloats * sizeof(float), stream, a);
    return launch(chunk_walk_kernel<T, DP, 32, SOLVE, CHANNEL, TV>, grid, WalkShape<T, DP, 32, SOLVE, CHANNEL>::kFloats * sizeof(float), stream, a);
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

