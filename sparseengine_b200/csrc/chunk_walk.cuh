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
// 16-bit or split operands.  Every exponent is a difference of sums of logarithms that is at most 0 up to the 64-bit sums' rounding
// (no token's logarithm lies below -1e4) or, for decays per channel, a product of decays of at most T tokens: no term overflows.
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
    const float* rs;               // [tokens][H]: factor on q's products with S_0, e^(B_t) (decays per head)
    const float* ts;               // [tokens][H]: factor on u where k takes it into the state, e^(B_n - B_t)
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

// Two groups of four warps share a chunk's products.  Without a system to solve, group 0 makes the outputs (q S_0, then P u, in
// four slices) while group 1 sums and stores those of the chunk before, updates the state into a second buffer and brings the
// next values: one barrier for all per chunk, and one at which group 1 only arrives.  With one, group 0 makes u = U - W S_0 and then the state's update while group 1 makes q S_0 and then the
// outputs: two barriers.  A thread holds T / 8 rows x C / 4 columns of its warp's slice (8 x 8 at best: an FMA costs a quarter of
// a shared-memory wavefront then, and both units are as busy).  q, k, P and W of the next chunk are copied as soon as the last
// reader of this one's has passed.
template <int T, int DP, int C, bool SOLVE, bool CHANNEL>
struct WalkShape {
    static constexpr int kSlices = 4;                                 // of the inner dimension (or the tokens), a warp each
    static constexpr int kRowGroups = DP / 64;                        // 64 rows of the state per warp ...
    static constexpr int kTimeSplit = 4 / kRowGroups;                 // ... and a slice of the tokens
    static constexpr int kQP = DP + 4, kPP = T + 4;
    static constexpr int kFloats = 3 * T * kQP + T * kPP + (SOLVE ? 2 : 3) * T * C + (SOLVE ? 1 : 2) * DP * C +
                                   kSlices * T * C + (kTimeSplit - 1) * DP * C + 2 * T + (CHANNEL ? DP : 0);
};

__device__ __forceinline__ void group_sync(int group) { asm volatile("bar.sync %0, 128;" ::"r"(group + 1) : "memory"); }

template <int T, int DP, int C, bool SOLVE, bool CHANNEL, typename TV>
__global__ void __launch_bounds__(kThreads, 1)
chunk_walk_kernel(const WalkArgs a) {
    using Shape = WalkShape<T, DP, C, SOLVE, CHANNEL>;
    constexpr int QP = Shape::kQP, PP = Shape::kPP, KS = Shape::kSlices, TS = Shape::kTimeSplit, RG = Shape::kRowGroups;
    constexpr int RM = T / 8, RC = C / 4;            // rows and columns of a thread's output tile
    constexpr int NQ = T * C / 4 / 128;              // quads of the chunk's value columns per thread of a group
    extern __shared__ __align__(16) float sm[];
    float* qs = sm;                                  // [T][QP]
    float* ks = qs + T * QP;                         // [T][QP], twice without a system to solve
    float* ws = ks + T * QP;                         // [T][QP]: W, or the second k
    float* ps = ws + T * QP;                         // [T][PP]
    float* us = ps + T * PP;                         // [T][C]: u; twice without a system to solve
    float* u2 = us + (SOLVE ? 1 : 2) * T * C;        // [T][C]: e^(B_n - B_t) u (decays per head)
    float* Ss = u2 + T * C;                          // [DP][C]; twice without a system to solve
    float* part = Ss + (SOLVE ? 1 : 2) * DP * C;     // [KS][T][C]
    float* part2 = part + KS * T * C;                // [TS - 1][DP][C]
    float* rss = part2 + (TS - 1) * DP * C;          // [2][T]
    float* tots = rss + 2 * T;                       // [DP]
    const int e = blockIdx.x, h = blockIdx.y, c0 = blockIdx.z * C;
    const int t_first = a.cu_q[e], t_last = a.cu_q[e + 1];
    if (t_last <= t_first) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lr = lane >> 2, lc = lane & 3;
    const int group = warp >> 2, gw = warp & 3, gt = tid & 127;          // the group, and this thread's place in it
    const int d = a.d, dv = a.dv;

    float* S0 = a.state + (size_t)a.seq_rows[e] * a.state_stride + (size_t)h * d * dv;
    for (int i = tid; i < DP * C; i += kThreads) {   // the faster index in memory runs over neighbouring threads
        const int row = a.s_row == 1 ? i % DP : i / C, c = a.s_row == 1 ? i / DP : i % C;
        Ss[row * C + c] = row < d && c0 + c < dv ? S0[(size_t)row * a.s_row + (size_t)(c0 + c) * a.s_col] : 0.f;
    }

    // T rows of d columns to shared memory by one group; rows from n on and columns from d on are zeros
    auto load_rows = [&](float* tile, const float* src, size_t stride, int t0, int n) {
#pragma unroll 4
        for (int i = gt; i < T * (DP / 4); i += 128) {
            const int t = i / (DP / 4), c = (i % (DP / 4)) * 4;
            const bool in = t < n && c < d;
            cp16(tile + t * QP + c, src + (size_t)(t0 + (in ? t : 0)) * stride + (in ? c : 0), in);
        }
    };
    auto load_p = [&](int t0, int n) {
#pragma unroll 4
        for (int i = gt; i < T * (T / 4); i += 128) {
            const int t = i / (T / 4), c = (i % (T / 4)) * 4;
            cp16(ps + t * PP + c, a.p + ((size_t)(t0 + (t < n ? t : 0)) * a.H + h) * T + c, t < n);
        }
    };
    const float* qb = a.q + (size_t)(h / a.rep) * d;
    const float* kb = a.k + (size_t)(h / a.rep) * d;
    const float* wb = SOLVE ? a.w + (size_t)h * d : nullptr;
    const TV* vb = static_cast<const TV*>(a.v) + (size_t)h * dv + c0;
    // value rows (or U) of a chunk, quad by quad, with the factors that go with their tokens
    float4 vreg[NQ];
    float vfac[NQ], tfac[NQ], rfac = 0.f;
    auto load_v = [&](int t0, int n) {
#pragma unroll
        for (int x = 0; x < NQ; ++x) {
            const int i = x * 128 + gt, t = i / (C / 4), c = (i % (C / 4)) * 4;
            const bool in = t < n && c0 + c < dv;
            const size_t at = (size_t)(t0 + t) * a.H + h;
            vreg[x] = in ? load4(vb + (size_t)(t0 + t) * a.v_stride + c) : make_float4(0.f, 0.f, 0.f, 0.f);
            vfac[x] = !SOLVE && in && a.v_scale != nullptr ? a.v_scale[at] : 1.f;
            tfac[x] = !CHANNEL && in ? a.ts[at] : 1.f;
        }
    };
    auto load_factors = [&](int t0, int n) {         // e^(B_t) of the chunk's tokens, or e^(B_n) of the channels
        if (!CHANNEL && gt < T) rfac = gt < n ? a.rs[(size_t)(t0 + gt) * a.H + h] : 0.f;
        if (CHANNEL) rfac = gt < d ? a.tot[((size_t)(t_first / T + e + (t0 - t_first) / T) * a.H + h) * d + gt] : 0.f;
    };
    int odd = 0;                                     // a value that is not finite
    auto put_u = [&](int x, float4 u, float* to) {   // u and e^(B_n - B_t) u of one quad
        const int i = x * 128 + gt;
        odd |= !(isfinite(u.x) && isfinite(u.y) && isfinite(u.z) && isfinite(u.w));
        st4(to + i * 4, u);
        if (!CHANNEL) st4(u2 + i * 4, make_float4(u.x * tfac[x], u.y * tfac[x], u.z * tfac[x], u.w * tfac[x]));
    };
    auto put_values = [&](float* to) {
#pragma unroll
        for (int x = 0; x < NQ; ++x) {
            float4 v = vreg[x];
            if (a.silu) v = make_float4(value_silu<TV>(v.x), value_silu<TV>(v.y), value_silu<TV>(v.z), value_silu<TV>(v.w));
            put_u(x, make_float4(v.x * vfac[x], v.y * vfac[x], v.z * vfac[x], v.w * vfac[x]), to);
        }
    };
    // acc = rows of x . S, a warp's slice of the inner dimension
    auto state_product = [&](const float* x, const float* S, float (&acc)[RM][RC]) {
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
            for (int c = 0; c < RC; ++c) acc[i][c] = 0.f;
#pragma unroll 2
        for (int k = gw * (DP / KS); k < (gw + 1) * (DP / KS); k += 4) {
            float sv[4][RC];
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int g = 0; g < RC / 4; ++g) *reinterpret_cast<float4*>(&sv[j][4 * g]) = ld4(S + (k + j) * C + 16 * g + lc * 4);
#pragma unroll
            for (int i = 0; i < RM; ++i) {
                const float4 v = ld4(x + (lr + 8 * i) * QP + k);
#pragma unroll
                for (int c = 0; c < RC; ++c) acc[i][c] = fmaf(v.w, sv[3][c], fmaf(v.z, sv[2][c], fmaf(v.y, sv[1][c], fmaf(v.x, sv[0][c], acc[i][c]))));
            }
        }
    };
    auto put_part = [&](const float (&v)[RM][RC]) {
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
            for (int g = 0; g < RC / 4; ++g)
                st4(part + (gw * T + lr + 8 * i) * C + 16 * g + lc * 4, make_float4(v[i][4 * g], v[i][4 * g + 1], v[i][4 * g + 2], v[i][4 * g + 3]));
    };
    auto sum_part = [&](int x) {                     // the sum over the slices of one quad
        float4 s = ld4(part + (x * 128 + gt) * 4);
#pragma unroll
        for (int z = 1; z < KS; ++z) {
            const float4 v = ld4(part + z * T * C + (x * 128 + gt) * 4);
            s = make_float4(s.x + v.x, s.y + v.y, s.z + v.z, s.w + v.w);
        }
        return s;
    };
    // acc = e^(B_t) acc + P u, a warp's slice of the tokens s; P is zero for s > t
    auto add_tokens = [&](const float* u, const float* factors, int any_odd, float (&acc)[RM][RC]) {
        if (!CHANNEL)
#pragma unroll
            for (int i = 0; i < RM; ++i) {
                const float f = factors[lr + 8 * i];
#pragma unroll
                for (int c = 0; c < RC; ++c) acc[i][c] *= f;
            }
        auto run = [&](bool guarded) {
#pragma unroll 1
            for (int s = 4 * gw; s < T; s += 4 * KS) {           // dealt out in turn: early tokens have more rows
                float uv[4][RC];
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int g = 0; g < RC / 4; ++g) *reinterpret_cast<float4*>(&uv[j][4 * g]) = ld4(u + (s + j) * C + 16 * g + lc * 4);
#pragma unroll
                for (int i = 0; i < RM; ++i) {
                    if (8 * i + 7 < s) continue;     // rows before these tokens
                    const int t = lr + 8 * i;
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
        if (any_odd) run(true);                      // a token that a row does not see does not touch it, whatever it holds
        else run(false);
    };
    auto put_outputs = [&](int t0, int n) {
        const float skip = a.skip != nullptr ? a.skip[h] : 0.f;
        float4 raw[NQ];
        if (!SOLVE && a.skip != nullptr)
#pragma unroll
            for (int x = 0; x < NQ; ++x) {
                const int i = x * 128 + gt, t = i / (C / 4), c = (i % (C / 4)) * 4;
                raw[x] = t < n && c0 + c < dv ? load4(vb + (size_t)(t0 + t) * a.v_stride + c) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
        for (int x = 0; x < NQ; ++x) {
            const int i = x * 128 + gt, t = i / (C / 4), c = (i % (C / 4)) * 4;
            if (t < n && c0 + c < dv) {
                float4 s = sum_part(x);
                if (!SOLVE && a.skip != nullptr) {
                    const float4 v = raw[x];
                    s = make_float4(fmaf(skip, v.x, s.x), fmaf(skip, v.y, s.y), fmaf(skip, v.z, s.z), fmaf(skip, v.w, s.w));
                }
                st4(a.o + ((size_t)(t0 + t) * a.H + h) * dv + c0 + c, s);
            }
        }
    };
    // to = e^(B_n) from + sum_s k_s u_s^T: a warp takes 64 rows, all columns and a slice of the tokens; 8 rows x RC columns a thread
    auto update_state = [&](const float* k, const float* u, const float* from, float* to, float total) {
        const int row0 = (gw % RG) * 64 + lr * 8, slice = gw / RG;
        float st[8][RC] = {};
#pragma unroll 4
        for (int s = slice * (T / TS); s < (slice + 1) * (T / TS); ++s) {
            const float4 ka = ld4(k + s * QP + row0), kc = ld4(k + s * QP + row0 + 4);
            const float k8[8] = {ka.x, ka.y, ka.z, ka.w, kc.x, kc.y, kc.z, kc.w};
            float uv[RC];
#pragma unroll
            for (int g = 0; g < RC / 4; ++g) *reinterpret_cast<float4*>(&uv[4 * g]) = ld4(u + s * C + 16 * g + lc * 4);
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int c = 0; c < RC; ++c) st[i][c] = fmaf(k8[i], uv[c], st[i][c]);
        }
        if (slice > 0)
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int g = 0; g < RC / 4; ++g)
                    st4(part2 + ((slice - 1) * DP + row0 + i) * C + 16 * g + lc * 4, make_float4(st[i][4 * g], st[i][4 * g + 1], st[i][4 * g + 2], st[i][4 * g + 3]));
        group_sync(group);
        if (slice == 0)
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int g = 0; g < RC / 4; ++g) {
                    const int at = (row0 + i) * C + 16 * g + lc * 4;
                    const float f = CHANNEL ? tots[row0 + i] : total;
                    float4 s = ld4(from + at);
                    s = make_float4(fmaf(f, s.x, st[i][4 * g]), fmaf(f, s.y, st[i][4 * g + 1]), fmaf(f, s.z, st[i][4 * g + 2]), fmaf(f, s.w, st[i][4 * g + 3]));
#pragma unroll
                    for (int z = 0; z < TS - 1; ++z) {
                        const float4 v = ld4(part2 + z * DP * C + at);
                        s = make_float4(s.x + v.x, s.y + v.y, s.z + v.z, s.w + v.w);
                    }
                    st4(to + at, s);
                }
    };

    const int first_n = min(T, t_last - t_first);
    float* last_state = Ss;
    if (!SOLVE) {
        if (group == 0) {
            load_rows(qs, qb, a.qk_stride, t_first, first_n);
            cp_commit();
        } else {
            load_rows(ks, kb, a.qk_stride, t_first, first_n);
            cp_commit();
            load_v(t_first, first_n);
            load_factors(t_first, first_n);
            put_values(us);
            if (gt < T) rss[gt] = rfac;
        }
        int cur = 0;
        for (int t0 = t_first; t0 < t_last; t0 += T, cur ^= 1) {
            const int n = min(T, t_last - t0), next = t0 + T, next_n = min(T, t_last - next);
            const float total = a.eb[(size_t)(t0 + n - 1) * a.H + h];
            cp_wait<0>();                            // q, k
            const int any_odd = __syncthreads_or(odd);       // state, u and factors of this chunk are there as well
            odd = 0;
            if (group == 0) {
                float acc[RM][RC];
                state_product(qs, Ss + cur * DP * C, acc);
                asm volatile("bar.sync 3, 256;" ::: "memory");       // P is there, the last chunk's sums and q have been read
                if (next < t_last) load_rows(qs, qb, a.qk_stride, next, next_n);
                cp_commit();
                add_tokens(us + cur * T * C, rss + cur * T, any_odd, acc);
                put_part(acc);
            } else {
                load_p(t0, n);
                cp_commit();
                if (next < t_last) {
                    load_rows(ks + (cur ^ 1) * T * QP, kb, a.qk_stride, next, next_n);
                    load_v(next, next_n);
                    load_factors(next, next_n);
                }
                cp_commit();
                if (t0 > t_first) put_outputs(t0 - T, T);    // the last chunk's
                cp_wait<1>();                        // P
                asm volatile("bar.arrive 3, 256;" ::: "memory");
                update_state(ks + cur * T * QP, u2, Ss + cur * DP * C, Ss + (cur ^ 1) * DP * C, total);
                if (next < t_last) {                 // u2 has been read (the barrier inside)
                    put_values(us + (cur ^ 1) * T * C);
                    if (gt < T) rss[(cur ^ 1) * T + gt] = rfac;
                }
            }
        }
        __syncthreads();
        const int last = (t_last - t_first - 1) / T * T;
        if (group == 1) put_outputs(t_first + last, t_last - t_first - last);
        last_state = Ss + cur * DP * C;
    } else {
        if (group == 0) {
            load_rows(ws, wb, (size_t)a.H * d, t_first, first_n);
            cp_commit();
            load_rows(ks, kb, a.qk_stride, t_first, first_n);
            cp_commit();
            load_v(t_first, first_n);
        } else {
            load_rows(qs, qb, a.qk_stride, t_first, first_n);
            cp_commit();
            load_p(t_first, first_n);
            cp_commit();
        }
        load_factors(t_first, first_n);
        for (int t0 = t_first; t0 < t_last; t0 += T) {
            const int n = min(T, t_last - t0), next = t0 + T, next_n = min(T, t_last - next);
            const float total = CHANNEL ? 0.f : a.eb[(size_t)(t0 + n - 1) * a.H + h];
            cp_wait<1>();                            // W or q (k and P may still be on their way)
            __syncthreads();                         // and the state is up to date
            float acc[RM][RC];
            odd = 0;
            if (CHANNEL ? (group == 0 && gt < DP) : (group == 1 && gt < T)) (CHANNEL ? tots : rss)[gt] = rfac;
            state_product(group == 0 ? ws : qs, Ss, acc);
            if (group == 0) {
                put_part(acc);
                group_sync(0);
#pragma unroll
                for (int x = 0; x < NQ; ++x) {
                    const float4 s = sum_part(x);
                    put_u(x, make_float4(vreg[x].x - s.x, vreg[x].y - s.y, vreg[x].z - s.z, vreg[x].w - s.w), us);
                }
            }
            cp_wait<0>();
            const int any_odd = __syncthreads_or(odd);       // u, k and P are there, W and q have been read
            if (next < t_last) {
                if (group == 0) load_rows(ws, wb, (size_t)a.H * d, next, next_n);
                else load_rows(qs, qb, a.qk_stride, next, next_n);
                if (group == 0) load_v(next, next_n);
                load_factors(next, next_n);
            }
            cp_commit();
            if (group == 0) {
                update_state(ks, CHANNEL ? us : u2, Ss, Ss, total);
                if (next < t_last) load_rows(ks, kb, a.qk_stride, next, next_n);       // k has been read (the barrier inside)
                cp_commit();
            } else {
                add_tokens(us, rss, any_odd, acc);
                put_part(acc);
                group_sync(1);
                if (next < t_last) load_p(next, next_n);
                cp_commit();
                put_outputs(t0, n);
            }
        }
    }
    cp_wait<0>();
    __syncthreads();
    for (int i = tid; i < DP * C; i += kThreads) {
        const int row = a.s_row == 1 ? i % DP : i / C, c = a.s_row == 1 ? i / DP : i % C;
        if (row < d && c0 + c < dv) S0[(size_t)row * a.s_row + (size_t)(c0 + c) * a.s_col] = last_state[row * C + c];
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

