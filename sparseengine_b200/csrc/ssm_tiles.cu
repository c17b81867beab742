// The state-space recurrence over prompt portions by chunks of 128 tokens side by side (chunk_tiles.cuh), for states of 128 rows and heads of 64 columns
// beside bfloat16 activations:
//
//     y_t = e^(B_t) C_t . S_0 + sum_{s <= t} e^(B_t - B_s) (C_t . B_s) u_s + D x_t,     S = e^(B_n) S_0 + sum_s e^(B_n - B_s) B_s u_s^T,     u = step x
//
// (B_t the sum of the log decays up to and with token t.)  A group's heads share C and B: a block takes up to eight of them and a chunk, cuts C and B into terms once
// and forms C B^T once.  Three kernels: `states` leaves what each chunk adds, `scan` turns that into the states at the chunks' starts, `outputs` does
// the rest.
#include "chunk_tiles.cuh"

namespace se {
namespace tiles {

constexpr int kV = 64, kHeads = 8;                   // columns of a head's state; heads that a block takes at most
constexpr int kSTerm = kV * 256, kSHalf = kV * 128;  // bytes of a term of the state (rows along its columns), of half of one
constexpr int kUTerm = kT * 128;                     // of the values: rows are tokens

struct StateSpace {
    const float* xbc;              // [tokens][H * 64 + 2 G * 128]: values, B, C
    const __nv_bfloat16* proj;                // steps' columns from dt_off on
    int pitch, dt_off;
    const float* dt_bias;
    const float* a_log;
    const float* d_skip;
    float* states;                 // [places][H][64][128]: what a chunk adds, then the state at its start
    float* totals;                 // [places][H]: e^(B_n)
    float* state;
    long long state_stride;
    const int* cu_q;
    const int* seq_rows;
    float* y;
    int entries, H, G, blocks, per;        // blocks per group of heads, heads per block
    int* error;
};

struct Tables { float hi[kHeads][kT], lo[kHeads][kT], step[kHeads][kT]; };

// B_t of a block's heads as two 32-bit parts, and the steps (0 where there is no token), a warp per head and four tokens a lane
__device__ __forceinline__ void fill_tables(const StateSpace& p, Tables& s, int h0, int heads, int first, int n) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp >= heads) return;
    const int h = h0 + warp;
    const float rate = expf(p.a_log[h]), bias = p.dt_bias[h];
    float step[4];
    double sum[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int t = 4 * lane + j;
        step[j] = t < n ? walk::softplus32(to_float(p.proj[(size_t)(first + t) * p.pitch + p.dt_off + h]) + bias) : 0.f;
        sum[j] = (t < n ? walk::log_decay(rate, step[j]) : 0.0) + (j ? sum[j - 1] : 0.0);
    }
    double before;
    walk::sum_before(sum[3], lane, before);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int t = 4 * lane + j;
        const double b = before + sum[j];
        const float hi = (float)b;
        s.hi[warp][t] = hi;
        s.lo[warp][t] = (float)(b - (double)hi);
        s.step[warp][t] = step[j];
    }
}
// e^(B_t - B_s)
__device__ __forceinline__ float decay_between(const Tables& s, int h, int t, int t0) { return expf((s.hi[h][t] - s.hi[h][t0]) + (s.lo[h][t] - s.lo[h][t0])); }

// B's or C's rows of a chunk in three terms: a row per warp at a time
__device__ __forceinline__ void put_rows(uint32_t at, const float* src, size_t stride, int n) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = 16 * i + warp < n ? ld4(src + (size_t)(16 * i + warp) * stride + 4 * lane) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 8; ++i) put4(at + (lane >> 4) * kHalf, kTerm, 16 * i + warp, lane & 15, v[i]);
}
// A head's values: two rows a warp at a time, four columns a lane
__device__ __forceinline__ void fetch_rows(float4 (&v)[4], const float* src, size_t stride, int n) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int t = 32 * i + 2 * warp + (lane >> 4);
        v[i] = t < n ? ld4(src + (size_t)t * stride + 4 * (lane & 15)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
}
template <typename Factor>
__device__ __forceinline__ void put_values(uint32_t at, uint32_t term, const float4 (&v)[4], Factor factor) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int t = 32 * i + 2 * warp + (lane >> 4);
        const float f = factor(t);
        put4(at, term, t, lane & 15, make_float4(v[i].x * f, v[i].y * f, v[i].z * f, v[i].w * f));
    }
}

// What each chunk adds to its heads' states: rows of the state = the M side, B's rows as they lie, two heads' columns the N side (one at a time, N = 64, shared memory
// holds the products up: 32 us, 27 so).  A pair's sums are stored while the next pair's products run.
__global__ void __launch_bounds__(kThreads, 1)
ssm_states_kernel(const StateSpace p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023) & ~1023u, keys = base, values = base + 3 * kTerm;       // values: terms of two heads' columns side by side
    Tables& tab = *reinterpret_cast<Tables*>(smem_raw + (base - smem_u32(smem_raw)) + 3 * kTerm + 6 * kUTerm);
    __shared__ Shared sh;
    int first, n;
    chunk_of<kT>(blockIdx.x, p.cu_q, p.entries, first, n);
    if (n <= 0) return;
    const int rep = p.H / p.G, g = blockIdx.y / p.blocks, h0 = g * rep + (blockIdx.y - g * p.blocks) * p.per, heads = min(p.per, (g + 1) * rep - h0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row = (warp & 3) * 32 + lane, col = (warp >> 2) * 16;
    const size_t width = (size_t)p.H * kV + 2 * (size_t)p.G * kD;
    const float* x = p.xbc + (size_t)first * width;
    const float* b = x + (size_t)p.H * kV + (size_t)g * kD;
    const uint32_t tmem = (uint32_t)fa::uniform((int)begin(sh));
    const bool issuer = fa::uniform(warp) == 0;
    const uint32_t mine = tmem + ((uint32_t)((warp & 3) * 32) << 16) + col;
    float4 v[2][4];
    auto fetch = [&](int i) {
        fetch_rows(v[0], x + (size_t)(h0 + i) * kV, width, n);
        if (i + 1 < heads) fetch_rows(v[1], x + (size_t)(h0 + i + 1) * kV, width, n);
    };
    fetch(0);
    fill_tables(p, tab, h0, heads, first, n);
    put_rows(keys, b, width, n);
    __syncthreads();
    const int pairs = (heads + 1) / 2;
    bool ok = true;
    for (int i = 0; i <= pairs && ok; ++i) {         // pair i's products are issued, pair i - 1's sums stored
        if (i > 0 && !(ok = products_done(sh, i - 1, p.error))) break;
        if (i < pairs) {
#pragma unroll
            for (int j = 0; j < 2; ++j)
                if (2 * i + j < heads)
                    put_values(values + j * kUTerm, 2 * kUTerm, v[j], [&](int t) { return t < n ? decay_between(tab, 2 * i + j, n - 1, t) * tab.step[2 * i + j][t] : 0.f; });
            fence_smem();
            fence_before();
            __syncthreads();
            if (issuer) {
                fence_after();
                if (fa::elect_one()) {
                    product<true, true, 3>(tmem + (i & 1) * 4 * kV, tmem + (i & 1) * 4 * kV + 2 * kV, keys, kHalf, kTerm, values, kUTerm, 2 * kUTerm, instr(2 * i + 1 < heads ? 2 * kV : kV, true, true));
                    fa::umma_commit(smem_u32(&sh.done));
                }
                __syncwarp();
            }
            if (i + 1 < pairs) fetch(2 * i + 2);
        }
        if (i == 0) continue;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int own = 2 * (i - 1) + j, h = h0 + own;
            if (own >= heads) break;
            float sum[16], z = 0.f;
            ld_sum16(mine + ((i - 1) & 1) * 4 * kV + j * kV, mine + ((i - 1) & 1) * 4 * kV + 2 * kV + j * kV, sum);
#pragma unroll
            for (int c = 0; c < 16; ++c) z = fmaf(sum[c], 0.f, z);
            if (__any_sync(0xffffffffu, z != 0.f)) {
#pragma unroll
                for (int c = 0; c < 16; ++c) sum[c] = 0.f;
#pragma unroll 1
                for (int t = 0; t < n; ++t) {
                    const float k = b[(size_t)t * width + row], f = decay_between(tab, own, n - 1, t) * tab.step[own][t];
#pragma unroll
                    for (int c = 0; c < 16; ++c) sum[c] = fmaf(k, x[(size_t)t * width + (size_t)h * kV + col + c] * f, sum[c]);
                }
            }
            float* to = p.states + ((size_t)blockIdx.x * p.H + h) * (kV * kD) + row;
#pragma unroll
            for (int c = 0; c < 16; ++c) to[(size_t)(col + c) * kD] = sum[c];
            if (threadIdx.x == 0) p.totals[(size_t)blockIdx.x * p.H + h] = expf(tab.hi[own][n - 1] + tab.lo[own][n - 1]);
        }
    }
    end(sh);
}

// What chunks add -> the states at their starts; the last one goes back to the entry's row.  Four elements a thread; four chunks asked for together.
__global__ void __launch_bounds__(256)
ssm_scan_kernel(const StateSpace p) {
    grid_dependency_trigger();                       // the outputs' kernel may start: it has C B^T to form first
    const int e = blockIdx.z, h = blockIdx.y, i = (blockIdx.x * 256 + threadIdx.x) * 4;
    const int t0 = p.cu_q[e], chunks = ceil_div(p.cu_q[e + 1] - t0, kT);
    if (chunks <= 0) return;
    float* own = p.state + (size_t)p.seq_rows[e] * p.state_stride + (size_t)h * kV * kD + i;
    const size_t place = (size_t)(t0 / kT + e);
    float4 S = ld4(own);
    for (int c0 = 0; c0 < chunks; c0 += 4) {
        float4 add[4];
        float f[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const size_t at = (place + min(c0 + c, chunks - 1)) * p.H + h;
            add[c] = ld4(p.states + at * (kV * kD) + i);
            f[c] = p.totals[at];
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (c0 + c >= chunks) break;
            walk::st4(p.states + ((place + c0 + c) * p.H + h) * (kV * kD) + i, S);
            S = make_float4(fmaf(f[c], S.x, add[c].x), fmaf(f[c], S.y, add[c].y), fmaf(f[c], S.z, add[c].z), fmaf(f[c], S.w, add[c].w));
        }
    }
    walk::st4(own, S);
}

// Bound by a head's steps one after another (some 14,000 cycles, of which its products take 3,800 and shared memory gives them 128 bytes a cycle).  Each warp's weights are eight
// columns of every 32, so that all share the exponents of the diagonal (32 columns a warp, and one warp of four with all of them: 87 us, 77 so); two warps issue, because
// a warp is held by the products it issues (one for both 116, two 87); outputs leave through shared memory (a row a thread 77, 63 so; 67 with
// products in two parts).
// Columns of tensor memory: C B^T 0-127, P's terms 128-319, what the state gives in two parts 320-383 and 384-447, P u 384-447 and 448-511.  While a head's P u
// is summed the next head's state is cut and the first part of its product with C queued behind, the second part once P u has been read.
__global__ void __launch_bounds__(kThreads, 1)
ssm_outputs_kernel(const StateSpace p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023) & ~1023u, queries = base, keys = base + 3 * kTerm, state = keys, values = keys + 3 * kSTerm;
    Tables& tab = *reinterpret_cast<Tables*>(smem_raw + (base - smem_u32(smem_raw)) + 6 * kTerm);
    __shared__ Shared sh;
    __shared__ __align__(8) uint64_t state_done;
    int first, n;
    chunk_of<kT>(blockIdx.x, p.cu_q, p.entries, first, n);
    if (n <= 0) {
        grid_dependency_wait();                      // nothing of this kernel ends before the one ahead
        return;
    }
    const int rep = p.H / p.G, g = blockIdx.y / p.blocks, h0 = g * rep + (blockIdx.y - g * p.blocks) * p.per, heads = min(p.per, (g + 1) * rep - h0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, part = warp >> 2, row = (warp & 3) * 32 + lane, vcol = part * 16;
    const size_t width = (size_t)p.H * kV + 2 * (size_t)p.G * kD;
    const float* x = p.xbc + (size_t)first * width;
    const float* b = x + (size_t)p.H * kV + (size_t)g * kD;
    const float* c = b + (size_t)p.G * kD;
    const float* S = p.states + (size_t)blockIdx.x * p.H * (kV * kD);
    if (threadIdx.x == 0) fa::mbar_init(smem_u32(&state_done), 1);
    const uint32_t tmem = (uint32_t)fa::uniform((int)begin(sh));
    const int role = fa::uniform(warp);              // 0 issues P u, 1 what the state gives
    const uint32_t mine = tmem + ((uint32_t)((warp & 3) * 32) << 16), weights = 128, old = 320, shared = 384, sums = 448;
    uint32_t round = 0;
    bool ok = true;
    float4 uv[4];
    auto put_state = [&](int i) {                    // a column of it per warp at a time
        float4 sv[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) sv[j] = ld4(S + ((size_t)(h0 + i) * kV + 16 * j + warp) * kD + 4 * lane);
#pragma unroll
        for (int j = 0; j < 4; ++j) put4(state + (lane >> 4) * kSHalf, kSTerm, 16 * j + warp, lane & 15, sv[j]);
    };
    auto issue_state = [&](int half) {
        if (role == 1) {
            fence_after();
            if (fa::elect_one()) {
                if (half == 0)
                    product_first<false, false, 3>(tmem + old, queries, kHalf, kTerm, state, kSHalf, kSTerm, instr(kV, false, false));
                else {
                    product_second<false, false>(tmem + shared, queries, kHalf, state, kSHalf, instr(kV, false, false));
                    fa::umma_commit(smem_u32(&state_done));
                }
            }
            __syncwarp();
        }
    };
    fill_tables(p, tab, h0, heads, first, n);
    put_rows(queries, c, width, n);
    put_rows(keys, b, width, n);
    fence_smem();
    __syncthreads();
    if (role == 0) {
        if (fa::elect_one()) {
            product<false, false, 3>(tmem, tmem + weights, queries, kHalf, kTerm, keys, kHalf, kTerm, instr(kT, false, false));
            fa::umma_commit(smem_u32(&sh.done));
        }
        __syncwarp();
    }
    fetch_rows(uv, x + (size_t)h0 * kV, width, n);
    ok = products_done(sh, round++, p.error);        // B's terms give way to the first head's state and values
    grid_dependency_wait();                          // the states at the chunks' starts
    if (ok) {
        if (part <= (warp & 3)) {                    // both parts of C B^T together, where tokens see others (a warp's 32 columns)
#pragma unroll
            for (int x = 0; x < 32; x += 16) {
                float v[16];
                ld_sum16(mine + 32 * part + x, mine + weights + 32 * part + x, v);
                st8(mine + 32 * part + x, reinterpret_cast<uint32_t*>(v));
                st8(mine + 32 * part + x + 8, reinterpret_cast<uint32_t*>(v + 8));
            }
            wait_st();
        }
        put_state(0);
        fence_smem();
        fence_before();
        __syncthreads();
        fence_after();
        issue_state(0);
        issue_state(1);
    }
    for (int i = 0; i < heads && ok; ++i) {
        const int h = h0 + i;
        // P of this head: the block on the diagonal by its own exponents, those before it by e^(B_t - B_r) e^(B_r - B_s), r the block's first token
        put_values(values, kUTerm, uv, [&](int t) { return tab.step[i][t]; });
        const int block = warp & 3, r = 32 * block;  // rows r .. r + 31; a warp's columns are eight of each block of 32
        const float f = decay_between(tab, i, row, r);
        const float before = lane < 8 * block ? decay_between(tab, i, r, 32 * (lane >> 3) + 8 * part + (lane & 7)) : 0.f;
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            uint32_t w[3][4] = {};
            if (x <= block) {
                uint32_t v[8];
                ld8(mine + 32 * x + 8 * part, v);
                wait_ld();
                float e[8];
                if (x < block) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) e[j] = __uint_as_float(v[j]) * (f * __shfl_sync(0xffffffffu, before, 8 * x + j));
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int s = 8 * part + j;
                        const float d = decay_between(tab, i, row, r + s);
                        e[j] = s <= lane ? __uint_as_float(v[j]) * d : 0.f;
                    }
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    uint32_t t3[3];
                    cut(e[2 * j], e[2 * j + 1], t3);
#pragma unroll
                    for (int y = 0; y < 3; ++y) w[y][j] = t3[y];
                }
            }
#pragma unroll
            for (int y = 0; y < 3; ++y) st4(mine + weights + y * 64 + 16 * x + 4 * part, w[y]);
        }
        // the state's product is there: its terms may give way, its columns to P u
        ok = warp_wait(sh, state_done, i);
        fence_after();
        float u[16];
        ld_sum16(mine + old + vcol, mine + shared + vcol, u);
        wait_st();
        fence_smem();
        fence_before();
        ok = __syncthreads_and(ok);
        if (!ok) {
            if (threadIdx.x == 0) atomicCAS(p.error, 0, kErrorCode);
            break;
        }
        fence_after();
        if (role == 0) {
            if (fa::elect_one()) {
                product_ts<true, 3>(tmem + shared, tmem + sums, tmem + weights, values, 0, kUTerm, instr(kV, false, true));
                fa::umma_commit(smem_u32(&sh.done));
            }
            __syncwarp();
        }
        if (i + 1 < heads) {
            put_state(i + 1);
            fence_smem();
            __syncthreads();
            issue_state(0);
            fetch_rows(uv, x + (size_t)(h + 1) * kV, width, n);
        }
        const float skip = p.d_skip[h];
        float4 own[4];                               // the values as they are
        fetch_rows(own, x + (size_t)h * kV, width, n);
        if (!(ok = products_done(sh, round++, p.error))) break;
        float o[16];
        ld_sum16(mine + shared + vcol, mine + sums + vcol, o);
        fence_before();
        const float lead = expf(tab.hi[i][row] + tab.lo[i][row]);
        float z = 0.f, y[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            y[j] = fmaf(lead, u[j], o[j]);
            z = fmaf(y[j], 0.f, z);
        }
        float* to = p.y + ((size_t)first * p.H + h) * kV;
        const bool finite = !__syncthreads_or(z != 0.f && row < n);
        if (i + 1 < heads) issue_state(1);
        if (finite) {
            // through shared memory (the values have been read), so that neighbouring threads store neighbours
            uint8_t* rows = smem_raw + (values - smem_u32(smem_raw));
#pragma unroll
            for (int j = 0; j < 4; ++j)
                *reinterpret_cast<float4*>(rows + row * 256 + (((4 * part + j) ^ (row & 7)) << 4)) = make_float4(y[4 * j], y[4 * j + 1], y[4 * j + 2], y[4 * j + 3]);
            __syncthreads();
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int r = 32 * j + 2 * warp + (lane >> 4), q = lane & 15;
                const float4 v = *reinterpret_cast<const float4*>(rows + r * 256 + ((q ^ (r & 7)) << 4));
                if (r < n)
                    walk::st4(to + (size_t)r * p.H * kV + 4 * q, make_float4(fmaf(skip, own[j].x, v.x), fmaf(skip, own[j].y, v.y), fmaf(skip, own[j].z, v.z), fmaf(skip, own[j].w, v.w)));
            }
            __syncthreads();                         // before the next head's values
        } else {                                     // token by token: a column of the state and 16 rows a thread
            const int v0 = threadIdx.x >> 3, d0 = (threadIdx.x & 7) * 16;
            float s[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) s[j] = S[((size_t)h * kV + v0) * kD + d0 + j];
#pragma unroll 1
            for (int t = 0; t < n; ++t) {
                const float xv = x[(size_t)t * width + (size_t)h * kV + v0], uv1 = xv * tab.step[i][t];
                const float keep = t ? decay_between(tab, i, t, t - 1) : expf(tab.hi[i][0] + tab.lo[i][0]);
                float sum = 0.f;
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    s[j] = fmaf(keep, s[j], b[(size_t)t * width + d0 + j] * uv1);
                    sum = fmaf(c[(size_t)t * width + d0 + j], s[j], sum);
                }
#pragma unroll
                for (int m = 1; m < 8; m <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, m);
                if (d0 == 0) to[(size_t)t * p.H * kV + v0] = fmaf(skip, xv, sum);
            }
        }
    }
    end(sh);
}

static int launch_ssm(const StateSpace& p, int places, cudaStream_t stream) {
    const int states_smem = 3 * kTerm + 6 * kUTerm + (int)sizeof(Tables) + 1024, outputs_smem = 6 * kTerm + (int)sizeof(Tables) + 1024;
    cudaError_t e = cudaFuncSetAttribute(ssm_states_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, states_smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(ssm_outputs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, outputs_smem);
    if (e != cudaSuccess) return (int)e;
    const dim3 grid(places, p.G * p.blocks);
    ssm_states_kernel<<<grid, kThreads, states_smem, stream>>>(p);
    ssm_scan_kernel<<<dim3(kV * kD / 1024, p.H, p.entries), 256, 0, stream>>>(p);
    if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
    return (int)SE_LAUNCH_DEPENDENT("ssm", ssm_outputs_kernel, grid, dim3(kThreads), (size_t)outputs_smem, stream, p);
}

}  // namespace tiles
}  // namespace se

using namespace se::tiles;

extern "C" int se_ssm_tiles_supported(int state_size, int head_dim) { return state_size == kD && head_dim == kV; }

// Arguments as se_ssm_walk's, proj bfloat16.  work: float [(tokens / 128 + entries) * H * (64 * 128 + 1)].  per: heads of a group that a block takes at most (C and B are
// cut and multiplied once per block).
extern "C" int se_ssm_tiles(const float* xbc, const void* proj, int pitch, int dt_off, const float* dt_bias, const float* a_log, const float* d_skip,
                            float* state, long long state_stride, const int* cu_q, const int* seq_rows, float* y, float* work, int* error, int tokens,
                            int entries, int H, int P, int N, int G, int per, cudaStream_t stream) {
    if (entries <= 0 || tokens <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G || per < 1 || per > kHeads) return SE_ERR_ARGUMENT;
    const long long places = tokens / kT + entries;
    const int blocks = (H / G + per - 1) / per;
    auto aligned = [](const void* a) { return (reinterpret_cast<uintptr_t>(a) & 15) == 0; };
    if (!se_ssm_tiles_supported(N, P) || H > 65535 || (long long)G * blocks > 65535 || entries > 65535 || places > 0x7fffffffLL || state_stride % 4 ||
        !aligned(xbc) || !aligned(state) || !aligned(y) || !aligned(work))
        return SE_ERR_UNSUPPORTED;
    StateSpace p;
    p.xbc = xbc; p.proj = (const __nv_bfloat16*)proj; p.pitch = pitch; p.dt_off = dt_off; p.dt_bias = dt_bias; p.a_log = a_log; p.d_skip = d_skip;
    p.states = work; p.totals = work + (size_t)places * H * (kV * kD); p.state = state; p.state_stride = state_stride; p.cu_q = cu_q; p.seq_rows = seq_rows;
    p.y = y; p.entries = entries; p.H = H; p.G = G; p.blocks = blocks; p.per = per; p.error = error;
    return launch_ssm(p, (int)places, stream);
}
