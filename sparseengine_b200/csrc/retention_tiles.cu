// Retention over prompt portions by chunks of 128 tokens side by side (chunk_tiles.cuh), bfloat16 activations, heads of 128 x 128:
//
//     o_t = g^(t+1) q_t . S_0 + sum_{s <= t} g^(t-s) (q_t . k_s) v_s,      S = g^n S_0 + sum_s g^(n-1-s) k_s v_s^T
//
// Three kernels after one that works out angles and powers once for all heads: `states` (a block per head and segment of an entry's chunks) leaves the
// state at each chunk's start, `join` (where an entry has several segments) the states at the segments' starts, `outputs` (a block per chunk and head)
// the rest: q and k turned on their way from the projection, both products with q, the decays, P v, and where the mixer norms each head the norm and the gate.
//
// Measured, 8,192 tokens of 32 heads (the walk, its preparation and the norm: 676 us): 302, of them angles 4, states 74, join 6, outputs 214, starts and ends 4; 2,048 tokens of 16
// heads 147 and 59; four entries of 100 tokens, 32 heads, 54 and 39.  Errors: chunk_tiles.cuh; 16-bit inputs and outputs leave 4e-3.
#include "chunk_tiles.cuh"

namespace se {
namespace tiles {

struct Retention {
    const __nv_bfloat16* proj;
    int pitch, q_off, k_off, v_off, g_off;
    const float2* turn;            // [tokens][64] cosine and sine, or null: q and k as they are
    const float* powers;           // [H][powers_pitch]: g^0 .. g^128, then g^(128 j) for j = 0 ..
    int powers_pitch;
    float* states;                 // [places][H][128 columns][128 rows]: at a chunk's start, from its segment's start on
    float* starts;                 // [entries * segments][H][128][128]: what a segment leaves by itself, then the state at its start
    int segments, seg_chunks;      // per entry at most; chunks of a segment (the last one takes what is left: a captured step may meet longer entries)
    float* state;
    long long state_stride;
    const int* cu_q;
    const int* seq_rows;
    int entries, H, places;
    float k_scale, eps;
    __nv_bfloat16* out;            // [tokens][H * 128] after norm and gate, or null:
    float* o;                      // [tokens][H * 128]
    int* error;
};

__global__ void __launch_bounds__(256)
retention_tables_kernel(float2* __restrict__ turn, const int* __restrict__ positions, const float* __restrict__ inv_freq, int tokens, int turn_blocks,
                        float* __restrict__ powers, int pitch, const float* __restrict__ decay) {
    if ((int)blockIdx.x < turn_blocks) {
        const int x = blockIdx.x * 256 + threadIdx.x;
        if (x >= tokens * 64) return;
        float s, c;
        sincosf((float)positions[x >> 6] * inv_freq[x & 63], &s, &c);
        turn[x] = make_float2(c, s);
        return;
    }
    const int h = blockIdx.x - turn_blocks;
    const double g = (double)decay[h];
    for (int i = threadIdx.x; i < pitch; i += 256) powers[(size_t)h * pitch + i] = (float)pow(g, (double)(i <= kT ? i : (i - kT - 1) * kT));
}

// g^(128 j) of a head
__device__ __forceinline__ float chunks_power(const Retention& p, int h, int j) {
    const float* power = p.powers + (size_t)h * p.powers_pitch;
    return j <= p.seg_chunks ? power[kT + 1 + j] : (float)pow((double)power[1], (double)j * kT);
}

// a pair of a row turned by its angle
__device__ __forceinline__ void rotate(float2 cs, float& a, float& b) {
    const float a0 = a;
    a = a0 * cs.x - b * cs.y;
    b = b * cs.x + a0 * cs.y;
}
// element d of a token's q or k row (columns from `off` on), turned
__device__ __forceinline__ float column_of(const Retention& p, int off, size_t token, int h, int d) {
    const __nv_bfloat16* row = p.proj + token * p.pitch + off + (size_t)h * kD;
    float lo = __bfloat162float(row[d & 63]), hi = __bfloat162float(row[64 + (d & 63)]);
    if (p.turn != nullptr) rotate(p.turn[token * 64 + (d & 63)], lo, hi);
    return d < 64 ? lo : hi;
}
__device__ __forceinline__ float key_of(const Retention& p, size_t token, int h, int d) { return column_of(p, p.k_off, token, h, d) * p.k_scale; }
// four pairs of columns of a row turned (two pairs a float4) and cut: to the row's place in the halves of an operand
__device__ __forceinline__ void put_pairs(uint32_t at, int row, int quad, uint2 lo, uint2 hi, float4 c0, float4 c1, float f) {
    float x[4] = {__uint_as_float(lo.x << 16), __uint_as_float(lo.x & 0xffff0000u), __uint_as_float(lo.y << 16), __uint_as_float(lo.y & 0xffff0000u)};
    float y[4] = {__uint_as_float(hi.x << 16), __uint_as_float(hi.x & 0xffff0000u), __uint_as_float(hi.y << 16), __uint_as_float(hi.y & 0xffff0000u)};
    rotate(make_float2(c0.x, c0.y), x[0], y[0]);
    rotate(make_float2(c0.z, c0.w), x[1], y[1]);
    rotate(make_float2(c1.x, c1.y), x[2], y[2]);
    rotate(make_float2(c1.z, c1.w), x[3], y[3]);
    put4(at, kTerm, row, quad, make_float4(x[0] * f, x[1] * f, x[2] * f, x[3] * f));
    put4(at + kHalf, kTerm, row, quad, make_float4(y[0] * f, y[1] * f, y[2] * f, y[3] * f));
}
// a head's rows as they are, columns from `off` on: [128 tokens][64 columns], twice
__device__ __forceinline__ void fetch_rows(const Retention& p, uint32_t at, int off, int first, int n, int h) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int x = i * kThreads + threadIdx.x, t = x >> 4, c = x & 15;
        const bool in = t < n;
        cp16(at + (c >> 3) * kHalf + fa::sw128(t, c & 7), p.proj + (size_t)(first + (in ? t : 0)) * p.pitch + off + (size_t)h * kD + c * 8, in);
    }
}

// a chunk's angles: [128][64] cosines and sines, 16-byte pieces of a row in the order of its last three bits
__device__ __forceinline__ void fetch_angles(const Retention& p, uint32_t at, int first, int n) {
    if (p.turn == nullptr) return;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int x = i * kThreads + threadIdx.x, r = x >> 5, c = x & 31;
        cp16(at + r * 512 + ((c ^ (r & 7)) << 4), p.turn + (size_t)(first + min(r, n - 1)) * 64 + 2 * c, true);
    }
}
// of pairs 2 c and 2 c + 1 of row r
__device__ __forceinline__ float4 angle_at(const Retention& p, const uint8_t* angles, int r, int c) {
    return p.turn != nullptr ? *reinterpret_cast<const float4*>(angles + r * 512 + ((c ^ (r & 7)) << 4)) : make_float4(1.f, 0.f, 1.f, 0.f);
}

// Bound by a chunk's steps one after another (cuts of k 3,000 cycles, products 2,200 beside copies and stores of 3,000, the state's update 600; 4.6 us a chunk, the tensor pipe 18 % busy): 128 rows of the
// state by 128 columns in registers, a row and 32 columns a thread.  The next chunk's k and angles are fetched while this one's products run.  As many segments as fill the device, because the alternative, what every chunk adds and a
// scan over it, reads and writes the states (134 MB for 8,192 tokens of 32 heads) once more.
__global__ void __launch_bounds__(kThreads, 1)
retention_states_kernel(const Retention p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023) & ~1023u, keys = base, values = base + 3 * kTerm, raw = base + 4 * kTerm, angles = base + 5 * kTerm;
    const uint8_t* sm = smem_raw + (base - smem_u32(smem_raw));
    __shared__ Shared sh;
    __shared__ float power[kT + 1];
    const int e = blockIdx.x / p.segments, seg = blockIdx.x - e * p.segments, h = blockIdx.y;
    const int t_first = p.cu_q[e], t_last = p.cu_q[e + 1];
    const int chunks = ceil_div(t_last - t_first, kT), c0 = seg * p.seg_chunks, c1 = seg == p.segments - 1 ? chunks : min(c0 + p.seg_chunks, chunks);
    if (c0 >= c1) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row = (warp & 3) * 32 + lane, col = (warp >> 2) * 32;
    for (int i = threadIdx.x; i <= kT; i += kThreads) power[i] = p.powers[(size_t)h * p.powers_pitch + i];
    fetch_rows(p, raw, p.k_off, t_first + c0 * kT, min(kT, t_last - t_first - c0 * kT), h);
    fetch_angles(p, angles, t_first + c0 * kT, min(kT, t_last - t_first - c0 * kT));
    walk::cp_commit();
    const uint32_t tmem = (uint32_t)fa::uniform((int)begin(sh));
    const bool issuer = fa::uniform(warp) == 0;
    const uint32_t mine = tmem + ((uint32_t)((warp & 3) * 32) << 16) + col;
    float S[32];
    float* own = p.state + (size_t)p.seq_rows[e] * p.state_stride + ((size_t)h * kD + row) * kD + col;
#pragma unroll
    for (int c = 0; c < 32; c += 4) {
        const float4 v = seg == 0 ? ld4(own + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        S[c] = v.x; S[c + 1] = v.y; S[c + 2] = v.z; S[c + 3] = v.w;
    }
    auto store = [&](float* to) {                    // [column][row]
#pragma unroll
        for (int c = 0; c < 32; ++c) to[(size_t)(col + c) * kD + row] = S[c];
    };
    uint32_t round = 0;
    for (int c = c0; c < c1; ++c, ++round) {
        const int first = t_first + c * kT, n = min(kT, t_last - first);
        walk::cp_wait<0>();
        __syncthreads();                             // k and angles are there
        fetch_rows(p, values, p.v_off, first, n, h);
        walk::cp_commit();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int t = 32 * i + 2 * warp + (lane >> 4), quad = lane & 15;
            const uint8_t* from = sm + 4 * kTerm + fa::sw128(t, quad >> 1) + (quad & 1) * 8;
            put_pairs(keys, t, quad, *reinterpret_cast<const uint2*>(from), *reinterpret_cast<const uint2*>(from + kHalf),
                      angle_at(p, sm + 5 * kTerm, t, 2 * quad), angle_at(p, sm + 5 * kTerm, t, 2 * quad + 1), t < n ? power[n - 1 - t] * p.k_scale : 0.f);
        }
        walk::cp_wait<0>();
        fence_smem();
        fence_before();                              // the last chunk's sums have been read
        __syncthreads();
        if (issuer) {
            fence_after();
            if (fa::elect_one()) {
                product<true, true, 1>(tmem, tmem + kD, keys, kHalf, kTerm, values, kHalf, kTerm, instr(kD, true, true));
                fa::umma_commit(smem_u32(&sh.done));
            }
            __syncwarp();
        }
        if (c + 1 < c1) {
            fetch_rows(p, raw, p.k_off, first + kT, min(kT, t_last - first - kT), h);
            fetch_angles(p, angles, first + kT, min(kT, t_last - first - kT));
            walk::cp_commit();
        }
        store(p.states + ((size_t)(t_first / kT + e + c) * p.H + h) * (kD * kD));
        if (!products_done(sh, round, p.error)) break;
        float v[32], z = 0.f;
        ld_sum16(mine, mine + kD, v);
        ld_sum16(mine + 16, mine + kD + 16, v + 16);
#pragma unroll
        for (int x = 0; x < 32; ++x) z = fmaf(v[x], 0.f, z);
        const float total = power[n];
        if (!__syncthreads_or(z != 0.f)) {
#pragma unroll
            for (int x = 0; x < 32; ++x) S[x] = fmaf(total, S[x], v[x]);
        } else {
#pragma unroll 1
            for (int t = 0; t < n; ++t) {
                const float k = key_of(p, (size_t)first + t, h, row);
                const __nv_bfloat16* vr = p.proj + (size_t)(first + t) * p.pitch + p.v_off + (size_t)h * kD + col;
#pragma unroll
                for (int x = 0; x < 32; ++x) S[x] = fmaf(power[1], S[x], k * __bfloat162float(vr[x]));
            }
        }
    }
    walk::cp_wait<0>();
    if (p.segments > 1) store(p.starts + ((size_t)blockIdx.x * p.H + h) * (kD * kD));
    else
#pragma unroll
        for (int c = 0; c < 32; c += 4) *reinterpret_cast<float4*>(own + c) = make_float4(S[c], S[c + 1], S[c + 2], S[c + 3]);
    end(sh);
}

// A segment's end by itself -> the state at its start; the last one goes back to the entry's row.  32 x 32 elements a block.
__global__ void __launch_bounds__(256)
retention_join_kernel(const Retention p) {
    __shared__ float turned[32][33];
    grid_dependency_trigger();                       // the outputs' kernel may fetch its first chunk
    const int e = blockIdx.z, h = blockIdx.y, c0 = (blockIdx.x >> 2) * 32, r0 = (blockIdx.x & 3) * 32, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int len = p.cu_q[e + 1] - p.cu_q[e], chunks = ceil_div(len, kT);
    if (len <= 0) return;
    const float* power = p.powers + (size_t)h * p.powers_pitch;
    float S[4] = {};
    const int most = min(p.segments, ceil_div(chunks, p.seg_chunks));
    for (int seg0 = 0; seg0 < most; seg0 += 4) {     // four segments asked for together
        float left[4][4];
        float* at = p.starts + ((size_t)(e * p.segments + seg0) * p.H + h) * (kD * kD) + r0 + tx;
        const size_t step = (size_t)p.H * kD * kD;
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
            for (int i = 0; i < 4; ++i) left[x][i] = seg0 + x < most ? at[x * step + (size_t)(c0 + ty + 8 * i) * kD] : 0.f;
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            if (seg0 + x >= most) break;
            const int rest = len - (seg0 + x) * p.seg_chunks * kT, tokens = seg0 + x == p.segments - 1 ? rest : min(rest, p.seg_chunks * kT);
            const float f = chunks_power(p, h, tokens / kT) * power[tokens % kT];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (seg0 + x) at[x * step + (size_t)(c0 + ty + 8 * i) * kD] = S[i];
                S[i] = seg0 + x ? fmaf(f, S[i], left[x][i]) : left[x][i];
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) turned[ty + 8 * i][tx] = S[i];
    __syncthreads();
    float* own = p.state + (size_t)p.seq_rows[e] * p.state_stride + (size_t)h * kD * kD;
#pragma unroll
    for (int i = 0; i < 4; ++i) own[(size_t)(r0 + ty + 8 * i) * kD + c0 + tx] = turned[tx][ty + 8 * i];
}

// A block takes chunks in turn.  The next chunk's q, k and angles are fetched into room that this one's products have left (the state's terms, the last of
// k's) while its weights are made and P v runs; the state comes into registers meanwhile.  Bound by the steps of a chunk, 15 us, one after another: the
// products take 8,000 cycles of 29,000, instructions issue in 47 %; a warp is held by the products that it issues, so warp 0 cuts no part of the state (all sixteen: 232 us, 224 without it).
// Measured, 8,192 tokens of 32 heads: 214 us.  While products had one part (224): q and angles row by row from memory and outputs and gates a row a
// thread 292, the latter alone 240; a warp group per operand, which leaves 64 to 112 registers a thread and spills, 253 to 288; a warp that only issues products, 112 registers, 274.
//   columns of tensor memory: q's terms, then P's 0-191; a product's two parts 192-447: the scores, what the state gives, P v in turn
__global__ void __launch_bounds__(kThreads, 1)
retention_outputs_kernel(const Retention p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023) & ~1023u, keys = base, state = base + 3 * kTerm, values = base + 6 * kTerm;
    const uint32_t raw_k = keys + 2 * kTerm, raw_q = state, angles = state + kTerm;
    uint8_t* sm = smem_raw + (base - smem_u32(smem_raw));
    float* plain = reinterpret_cast<float*>(sm);                                          // for the form token by token
    float (*squares)[kT] = reinterpret_cast<float (*)[kT]>(sm + 6 * kTerm);               // where the values have been read
    __shared__ Shared sh;
    __shared__ __align__(8) uint64_t scores_done;
    __shared__ float power[kT + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, part = warp >> 2, row = (warp & 3) * 32 + lane, col = part * 32, quad = lane & 15;
    if (threadIdx.x == 0) fa::mbar_init(smem_u32(&scores_done), 1);
    const uint32_t tmem = (uint32_t)fa::uniform((int)begin(sh));
    const uint32_t mine = tmem + ((uint32_t)((warp & 3) * 32) << 16), one = 192, two = 320;
    const bool issuer = fa::uniform(warp) == 0;
    uint32_t round = 0;
    int last_h = -1;
    bool ok = true;
    struct Item { int e, h, first, n, place, seg, inner; };      // inner: the chunk's number in its segment
    __shared__ Item items[2];                        // this item and the next one, n = 0 after the last
    int at = blockIdx.x;
    auto find = [&](Item& t) {                       // by one thread
        t.n = 0;
        for (; at < p.places * p.H && t.n <= 0; at += gridDim.x) {
            const int place = at / p.H;
            int first, n;
            const int e = chunk_of<kT>(place, p.cu_q, p.entries, first, n);
            if (n <= 0) continue;
            const int chunk = place - p.cu_q[e] / kT - e, seg = min(chunk / p.seg_chunks, p.segments - 1);
            t = Item{e, at - place * p.H, first, n, place, seg, chunk - seg * p.seg_chunks};
        }
        t.n = max(t.n, 0);
    };
    auto fetch = [&](const Item& t) {
        fetch_rows(p, raw_k, p.k_off, t.first, t.n, t.h);
        fetch_rows(p, raw_q, p.q_off, t.first, t.n, t.h);
        fetch_angles(p, angles, t.first, t.n);
        walk::cp_commit();
    };
    auto angle = [&](int r, int c) { return angle_at(p, sm + 4 * kTerm, r, c); };
    if (threadIdx.x == 32) find(items[0]);
    __syncthreads();
    if (items[0].n > 0) fetch(items[0]);
    grid_dependency_wait();                          // the states at the chunks' and the segments' starts (angles and powers are older than the kernel before this one)
    for (uint32_t j = 0; items[j & 1].n > 0; ++j) {
        const Item& t = items[j & 1];
        const Item& next = items[(j & 1) ^ 1];
        const int first = t.first, n = t.n, h = t.h;
        const bool in = row < n;
        if (h != last_h) {                           // (read last before the barriers of the item before)
            for (int i = threadIdx.x; i <= kT; i += kThreads) power[i] = p.powers[(size_t)h * p.powers_pitch + i];
            last_h = h;
        }
        const float* S = p.states + ((size_t)t.place * p.H + h) * (kD * kD);
        const float* S_seg = t.seg > 0 ? p.starts + ((size_t)(t.e * p.segments + t.seg) * p.H + h) * (kD * kD) : nullptr;
        const float lead = S_seg != nullptr ? chunks_power(p, h, t.inner) : 0.f;
        // the state at the chunk's start: a column of it per warp at a time, four of them ahead; none for the warp that issues, which the scores' products hold
        constexpr int kOthers = kThreads / 32 - 1;
        float4 own_S[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) own_S[i] = issuer ? make_float4(0.f, 0.f, 0.f, 0.f) : ld4(S + (size_t)(kOthers * i + warp - 1) * kD + 4 * lane);
        walk::cp_wait<0>();
        __syncthreads();                             // k, q and angles are there
        fetch_rows(p, values, p.v_off, first, n, h);
        walk::cp_commit();
        {
            uint2 lo[4], hi[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = 32 * i + 2 * warp + (lane >> 4);
                const uint8_t* from = sm + 2 * kTerm + fa::sw128(r, quad >> 1) + (quad & 1) * 8;
                lo[i] = *reinterpret_cast<const uint2*>(from);
                hi[i] = *reinterpret_cast<const uint2*>(from + kHalf);
            }
            __syncthreads();                         // before the last of k's terms takes its place
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = 32 * i + 2 * warp + (lane >> 4);
                put_pairs(keys, r, quad, lo[i], hi[i], angle(r, 2 * quad), angle(r, 2 * quad + 1), p.k_scale);
            }
        }
        // q: a row and 16 pairs of columns a thread, to tensor memory
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const uint8_t* from = sm + 3 * kTerm + fa::sw128(row, part * 2 + x);
            const uint4 a = *reinterpret_cast<const uint4*>(from), b = *reinterpret_cast<const uint4*>(from + kHalf);
            const uint32_t a4[4] = {a.x, a.y, a.z, a.w}, b4[4] = {b.x, b.y, b.z, b.w};
            uint32_t lo[3][4], hi[3][4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float a0 = __uint_as_float(a4[j] << 16), a1 = __uint_as_float(a4[j] & 0xffff0000u), b0 = __uint_as_float(b4[j] << 16), b1 = __uint_as_float(b4[j] & 0xffff0000u);
                const float4 cs = angle(row, part * 8 + 4 * x + j);
                rotate(make_float2(cs.x, cs.y), a0, b0);
                rotate(make_float2(cs.z, cs.w), a1, b1);
                uint32_t w[3];
                cut(a0, a1, w);
#pragma unroll
                for (int y = 0; y < 3; ++y) lo[y][j] = w[y];
                cut(b0, b1, w);
#pragma unroll
                for (int y = 0; y < 3; ++y) hi[y][j] = w[y];
            }
#pragma unroll
            for (int y = 0; y < 3; ++y) {
                st4(mine + y * 64 + part * 8 + 4 * x, lo[y]);
                st4(mine + y * 64 + 32 + part * 8 + 4 * x, hi[y]);
            }
        }
        wait_st();
        fence_smem();
        fence_before();
        __syncthreads();                             // q and the angles have been read
        if (issuer) {
            fence_after();
            if (fa::elect_one()) {
                product_ts<false, 3>(tmem + one, tmem + two, tmem, keys, kHalf, kTerm, instr(kT, false, false));
                fa::umma_commit(smem_u32(&scores_done));
            }
            __syncwarp();
        } else {
#pragma unroll
            for (int i = 0; i < 12; i += 4) {
                float4 seg[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int c = kOthers * (i + j) + warp - 1;
                    if (c >= kD) continue;
                    if (i > 0) own_S[j] = ld4(S + (size_t)c * kD + 4 * lane);
                    if (S_seg != nullptr) seg[j] = ld4(S_seg + (size_t)c * kD + 4 * lane);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int c = kOthers * (i + j) + warp - 1;
                    if (c >= kD) continue;
                    float4 v = own_S[j];
                    if (S_seg != nullptr) v = make_float4(fmaf(lead, seg[j].x, v.x), fmaf(lead, seg[j].y, v.y), fmaf(lead, seg[j].z, v.z), fmaf(lead, seg[j].w, v.w));
                    put4(state + (lane >> 4) * kHalf, kTerm, c, quad, v);
                }
            }
        }
        // the scores give way to what the state gives (a wait that ran out shows in the next one)
        ok = warp_wait(sh, scores_done, j);
        fence_after();
        float v[32];
#pragma unroll
        for (int x = 0; x < 32; x += 16)
            if (col + x <= (row | 31)) ld_sum16(mine + one + col + x, mine + two + col + x, v + x);
        walk::cp_wait<0>();
        fence_smem();
        fence_before();
        __syncthreads();
        if (issuer) {
            fence_after();
            if (fa::elect_one()) {
                product_ts<false, 3>(tmem + one, tmem + two, tmem, state, kHalf, kTerm, instr(kD, false, false));
                fa::umma_commit(smem_u32(&sh.done));
            }
            __syncwarp();
        }
        if (threadIdx.x == 32) find(items[(j & 1) ^ 1]);
        __syncwarp();
        {
            uint32_t w[3][8];
            auto weights = [&](int half) {
#pragma unroll
                for (int x = 0; x < 16; x += 2) {    // (the table's index is one of its own also where it is not used)
                    const int s = col + 16 * half + x;
                    const float fa_ = power[(row - s) & 127], fb = power[(row - s - 1) & 127];
                    const float a = s <= row ? v[16 * half + x] * fa_ : 0.f, b = s < row ? v[16 * half + x + 1] * fb : 0.f;
                    uint32_t c[3];
                    cut(a, b, c);
#pragma unroll
                    for (int y = 0; y < 3; ++y) w[y][x / 2] = c[y];
                }
            };
            weights(0);
            if (!(ok = products_done(sh, round++, p.error, ok))) break;      // q's terms give way
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                if (half) weights(1);
#pragma unroll
                for (int y = 0; y < 3; ++y) st8(mine + y * 64 + part * 16 + 8 * half, w[y]);
            }
        }
        float o[32];
        const float f = power[row + 1];
#pragma unroll
        for (int y = 0; y < 32; y += 16) {           // what the state gives, before P v takes its place
            ld_sum16(mine + one + col + y, mine + two + col + y, o + y);
#pragma unroll
            for (int x = 0; x < 16; ++x) o[y + x] *= f;
        }
        wait_st();
        fence_before();
        __syncthreads();
        if (issuer) {
            fence_after();
            if (fa::elect_one()) {
                product_ts<true, 1>(tmem + one, tmem + two, tmem, values, kHalf, kTerm, instr(kD, false, true));
                fa::umma_commit(smem_u32(&sh.done));
            }
            __syncwarp();
        }
        if (next.n > 0) fetch(next);
        // the gates as the outputs are stored: 16 bytes of a row a thread, two rows a warp
        uint4 gates[4];
        if (p.out != nullptr)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = 32 * i + 2 * warp + (lane >> 4);
                gates[i] = *reinterpret_cast<const uint4*>(p.proj + (size_t)(first + min(r, n - 1)) * p.pitch + p.g_off + (size_t)h * kD + 8 * quad);
            }
        if (!(ok = products_done(sh, round++, p.error))) break;
        float z = 0.f, sum = 0.f;
#pragma unroll
        for (int y = 0; y < 32; y += 16) {
            float own[16];
            ld_sum16(mine + one + col + y, mine + two + col + y, own);
#pragma unroll
            for (int x = 0; x < 16; ++x) {
                o[y + x] += own[x];
                z = fmaf(o[y + x], 0.f, z);
                sum = fmaf(o[y + x], o[y + x], sum);
            }
        }
        squares[part][row] = sum;
        fence_before();
        if (__syncthreads_or(z != 0.f)) {            // token by token: a column of the state and 32 rows a thread
            walk::cp_wait<0>();                      // what has been fetched for the next chunk is fetched again afterwards
            __syncthreads();
            float* qs = plain;                       // [128][128]
            float* ks = qs + kT * kD;
            float* os = ks + kT * kD;
            float* sums = os + kT * kD;              // [2][4][128]
#pragma unroll 1
            for (int x = threadIdx.x; x < kT * kD; x += kThreads) {
                qs[x] = x / kD < n ? column_of(p, p.q_off, (size_t)first + x / kD, h, x % kD) : 0.f;
                ks[x] = x / kD < n ? key_of(p, (size_t)first + x / kD, h, x % kD) : 0.f;
            }
            const int c = threadIdx.x & 127, r0 = (threadIdx.x >> 7) * 32;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                o[j] = S[(size_t)c * kD + r0 + j];
                if (S_seg != nullptr) o[j] = fmaf(lead, S_seg[(size_t)c * kD + r0 + j], o[j]);
            }
            __syncthreads();
#pragma unroll 1
            for (int i = 0; i < n; ++i) {
                const float v = __bfloat162float(p.proj[(size_t)(first + i) * p.pitch + p.v_off + (size_t)h * kD + c]);
                float x = 0.f;
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    o[j] = fmaf(power[1], o[j], ks[i * kD + r0 + j] * v);
                    x = fmaf(qs[i * kD + r0 + j], o[j], x);
                }
                float* to = sums + (i & 1) * 4 * kD;
                to[(r0 / 32) * kD + c] = x;
                __syncthreads();
                if (r0 == 0) os[i * kD + c] = (to[c] + to[kD + c]) + (to[2 * kD + c] + to[3 * kD + c]);
            }
            __syncthreads();
            sum = 0.f;
#pragma unroll
            for (int x = 0; x < 32; ++x) {
                o[x] = in ? os[row * kD + col + x] : 0.f;
                sum = fmaf(o[x], o[x], sum);
            }
            __syncthreads();
            squares[part][row] = sum;
            __syncthreads();
            if (next.n > 0) fetch(next);
        }
        // through shared memory (where k's first two terms were), so that neighbouring threads store neighbours
#pragma unroll
        for (int x = 0; x < 8; ++x)
            *reinterpret_cast<float4*>(sm + row * 512 + (((8 * part + x) ^ (row & 7)) << 4)) = make_float4(o[4 * x], o[4 * x + 1], o[4 * x + 2], o[4 * x + 3]);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = 32 * i + 2 * warp + (lane >> 4);
            if (r >= n) continue;
            const float4 a = *reinterpret_cast<const float4*>(sm + r * 512 + (((2 * quad) ^ (r & 7)) << 4));
            const float4 b = *reinterpret_cast<const float4*>(sm + r * 512 + (((2 * quad + 1) ^ (r & 7)) << 4));
            float y[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            const size_t to = ((size_t)(first + r) * p.H + h) * kD + 8 * quad;
            if (p.out == nullptr) {
                store8(p.o + to, y);
                continue;
            }
            const float inv = 1.0f / sqrtf(((squares[0][r] + squares[1][r]) + (squares[2][r] + squares[3][r])) / (float)kD + p.eps);
            const uint32_t g4[4] = {gates[i].x, gates[i].y, gates[i].z, gates[i].w};
#pragma unroll
            for (int x = 0; x < 8; ++x) {
                const float g = __uint_as_float(x & 1 ? g4[x / 2] & 0xffff0000u : g4[x / 2] << 16);
                y[x] = y[x] * inv * __fdividef(g, 1.f + __expf(-g));
            }
            store8(p.out + to, y);
        }
    }
    walk::cp_wait<0>();
    end(sh);
}

static bool aligned(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace tiles
}  // namespace se

using namespace se::tiles;

// 1 for what the kernels below take: heads of 128 x 128, all of a head's columns turned or none
extern "C" int se_retention_tiles_supported(int d, int dv, int rotary) { return d == kD && dv == kD && (rotary == 0 || rotary == kD); }

// work: float [(tokens / 128 + entries) * heads * 128 * 128 (the chunks' states) + (segments > 1 ? entries * segments : 0) * heads * 128 * 128
// + heads * (130 + seg_chunks) rounded up to 4 + (rotary ? tokens * 128 : 0)].  An entry's chunks in `segments` of seg_chunks (all of the longest entry's).
// out: after norm and gate (columns from g_off on), or null: o.
extern "C" int se_retention_tiles(const void* proj, int pitch, int q_off, int k_off, int v_off, int g_off, const float* inv_freq, const int* positions,
                                  int rotary, float k_scale, const float* decay, float* state, long long state_stride, const int* cu_q,
                                  const int* seq_rows, void* out, float* o, float eps, float* work, int* error, int tokens, int entries, int heads, int d,
                                  int dv, int segments, int seg_chunks, int sms, cudaStream_t stream) {
    if (entries <= 0 || tokens <= 0) return 0;
    if (!se_retention_tiles_supported(d, dv, rotary) || heads <= 0 || heads > 65535 || entries > 65535) return SE_ERR_UNSUPPORTED;
    if (segments < 1 || seg_chunks < 1 || (out == nullptr) == (o == nullptr) || (rotary && (inv_freq == nullptr || positions == nullptr))) return SE_ERR_ARGUMENT;
    if (pitch % 8 || q_off % 8 || k_off % 8 || v_off % 8 || g_off % 8 || state_stride % 4 || !aligned(proj) || !aligned(work) || !aligned(state) ||
        (out != nullptr && !aligned(out)) || (o != nullptr && !aligned(o)))
        return SE_ERR_UNSUPPORTED;
    const long long places = tokens / kT + entries;
    if (places * heads > 0x7fffffffLL || (long long)entries * segments > 0x7fffffffLL || (long long)tokens * 64 > 0x7fffffffLL - 256) return SE_ERR_UNSUPPORTED;
    Retention p = {};
    p.proj = (const __nv_bfloat16*)proj; p.pitch = pitch; p.q_off = q_off; p.k_off = k_off; p.v_off = v_off; p.g_off = g_off;
    p.states = work;
    p.starts = p.states + (size_t)places * heads * kD * kD;
    p.powers_pitch = kT + 2 + seg_chunks;
    float* powers = p.starts + (segments > 1 ? (size_t)entries * segments * heads * kD * kD : 0);
    float2* turn = reinterpret_cast<float2*>(powers + ((size_t)heads * p.powers_pitch + 3) / 4 * 4);
    p.powers = powers; p.turn = rotary ? turn : nullptr;
    p.segments = segments; p.seg_chunks = seg_chunks; p.state = state; p.state_stride = state_stride; p.cu_q = cu_q; p.seq_rows = seq_rows;
    p.entries = entries; p.H = heads; p.places = (int)places; p.k_scale = k_scale; p.eps = eps; p.out = (__nv_bfloat16*)out; p.o = o; p.error = error;
    const int turn_blocks = rotary ? (tokens * 64 + 255) / 256 : 0, states_smem = 7 * kTerm + 1024, outputs_smem = 7 * kTerm + 1024;
    retention_tables_kernel<<<turn_blocks + heads, 256, 0, stream>>>(turn, positions, inv_freq, tokens, turn_blocks, powers, p.powers_pitch, decay);
    cudaError_t e = cudaFuncSetAttribute(retention_states_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, states_smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(retention_outputs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, outputs_smem);
    if (e != cudaSuccess) return (int)e;
    retention_states_kernel<<<dim3(entries * segments, heads), kThreads, states_smem, stream>>>(p);
    if (segments > 1) retention_join_kernel<<<dim3(16, heads, entries), 256, 0, stream>>>(p);
    const long long items = places * heads;
    if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
    return (int)SE_LAUNCH_DEPENDENT_IF(segments > 1, "ret", retention_outputs_kernel, dim3((unsigned)(items < sms ? items : sms)), dim3(kThreads), (size_t)outputs_smem, stream, p);
}
