// Paged attention for prompt portions in 32-bit: one block per (batch entry, KV head, tile of 128 query rows), a "row"
// being one (query token, query head of the GQA group) pair, token-major, so that every K/V tile in shared memory serves
// all the heads that share it.  32-bit operands stay on the CUDA cores; the bound is the FMA rate.
//
// The kernel with one block per (token, head) (attention_plain.cu), which this one relieves of prompt portions, reads every
// key once per query row (from L2, 8 bytes per FMA pair) and spends five shuffles per key.  Here a thread keeps 8 rows x 4
// keys of scores and 8 rows x 4 or 8 columns of the output in registers: three 16-byte shared-memory reads per 32 (scores)
// and four per 64 (output) FMAs.  Keys arrive while the output of the tile before is summed and values while the scores
// are (cp.async).  Rows are private to a warp, so the softmax needs no barrier, and a warp without rows (a decoding request beside a
// prompt brings one per head of its group) only copies.  Measured at MiniMax M2's sizes (48 heads
// over 8, head size 128), prompts of 1, 300, 1,024 and 2,047 tokens in one step: 2.3 ms against about 26 ms.
//
// Query/key and value head sizes that are multiples of 4 up to 128; the options are the plain kernel's, and so is what a query
// sees (first_visible, keep_first).  Exponentials are expf, the probabilities stay 32-bit.  A block-table entry outside
// [0, num_pages) is not followed: its key is left out and a code goes to the error word.  A key that a row does not see does
// not touch it, whatever it holds: where a tile's values are not all finite, its products are left out (those of a seen key whose
// weight underflows to zero are not: there infinity times zero shows, as in the plain kernel).
#include "common.cuh"
#include <type_traits>

namespace se {
namespace f32 {

constexpr int kRows = 128, kKeys = 64, kThreads = 256;
constexpr int kPPitch = kKeys + 4;

struct Options {
    float softcap;                 // 0: none
    int sink;
    const float* gate;
    int gate_pitch, gate_per_head;
    const float* sink_logits;
    int keep_first;
    const float* slopes;
};

__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// DVT: value columns of the tile (64 or 128; those beyond dv stay zero)
template <int DVT>
__global__ void __launch_bounds__(kThreads, 1)
attn_prefill_f32_kernel(const float* __restrict__ q, const float* __restrict__ cache, const int* __restrict__ table,
                        int table_stride, const int* __restrict__ seq_rows, const int* __restrict__ cu_q,
                        const int* __restrict__ kv_len, float* __restrict__ out, int hq, int hkv, int d, int dv, int page_size,
                        float scale, int window, int num_pages, int* __restrict__ error, const Options opt) {
    constexpr int kCols = DVT / 16;                  // output columns per thread: 4 per group of 64
    extern __shared__ __align__(16) float sm[];
    const int dp = d + 4;                            // row pitch: eight neighbouring rows' 16-byte reads hit 32 banks
    float* qs = sm;                                  // [kRows][dp]
    float* ks = qs + kRows * dp;                     // [kKeys][dp]
    float* vs = ks + kKeys * dp;                     // [kKeys][DVT]
    float* ps = vs + kKeys * DVT;                    // [kRows][kPPitch]
    __shared__ int key_ok[2][kKeys];                 // whether a tile's key may be used (two tiles in flight)

    const int entry = blockIdx.z, kvh = blockIdx.x, group = hq / hkv;
    const int tok0 = cu_q[entry], q_len = cu_q[entry + 1] - tok0;
    const int total_rows = q_len * group;
    const int row_base = (int)(gridDim.y - 1 - blockIdx.y) * kRows;      // tiles with the most keys start first
    if (row_base >= total_rows) return;
    const int kv_end = kv_len[entry], q_start = kv_end - q_len;
    const int tid = threadIdx.x, tr = tid >> 4, tc = tid & 15;
    const bool live = row_base + (tid >> 5) * 16 < total_rows;           // this warp has rows

    const int last_row = min(row_base + kRows, total_rows) - 1;
    const int k_end = q_start + last_row / group + 1;
    const int k_lo = first_visible(q_start + row_base / group, window);
    const int kept = min(window > 0 ? opt.keep_first : 0, k_lo);
    const int kept_tiles = (kept + kKeys - 1) / kKeys;
    const int win_tile0 = max(k_lo / kKeys, kept_tiles);       // a tile that holds kept keys and the window's is visited once
    const int num_tiles = kept_tiles + max(0, (k_end + kKeys - 1) / kKeys - win_tile0);
    auto tile_key = [&](int it) { return (it < kept_tiles ? it : win_tile0 + it - kept_tiles) * kKeys; };

    const int* row_table = table + (size_t)seq_rows[entry] * table_stride;
    const size_t page_elems = (size_t)hkv * page_size * (d + dv);
    const size_t k_off = (size_t)kvh * page_size * d;
    const size_t v_off = (size_t)hkv * page_size * d + (size_t)kvh * page_size * dv;
    auto may_see = [&](int j) { return j < k_end && (j >= k_lo || j < kept); };

    // a tile's keys (or values) to shared memory; rows that no query of the block sees, and rows of bad pages, are zeros
    auto load = [&](int it, bool values) {
        const int j0 = tile_key(it), w4 = (values ? DVT : d) / 4, real4 = (values ? dv : d) / 4;
        for (int i = tid; i < kKeys * w4; i += kThreads) {
            const int r = i / w4, c = i - r * w4, j = j0 + r;
            float* dst = values ? vs + r * DVT + c * 4 : ks + r * dp + c * 4;
            bool ok = may_see(j);
            if (ok && c < real4) {
                const int page = row_table[j / page_size];
                ok = page_in_pool(page, num_pages, error, SE_CODE_BAD_PAGE_ATTN_PREFILL);
                if (ok) cp_async16(dst, cache + (size_t)page * page_elems + (values ? v_off + (size_t)(j % page_size) * dv
                                                                                   : k_off + (size_t)(j % page_size) * d) + c * 4);
            } else if (c >= real4) {
                ok = false;
            }
            if (!ok) *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
            if (!values && c == 0) key_ok[it & 1][r] = ok;
        }
        cp_commit();
    };
    load(0, false);
    load(0, true);
    // queries, times the scale
    for (int i = tid; i < kRows * (d / 4); i += kThreads) {
        const int r = i / (d / 4), c = i - r * (d / 4), row = row_base + r;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < total_rows) v = *reinterpret_cast<const float4*>(q + ((size_t)(tok0 + row / group) * hq + kvh * group + row % group) * d + c * 4);
        *reinterpret_cast<float4*>(qs + r * dp + c * 4) = make_float4(v.x * scale, v.y * scale, v.z * scale, v.w * scale);
    }

    int pos[8], first[8];                            // this thread's rows tr * 8 + i
    float m[8], l[8], slope[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int row = min(row_base + tr * 8 + i, total_rows - 1);
        pos[i] = q_start + row / group;
        first[i] = first_visible(pos[i], window);
        slope[i] = opt.slopes != nullptr ? opt.slopes[kvh * group + row % group] : 0.f;
        m[i] = -INFINITY;
        l[i] = 0.f;
    }
    float o[8][kCols] = {};
    const int keep_first = window > 0 ? opt.keep_first : 0;

    for (int it = 0; it < num_tiles; ++it) {
        const int j0 = tile_key(it);
        cp_wait<1>();                                // this tile's keys (its values may still be on their way)
        __syncthreads();
        if (live) {
            float s[8][4] = {};
            for (int k = 0; k < d; k += 4) {
                float4 kv[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) kv[c] = *reinterpret_cast<const float4*>(ks + (tc + 16 * c) * dp + k);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float4 qv = *reinterpret_cast<const float4*>(qs + (tr * 8 + i) * dp + k);
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        s[i][c] = fmaf(qv.w, kv[c].w, fmaf(qv.z, kv[c].z, fmaf(qv.y, kv[c].y, fmaf(qv.x, kv[c].x, s[i][c]))));
                }
            }
            int ok[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) ok[c] = key_ok[it & 1][tc + 16 * c];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float top = -INFINITY;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int j = j0 + tc + 16 * c;
                    float v = s[i][c];
                    if (opt.softcap > 0.f) v = opt.softcap * tanhf(v / opt.softcap);
                    v -= slope[i] * (float)(pos[i] - j);
                    s[i][c] = ok[c] && j <= pos[i] && (j >= first[i] || j < keep_first) ? v : -INFINITY;
                    top = fmaxf(top, s[i][c]);
                }
#pragma unroll
                for (int x = 8; x > 0; x >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x));
                const float m_new = fmaxf(m[i], top), base = m_new == -INFINITY ? 0.f : m_new;
                const float corr = expf(m[i] - base);    // nothing seen so far: exp(-inf) = 0
                m[i] = m_new;
                float sum = 0.f;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float p = expf(s[i][c] - base);
                    sum += p;
                    ps[(tr * 8 + i) * kPPitch + tc + 16 * c] = p;
                }
                l[i] = l[i] * corr + sum;
#pragma unroll
                for (int c = 0; c < kCols; ++c) o[i][c] *= corr;
            }
        }
        __syncthreads();                             // all warps are done with the keys
        if (it + 1 < num_tiles) load(it + 1, false);
        else cp_commit();
        cp_wait<1>();                                // this tile's values
        int odd = 0;                                 // a value that is not finite, among those this thread brought
        for (int i = tid; i < kKeys * (DVT / 4); i += kThreads) {
            const float4 v = reinterpret_cast<const float4*>(vs)[i];
            odd |= !(isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(v.w));
        }
        odd = __syncthreads_or(odd);
        auto add_values = [&](auto guarded) {
            for (int k = 0; k < kKeys; k += 4) {
                float4 p[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) p[i] = *reinterpret_cast<const float4*>(ps + (tr * 8 + i) * kPPitch + k);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    float v[kCols];
#pragma unroll
                    for (int g = 0; g < kCols / 4; ++g)
                        *reinterpret_cast<float4*>(v + 4 * g) = *reinterpret_cast<const float4*>(vs + (k + kk) * DVT + g * 64 + tc * 4);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float pv = kk == 0 ? p[i].x : kk == 1 ? p[i].y : kk == 2 ? p[i].z : p[i].w;
                        const int j = j0 + k + kk;
                        if (decltype(guarded)::value && !(key_ok[it & 1][k + kk] && j <= pos[i] && (j >= first[i] || j < keep_first))) continue;
#pragma unroll
                        for (int c = 0; c < kCols; ++c)
                            o[i][c] = fmaf(pv, v[c], o[i][c]);
                    }
                }
            }
        };
        if (live) {
            if (odd) add_values(std::true_type{});
            else add_values(std::false_type{});
        }
        __syncthreads();                             // all warps are done with the values
        if (it + 1 < num_tiles) load(it + 1, true);
        else cp_commit();
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int row = row_base + tr * 8 + i;
        float sum = l[i];
#pragma unroll
        for (int x = 8; x > 0; x >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
        if (row >= total_rows) continue;
        const int t = tok0 + row / group, h = kvh * group + row % group;
        float factor = 1.f;
        if (opt.sink) {
            const float logit = opt.sink_logits != nullptr ? opt.sink_logits[h] : 0.f, top = fmaxf(m[i], logit);
            factor = m[i] == -INFINITY ? 0.f : expf(m[i] - top);
            sum = sum * factor + expf(logit - top);
        }
        const float inv = factor / sum;
        float* dst = out + ((size_t)t * hq + h) * dv;
#pragma unroll
        for (int g = 0; g < kCols / 4; ++g) {
            const int c0 = g * 64 + tc * 4;
            if (c0 >= dv) continue;
            float v[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                v[c] = o[i][4 * g + c] * inv;
                if (opt.gate != nullptr)
                    v[c] /= 1.f + expf(-opt.gate[(size_t)t * opt.gate_pitch + (opt.gate_per_head ? (size_t)h : (size_t)h * dv + c0 + c)]);
            }
            *reinterpret_cast<float4*>(dst + c0) = make_float4(v[0], v[1], v[2], v[3]);
        }
    }
}

template <int DVT>
int launch(dim3 grid, size_t smem, cudaStream_t stream, const float* q, const float* cache, const int* table, int table_stride,
           const int* seq_rows, const int* cu_q, const int* kv_len, float* out, int hq, int hkv, int d, int dv, int page_size,
           float scale, int window, int num_pages, int* error, const Options& opt) {
    const cudaError_t e = cudaFuncSetAttribute(attn_prefill_f32_kernel<DVT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    attn_prefill_f32_kernel<DVT><<<grid, kThreads, smem, stream>>>(q, cache, table, table_stride, seq_rows, cu_q, kv_len, out, hq,
                                                                  hkv, d, dv, page_size, scale, window, num_pages, error, opt);
    return (int)cudaGetLastError();
}

}  // namespace f32
}  // namespace se

extern "C" int se_attn_prefill_f32_supported(int d, int dv, int hq, int hkv) {
    return d > 0 && d <= 128 && d % 4 == 0 && dv > 0 && dv <= 128 && dv % 4 == 0 && hkv > 0 && hkv <= 65535 && hq % hkv == 0;
}

// q: [tokens, hq, head_dim]; out: [tokens, hq, v_head_dim]; the other arguments as se_attn_prefill's, all of it in 32-bit.
extern "C" int se_attn_prefill_f32(const float* q, const float* cache, const int* table, int table_stride, const int* seq_rows,
                                   const int* cu_q, const int* kv_len, float* out, int entries, int max_q_len, int hq, int hkv,
                                   int head_dim, int v_head_dim, int page_size, float scale, int window, int num_pages, int* error,
                                   float softcap, int sink, const float* gate, int gate_pitch, const float* sink_logits,
                                   int keep_first, const float* slopes, int gate_per_head, cudaStream_t stream) {
    if (entries <= 0 || max_q_len <= 0) return 0;
    if (!se_attn_prefill_f32_supported(head_dim, v_head_dim, hq, hkv) || entries > 65535) return SE_ERR_UNSUPPORTED;
    if (softcap < 0.f || (gate != nullptr && gate_pitch < (gate_per_head ? hq : hq * v_head_dim)) || keep_first < 0) return SE_ERR_ARGUMENT;
    if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(cache) | reinterpret_cast<uintptr_t>(out)) & 15) return SE_ERR_UNSUPPORTED;
    const long long tiles = ((long long)max_q_len * (hq / hkv) + se::f32::kRows - 1) / se::f32::kRows;
    if (tiles > 65535) return SE_ERR_UNSUPPORTED;
    const se::f32::Options opt{softcap, sink || sink_logits != nullptr, gate, gate_pitch, gate_per_head, sink_logits, keep_first, slopes};
    const int dvt = v_head_dim <= 64 ? 64 : 128;
    const size_t smem = (size_t)((se::f32::kRows + se::f32::kKeys) * (head_dim + 4) + se::f32::kKeys * dvt + se::f32::kRows * se::f32::kPPitch) * sizeof(float);
    const dim3 grid(hkv, (int)tiles, entries);
    return (dvt == 64 ? se::f32::launch<64> : se::f32::launch<128>)(grid, smem, stream, q, cache, table, table_stride, seq_rows, cu_q,
                                                                    kv_len, out, hq, hkv, head_dim, v_head_dim, page_size, scale,
                                                                    window, num_pages, error, opt);
}
