// Plain paged attention: one block per (token, query head), any head size, any page
// size, float32 or bfloat16.  It is the 32-bit path's attention and the fallback for
// sizes the tensor-core kernels refuse.
//
// score = q·k * scale; query at position p sees keys max(0, p-window+1)..p of its own
// request (window 0 = all keys, window -n = the keys of p's own chunk of n positions); softmax state and accumulators in 32-bit; the
// probability is rounded to the activation type before it multiplies V; the output is
// rounded once.  The value head size `dv` may differ from the query/key size `d`: a page holds
// the keys [kv head][slot][d] and then the values [kv head][slot][dv].
// Options: `softcap` c > 0 caps the scaled score, s <- c tanh(s / c); `sink` adds a key of score 0
// that has no value (one more term, exp(0), in the softmax's denominator); `gate` (with its row
// pitch) multiplies the output element by element with sigmoid(gate[t][h * dv + i]), or with `gate_per_head` a
// whole head with sigmoid(gate[t][h]); `sink_logits`
// (one per query head) puts a learned logit in the place of the sink's 0, unscaled; `keep_first` n > 0
// (with a window) keeps keys 0..n-1 visible beside the window's; `slopes` (one per query head) takes
// slope * (i - j) off the score of query position i and key position j.  Reference: src/sparseengine/kernels/triton/context_flashattention_nopad.py:92-127,
// src/sparseengine/kernels/triton/gqa_flash_decoding_stage1.py:69-120.
//
// A block-table entry outside [0, num_pages) is not followed: the key is left out and a code
// goes to the error word (the reference checks such indices on the host behind a debug
// switch, src/sparseengine/layers/attention_backend.py:155-215).
#include "common.cuh"

namespace se {

constexpr int kMaxDimPerLane = 8;   // head_dim <= 256
constexpr int kAttnKeys = 4;        // keys of a warp in flight

// A block per (token, head), a warp per four keys in turn: their loads, and the shuffles that sum their scores, run side by side,
// and the running maximum moves once for the four.  What bounds it is the chain of loads and exponentials of a warp's keys one
// after another, so 16 warps share a token's keys where the blocks are few (a step of single tokens), 8 or 4 where they are many.
// Measured, 32-bit, 48 heads of 128, a layer's call, one key at a time by 4 warps and now: one request of 3,000 keys 1,262 and
// 248 us, four 1,325 and 396, sixty-four 2,818 and 2,014; of one key 49 and 50, 270 and 278.
template <typename T, int N, int WARPS>
__global__ void __launch_bounds__(32 * WARPS)
paged_attention_plain_kernel(const T* __restrict__ q, const T* __restrict__ cache, const int* __restrict__ table, int table_stride,
                             const int* __restrict__ seq_rows, const int* __restrict__ token_seq, const int* __restrict__ positions,
                             T* __restrict__ out, int hq, int hkv, int d, int dv, int page_size, float scale, int window, int num_pages,
                             int* __restrict__ error, float softcap, int sink, const T* __restrict__ gate, int gate_pitch,
                             const float* __restrict__ sink_logits, int keep_first, const float* __restrict__ slopes, int gate_per_head) {
    const int t = blockIdx.x, h = blockIdx.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int kvh = h / (hq / hkv);
    const int pos = positions[t];
    const int* row_table = table + (size_t)seq_rows[token_seq[t]] * table_stride;
    const int lo = first_visible(pos, window);
    const size_t page_elems = (size_t)hkv * page_size * (d + dv);
    const size_t v_off = (size_t)hkv * page_size * d + (size_t)kvh * page_size * dv;
    const size_t head_off = (size_t)kvh * page_size * d;

    float qr[N], acc[N];
    // the keys in the order they are visited: the kept first ones that lie before the window, then the window's
    const int kept = min(keep_first, lo), seen = kept + pos - lo + 1;
    const bool busy = warp * kAttnKeys < seen;
    const T* qp = q + ((size_t)t * hq + h) * d;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const int dim = lane + 32 * i;
        qr[i] = busy && dim < d ? to_float(qp[dim]) * scale : 0.f;
        acc[i] = 0.f;
    }
    float m = -INFINITY, l = 0.f;
    const float slope = slopes != nullptr ? slopes[h] : 0.f;
    for (int n0 = warp * kAttnKeys; n0 < seen; n0 += WARPS * kAttnKeys) {
        const T* vp[kAttnKeys];
        float s[kAttnKeys], v[kAttnKeys][N];
        bool there[kAttnKeys];                       // a warp-uniform choice: keys behind the last and on bad pages are left out
#pragma unroll
        for (int x = 0; x < kAttnKeys; ++x) {
            const int n = n0 + x, j = n < kept ? n : lo + n - kept;
            const int page = n < seen ? row_table[j / page_size] : 0;
            there[x] = n < seen && page_in_pool(page, num_pages, error, SE_CODE_BAD_PAGE_ATTN_PLAIN);
            const T* from = cache + (size_t)(there[x] ? page : 0) * page_elems;
            const T* kp = from + head_off + (size_t)(j % page_size) * d;
            vp[x] = from + v_off + (size_t)(j % page_size) * dv;
            s[x] = 0.f;
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const int dim = lane + 32 * i;
                if (there[x] && dim < d) s[x] += qr[i] * to_float(kp[dim]);
            }
        }
#pragma unroll
        for (int x = 0; x < kAttnKeys; ++x)
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const int dim = lane + 32 * i;
                v[x][i] = there[x] && dim < dv ? to_float(vp[x][dim]) : 0.f;
            }
        float m_new = m;
        bool any = false;
#pragma unroll
        for (int x = 0; x < kAttnKeys; ++x) {
            any |= there[x];
            const int n = n0 + x, j = n < kept ? n : lo + n - kept;
            s[x] = warp_sum(s[x]);
            if (softcap > 0.f) s[x] = softcap * tanhf(s[x] / softcap);
            s[x] -= slope * (float)(pos - j);
            if (there[x]) m_new = fmaxf(m_new, s[x]);
        }
        if (!any) continue;
        const float base = m_new == -INFINITY ? 0.f : m_new;         // scores of -inf weigh nothing, those that are no numbers show
        const float corr = expf(m - base);           // m = -inf on the first keys: exp(-inf) = 0
        l *= corr;
#pragma unroll
        for (int i = 0; i < N; ++i) acc[i] *= corr;
#pragma unroll
        for (int x = 0; x < kAttnKeys; ++x) {
            if (!there[x]) continue;
            const float p = expf(s[x] - base);
            const float pr = round_act<T>(p);
            l += p;
#pragma unroll
            for (int i = 0; i < N; ++i) acc[i] += pr * v[x][i];
        }
        m = m_new;
    }

    __shared__ float sm[WARPS], sl[WARPS];
    __shared__ float sacc[WARPS][32 * N];
    if (lane == 0) { sm[warp] = m; sl[warp] = l; }
    const int live = min(WARPS, (seen + kAttnKeys - 1) / kAttnKeys);           // warps that had keys
    if (warp < live)
#pragma unroll
        for (int i = 0; i < N; ++i) sacc[warp][lane + 32 * i] = acc[i];
    __syncthreads();
    float mt = -INFINITY;
    for (int w = 0; w < live; ++w) mt = fmaxf(mt, sm[w]);
    const float sink_logit = sink_logits != nullptr ? sink_logits[h] : 0.f;
    if (sink) mt = fmaxf(mt, sink_logit);
    float lt = sink ? expf(sink_logit - mt) : 0.f;
    for (int w = 0; w < live; ++w) lt += sl[w] == 0.f ? 0.f : sl[w] * expf(sm[w] - mt);     // 0: no key
    T* op = out + ((size_t)t * hq + h) * dv;
    for (int dim = threadIdx.x; dim < dv; dim += blockDim.x) {
        float o = 0.f;
        for (int w = 0; w < live; ++w) o += sl[w] == 0.f ? 0.f : sacc[w][dim] * expf(sm[w] - mt);
        o /= lt;
        if (gate != nullptr) o /= 1.f + expf(-to_float(gate[(size_t)t * gate_pitch + (gate_per_head ? (size_t)h : (size_t)h * dv + dim)]));
        op[dim] = from_float<T>(o);
    }
}

}  // namespace se

extern "C" int se_paged_attention_plain(const void* q, const void* cache, const int* table, int table_stride,
                                        const int* seq_rows, const int* token_seq, const int* positions, void* out,
                                        int tokens, int hq, int hkv, int d, int dv, int page_size, float scale, int window,
                                        int num_pages, int* error, float softcap, int sink, const void* gate, int gate_pitch,
                                        const float* sink_logits, int keep_first, const float* slopes, int gate_per_head, int sms, int dtype,
                                        cudaStream_t stream) {
    // sms: the device's SMs
    if (tokens <= 0) return 0;
    if (sms < 1) return SE_ERR_ARGUMENT;
    if (softcap < 0.f || (gate != nullptr && gate_pitch < (gate_per_head ? hq : hq * dv)) || keep_first < 0) return SE_ERR_ARGUMENT;
    if (sink_logits != nullptr) sink = 1;
    if (window <= 0) keep_first = 0;
    if (d > 32 * se::kMaxDimPerLane || d <= 0 || dv > 32 * se::kMaxDimPerLane || dv <= 0 || hkv <= 0 || hq % hkv)
        return SE_ERR_UNSUPPORTED;
    const dim3 grid(tokens, hq);
    const bool wide = d > 128 || dv > 128;
    const long long blocks = (long long)tokens * hq;
#define SE_PLAIN(N, WARPS)                                                                                                  \
    se::paged_attention_plain_kernel<T, N, WARPS><<<grid, 32 * WARPS, 0, stream>>>(                                        \
        (const T*)q, (const T*)cache, table, table_stride, seq_rows, token_seq, positions, (T*)out, hq, hkv, d, dv, page_size, \
        scale, window, num_pages, error, softcap, sink, (const T*)gate, gate_pitch, sink_logits, keep_first, slopes, gate_per_head)
    SE_DISPATCH_DTYPE(dtype, T, {
        // as many warps as leave all blocks on the device at once (64 registers a thread; 96 for the wide heads)
        if (wide && blocks <= sms) SE_PLAIN(8, 16);
        else if (wide) SE_PLAIN(8, 4);
        else if (blocks <= 2 * sms) SE_PLAIN(4, 16);
        else if (blocks <= 4 * sms) SE_PLAIN(4, 8);
        else SE_PLAIN(4, 4);
    });
#undef SE_PLAIN
    SE_LAUNCH_CHECK();
}
