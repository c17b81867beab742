// Prompt-portion attention on 5th-generation tensor cores (bfloat16, head size 128).
//
// One CTA per (batch entry, KV head, 256 query rows); a row is one (query token, query head
// of the GQA group) pair, token-major, so 128 rows span ~21 tokens of M2 and all six heads
// that share the KV head.  The CTA holds two query tiles of 128 rows, each with its own four
// softmax warps and its own MMA-issuing warp; the two tiles take turns on the tensor pipe and
// share every 64-key K/V tile that is loaded.  Per query tile and K/V tile:
//
//   S = Q·Kᵀ        tcgen05.mma, M 128 x N 64 x K 128, Q and K K-major in shared memory
//                   (128-byte swizzle), S in tensor memory (two buffers per query tile);
//   softmax         four warps, one thread per row: tcgen05.ld of its row of S, mask
//                   (causal, window, end of keys), running maximum and sum in 32-bit, P
//                   rounded to bfloat16 and written back to tensor memory over the row's
//                   scores (tcgen05.st, two values per column);
//   O += P·V        tcgen05.mma with the A operand (P) in tensor memory, M 128 x N 128 x K 64,
//                   V straight from its pages (dims contiguous: the MN-major B operand), O in
//                   tensor memory.
//
// Tensor memory is used in full: O of the two tiles (2 x 128 columns) and their S buffers
// (2 x 2 x 64), whose first halves hold P between the softmax and P·V; shared memory holds
// the two Q tiles and five K/V stages.  The running maximum only moves when a row's maximum grows by more than 2^8
// (then O and the sum are rescaled), so O is read back from tensor memory rarely; the final
// division by the sum is exact for whatever reference maximum was used.
//
// Warp roles (12 warps): warps 0 and 10 gather K/V tiles from their pages with cp.async into
// five stages, alternately, and tie each tile's barrier to their copies
// (cp.async.mbarrier.arrive.noinc), so a tile is announced the moment it has landed and the
// loaders never wait for data; warp 1 owns tensor memory and issues the MMAs of query tile 0,
// warp 11 those of tile 1 (S(j) first, then P·V of tile j-1 as its P arrives), independently
// of one another; warps 2-5 and 6-9 are the softmax/epilogue warps of tiles 0 and 1.  A K/V
// stage is free again when both issuers have committed its P·V.  Every mbarrier wait is
// bounded and reports through the error word.  The softmax's options (a cap on the scores, a sink
// of score 0, an output gate; mma_util.cuh's SoftmaxOptions) cost the softmax warps two more
// special-function operations per score for the cap, an add and a multiply-add per score for a distance
// bias, one term in the last sum for the sink, and one load and exponential per output element for the gate.  Arithmetic as the reference's prefill kernel
// (src/sparseengine/kernels/triton/context_flashattention_nopad.py:92-127).
//
// With PARTS the same kernel runs latent attention over keys and values that were formed per head from the latents (heads of 64
// unrotated and 64 rotated dims, values of 64): a key's first half comes from a product's rows, its second, which all heads share, from
// the latents' rows, and no page is looked up.
#include "common.cuh"
#include "fa_util.cuh"
#include "mma_util.cuh"

#include <initializer_list>

namespace se {
namespace fa {

constexpr int D = 128;
constexpr int kRows = 128;
constexpr int kKeys = 64;
constexpr int kTiles = 2;                            // query tiles per CTA
constexpr int kStages = 5;
constexpr int kLoaderWarp2 = 2 + 4 * kTiles;         // the second loader warp
constexpr int kMmaWarp2 = kLoaderWarp2 + 1;          // the MMA issuer of query tile 1 (tile 0: warp 1)
constexpr int kThreads = 32 * (kMmaWarp2 + 1);       // loader, MMA, 4 softmax warps per query tile, loader, MMA
constexpr int kHalfBytes = 64 * 128;                 // [64 rows][64 dims] bf16: rows of 128 bytes
constexpr int kQBytes = 2 * kRows * 128;             // two dim-halves of [128 rows][64 dims]
constexpr int kKVStageBytes = 4 * kHalfBytes;        // K halves, V halves

using se::mma::smem_u32;
using se::mma::cp_async16;
using se::mma::cp_async_commit;

struct Bars {
    uint64_t kv_full[kStages], kv_empty[kStages];
    uint64_t s_full[kTiles][2], s_empty[kTiles][2];      // per query tile: two S buffers
    uint64_t p_full[kTiles][2], p_empty[kTiles];         // per query tile: P of a tile is complete (one per S buffer); its P·V has finished
    uint64_t o_done[kTiles];                             // per query tile: the last P·V has finished (a warp that never had to
                                                         // wait for p_empty may be phases behind it, so the end has a barrier of its own)
};

// Where keys and values formed per head lie: rows of the keys that the entries see, each entry's from the first key that its first token
// sees on, entry after entry.
struct Parts {
    int q_pitch;
    const __nv_bfloat16* kv;       // [rows][kv_pitch]: heads' 64 key dims, from v_off on their 64 value dims
    int kv_pitch, v_off;
    const __nv_bfloat16* rot;      // [rows][rot_pitch]: the shared 64 rotated dims
    int rot_pitch, rows;
};

// The n lowest bits (none below 0, all from 32 on).
__device__ __forceinline__ uint32_t low_bits(int n) { return n >= 32 ? 0xffffffffu : (1u << max(n, 0)) - 1u; }

template <bool PARTS>
__global__ void __launch_bounds__(kThreads, 1)
attn_prefill_tc_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ cache,
                       const int* __restrict__ table, int table_stride, const int* __restrict__ seq_rows,
                       const int* __restrict__ cu_q, const int* __restrict__ kv_len, __nv_bfloat16* __restrict__ out,
                       int* error, int hq, int hkv, int page_size, float scale_log2, int window, int num_pages,
                       const se::mma::SoftmaxOptions opt, const Parts parts) {
    constexpr int DV = PARTS ? 64 : D;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* q_s = smem;                               // [2 tiles][2 halves][128 rows][128 B]
    uint8_t* kv_s = q_s + kTiles * kQBytes;            // [stages][K half0, K half1, V half0, V half1]
    __shared__ __align__(8) Bars bars;
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int abort_s;

    // Blocks start in the order of their index, x fastest: the KV heads are x, and the row tiles
    // are y taken from the end, so that the tiles with the most keys (the last rows of a causal
    // portion) start first and the short ones fill the tail of the launch.
    const int entry = blockIdx.z, kvh = blockIdx.x;
    const int group = hq / hkv;
    const int tok0 = cu_q[entry];
    const int q_len = cu_q[entry + 1] - tok0;
    const int total_rows = q_len * group;
    const int row_base = (int)(gridDim.y - 1 - blockIdx.y) * (kTiles * kRows);
    if (row_base >= total_rows) return;
    const int kv_end = kv_len[entry];
    const int q_start = kv_end - q_len;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    const int last_row = min(row_base + kTiles * kRows, total_rows) - 1;
    const int max_pos = q_start + last_row / group;
    const int first_pos = q_start + row_base / group;
    const int k_lo = first_visible(first_pos, window);
    const int k_begin = (k_lo / kKeys) * kKeys;
    const int k_end = max_pos + 1;
    // first keys that stay visible beside a window: those before the CTA's window come as tiles of their own, ahead
    // of the window's (tile j < kept_tiles holds keys 64 j .., of which those below `kept` are read)
    const int keep_first = window > 0 ? opt.keep_first : 0;
    const int kept = min(keep_first, k_lo);
    const int kept_tiles = (kept + kKeys - 1) / kKeys;
    const int num_tiles = kept_tiles + (k_end - k_begin + kKeys - 1) / kKeys;

    // The tiles [j0, j1) that some row of query tile x sees: with few query heads to a KV head its 128 rows see up to
    // two tiles fewer than the CTA's 256 at either end, and a tile without rows sees none.
    auto seen_tiles = [&](int x, int& j0, int& j1) {
        const int row0 = row_base + x * kRows, row1 = min(row0 + kRows, total_rows) - 1;
        if (row0 > row1) { j0 = j1 = 0; return; }
        j0 = keep_first > 0 ? 0 : (first_visible(q_start + row0 / group, window) - k_begin) / kKeys;
        j1 = kept_tiles + (q_start + row1 / group + 1 - k_begin + kKeys - 1) / kKeys;
    };

    auto bar = [&](uint64_t* b) { return smem_u32(b); };
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) { mbar_init(bar(&bars.kv_full[s]), 32); mbar_init(bar(&bars.kv_empty[s]), kTiles); }   // full: every lane of the tile's loader warp; empty: both query tiles' MMAs
        for (int x = 0; x < kTiles; ++x) {
            for (int b = 0; b < 2; ++b) {
                mbar_init(bar(&bars.s_full[x][b]), 1);
                mbar_init(bar(&bars.s_empty[x][b]), 4);      // one arrival per softmax warp
            }
            mbar_init(bar(&bars.p_full[x][0]), 4);
            mbar_init(bar(&bars.p_full[x][1]), 4);
            mbar_init(bar(&bars.p_empty[x]), 1);
            mbar_init(bar(&bars.o_done[x]), 1);
        }
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // Q tiles: the softmax warps copy chunks, and the first K/V tiles are fetched meanwhile; rows beyond the portion's rows are zero-filled
    for (int i = threadIdx.x - 64; i < kTiles * kRows * 16 && warp >= 2 && warp < kLoaderWarp2; i += 32 * 4 * kTiles) {
        const int r = i >> 4, c = i & 15;                  // r: 0..255 over both tiles
        const int row = row_base + r;
        const bool ok = row < total_rows;
        const int rr = ok ? row : total_rows - 1;
        const __nv_bfloat16* src = (PARTS ? q + (size_t)(tok0 + rr) * parts.q_pitch + kvh * D
                                          : q + ((size_t)(tok0 + rr / group) * hq + kvh * group + rr % group) * D) + c * 8;
        cp_async16(smem_u32(q_s) + (r >> 7) * kQBytes + (c >> 3) * (kRows * 128) + sw128(r & 127, c & 7), src, ok);
    }
    cp_async_commit();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();                                       // barriers and tensor memory
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp != 0 && warp != kLoaderWarp2) {               // Q, for all that compute
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("bar.sync 1, %0;" ::"n"(kThreads - 64) : "memory");
    }
    const uint32_t tmem = tmem_base_s;
    // tensor memory: O of tile x in columns 128 x .. 128 x + 127; S buffer b of tile x in 256 + 128 x + 64 b ..
    auto tmem_o = [&](int x) { return tmem + (uint32_t)(128 * x); };
    auto tmem_s = [&](int x, int b) { return tmem + (uint32_t)(256 + 128 * x + 64 * b); };

    const int* row_table = PARTS ? nullptr : table + (size_t)seq_rows[entry] * table_stride;
    const size_t page_elems = (size_t)2 * hkv * page_size * D;
    const size_t head_off = (size_t)kvh * page_size * D;
    const size_t v_off = (size_t)hkv * page_size * D;

    const int k_lo_window = k_lo, k_end_window = k_end;
    if (warp == 0 || warp == kLoaderWarp2) {
        // ---- loaders: K/V tiles from their pages ------------------------------------------
        // Lane l looks up where keys base+l and base+32+l live (two independent table loads per
        // lane and tile); the copy loop gets each row's address by shuffle, so no load sits
        // between the asynchronous copies.
        int rows_before = 0;                             // PARTS: the rows of the entries before this one
        if constexpr (PARTS) {
            for (int e = lane; e < entry; e += 32) rows_before += kv_len[e] - first_visible(kv_len[e] - (cu_q[e + 1] - cu_q[e]), window);
            rows_before = __reduce_add_sync(0xffffffffu, rows_before) - first_visible(q_start, window);
        }
        auto issue = [&](int tile) {
            uint8_t* st = kv_s + (size_t)(tile % kStages) * kKVStageBytes;
            const bool first = tile < kept_tiles;
            const int base = first ? tile * kKeys : k_begin + (tile - kept_tiles) * kKeys;
            const int k_lo = first ? 0 : k_lo_window, k_end = first ? kept : k_end_window;      // the keys of this tile that are read
            if constexpr (PARTS) {                   // zero-filled outside [k_lo, k_end), as below, and beyond the last row
                const int c = lane & 7;
                const size_t row0 = (size_t)(rows_before + base);
                const __nv_bfloat16* kv = parts.kv + kvh * 64 + c * 8;
                const __nv_bfloat16* rot = parts.rot + c * 8;
#pragma unroll 4
                for (int k = 0; k < kKeys / 4; ++k) {
                    const int r = 4 * k + (lane >> 3);
                    const bool ok = base + r < k_end && base + r >= k_lo && rows_before + base + r < parts.rows;
                    const size_t row = ok ? row0 + r : 0;
                    const uint32_t off = sw128(r, c);
                    cp_async16(smem_u32(st) + off, kv + row * parts.kv_pitch, ok);
                    cp_async16(smem_u32(st) + kHalfBytes + off, rot + row * parts.rot_pitch, ok);
                    cp_async16(smem_u32(st) + 2 * kHalfBytes + off, kv + row * parts.kv_pitch + parts.v_off, ok);
                }
                return;
            }
            // Keys outside [k_lo, k_end) are zero-filled, never read: a page the window has left
            // behind may belong to another request by now.  An entry that names no page of the pool
            // is not followed either (address 0 marks its row; a code goes to the error word).
            unsigned long long src_row[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int j = min(max(base + 32 * h + lane, k_lo), k_end - 1);
                const int page = row_table[j / page_size];
                const bool in_pool = page_in_pool(page, num_pages, error, SE_CODE_BAD_PAGE_ATTN_PREFILL_TC);
                src_row[h] = in_pool ? (unsigned long long)(cache + (size_t)page * page_elems + head_off + (size_t)(j % page_size) * D) : 0ull;
            }
            const int c = lane & 15;
#pragma unroll 4
            for (int k = 0; k < kKeys / 2; ++k) {
                const int r = 2 * k + (lane >> 4);
                const unsigned long long a = __shfl_sync(0xffffffffu, src_row[0], r & 31);
                const unsigned long long b = __shfl_sync(0xffffffffu, src_row[1], r & 31);
                const unsigned long long row_addr = r < 32 ? a : b;
                const bool ok = base + r < k_end && base + r >= k_lo && row_addr != 0ull;
                const __nv_bfloat16* src = reinterpret_cast<const __nv_bfloat16*>(ok ? row_addr : (unsigned long long)cache) + c * 8;
                const uint32_t off = (c >> 3) * kHalfBytes + sw128(r, c & 7);
                cp_async16(smem_u32(st) + off, src, ok);
                cp_async16(smem_u32(st) + 2 * kHalfBytes + off, src + v_off, ok);
            }
        };
        // Two loader warps take alternate tiles and run ahead as far as stages are free.  Each
        // lane ties the tile's barrier to its own copies (cp.async.mbarrier.arrive.noinc: the
        // arrival happens when the lane's earlier copies have landed), so the warp never waits
        // for data and a tile is announced the moment it is complete.
        const int first = warp == 0 ? 0 : 1;
        bool ok = true;
        for (int tile = first; tile < num_tiles && ok; tile += 2) {
            if (tile >= kStages) ok = mbar_wait(bar(&bars.kv_empty[tile % kStages]), ((tile / kStages) - 1) & 1, &abort_s);
            if (!ok) break;
            issue(tile);
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar(&bars.kv_full[tile % kStages])) : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (!ok) { abort_s = 1; if (lane == 0) atomicCAS(error, 0, 11); }
    } else if (warp == 1 || warp == kMmaWarp2) {
        // ---- MMA issuers: one warp per query tile ---------------------------------------
        // Order for a tile: S(j), then P·V of tile j-1 as its P arrives; S(j+1) is thus issued
        // before the softmax of tile j has finished.  The two issuers share the tensor pipe and
        // do not wait for one another; a K/V stage is free when both have committed its P·V.
        // The warp runs as a whole through uniform loops and one elected lane issues (fa_util.cuh): 8,192 tokens behind 16,384 keys 4,145 us,
        // issued under a divergent branch and with two more shuffles a tile in the softmax 4,206.
        const int x = warp == 1 ? 0 : 1;
        const uint32_t id_s = idesc(kKeys, 0), id_o = idesc(DV, 1);
        const int tiles = uniform(num_tiles);
        int j0, j1;
        seen_tiles(x, j0, j1);
        j0 = uniform(j0);
        j1 = uniform(j1);
        const uint32_t tm = (uint32_t)uniform((int)tmem), o_at = tm + 128 * x, s_at = tm + 256 + 128 * x;
        const uint64_t q_desc = desc_kmajor(smem_u32(q_s) + x * kQBytes);
        bool ok = true;
        auto wait = [&](uint64_t* b, uint32_t parity) {
            ok = __all_sync(0xffffffffu, mbar_wait(bar(b), parity, &abort_s));
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        };
        auto issue_pv = [&](int i, int stage) {
            wait(&bars.p_full[x][i & 1], (i >> 1) & 1);
            if (ok && elect_one()) {
                const uint64_t v = desc_mnmajor(smem_u32(kv_s) + stage * kKVStageBytes + 2 * kHalfBytes, kHalfBytes);
                const uint32_t pa = s_at + 64 * (i & 1);     // P of tile i lies over the first half of its S buffer
#pragma unroll
                for (int kk = 0; kk < kKeys / 16; ++kk)      // 16 keys per MMA: 8 columns of P, two 8-key groups of V
                    umma_ts(o_at, pa + (uint32_t)(kk * 8), v + (uint64_t)(kk * 128), id_o, (i > 0 || kk > 0) ? 1u : 0u);
                umma_commit(bar(&bars.p_empty[x]));
                umma_commit(bar(&bars.kv_empty[stage]));
            }
            __syncwarp();
        };
        int stage = 0, before = 0;                           // of tiles j and j - 1
        uint32_t turn = 0;                                   // how often the stages have gone round, modulo 2
        for (int j = 0; j < tiles && ok; ++j) {
            const int i = j - j0, b = i & 1;                 // S, P and their barriers count the query tile's own tiles
            wait(&bars.kv_full[stage], turn);
            if (j < j0 || j >= j1) {                         // not seen: the stage goes back (its last turn has ended, for it is full)
                if (ok && j == j1 && i > 0) issue_pv(i - 1, before);
                if (ok && elect_one()) mbar_arrive(bar(&bars.kv_empty[stage]));
                __syncwarp();
                stage = stage + 1 == kStages ? 0 : stage + 1;
                if (stage == 0) turn ^= 1;
                continue;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // the copies were generic-proxy writes
            if (ok && i >= 2) wait(&bars.s_empty[x][b], ((i >> 1) - 1) & 1);
            if (ok && elect_one()) {
                const uint64_t k_desc = desc_kmajor(smem_u32(kv_s) + stage * kKVStageBytes);
#pragma unroll
                for (int kb = 0; kb < 2; ++kb)
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        umma(s_at + 64 * b, q_desc + (uint64_t)(kb * (kRows * 128 / 16) + kk * 2), k_desc + (uint64_t)(kb * (kHalfBytes / 16) + kk * 2), id_s,
                             (kb > 0 || kk > 0) ? 1u : 0u);
                umma_commit(bar(&bars.s_full[x][b]));
            }
            __syncwarp();
            if (ok && i >= 1) issue_pv(i - 1, before);
            before = stage;
            stage = stage + 1 == kStages ? 0 : stage + 1;
            if (stage == 0) turn ^= 1;
        }
        if (ok && j1 == tiles && j1 > j0) issue_pv(j1 - j0 - 1, before);
        if (ok && elect_one()) umma_commit(bar(&bars.o_done[x]));
        __syncwarp();
        if (!ok && lane == 0) { abort_s = 1; atomicCAS(error, 0, 12); }
    } else if (warp < 2 + 4 * kTiles) {
        // ---- softmax and epilogue: warps 2-5 own query tile 0, warps 6-9 tile 1; one thread per row ----
        const int x = (warp - 2) >> 2;
        const int quarter = warp & 3;
        const int r = quarter * 32 + lane;                 // row of the tile = TMEM lane
        const int row = row_base + x * kRows + r;
        const bool valid = row < total_rows;
        const int rr = valid ? row : total_rows - 1;
        const int pos = q_start + rr / group;
        const int lo = first_visible(pos, window);
        const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
        float m_ref = -INFINITY, l = 0.f;                  // reference maximum (log2 units), running sum
        const float slope = se::mma::raw_slope(opt, kvh * group + rr % group);      // distance bias per token, raw units
        const int pos_first = __shfl_sync(0xffffffffu, pos, 0), lo_last = __shfl_sync(0xffffffffu, lo, 31);
        bool ok = true;
        int j0, j1;
        seen_tiles(x, j0, j1);
        for (int j = j0; j < j1 && ok; ++j) {
            const int i = j - j0, b = i & 1;
            if (!mbar_wait(bar(&bars.s_full[x][b]), (i >> 1) & 1, &abort_s)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            uint32_t sv[64];
            tmem_ld32(tmem_s(x, b) + lane_addr, sv);
            tmem_ld32(tmem_s(x, b) + 32 + lane_addr, sv + 32);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(&bars.s_empty[x][b]));
            if (opt.cap_in > 0.f) {
                // A polynomial form where every score of the warp's 32 x 64 block is small (the warp decides
                // as one: no divergence), else the exact form with its two more special-function operations.
                float amax = 0.f;
#pragma unroll
                for (int c = 0; c < 64; ++c) amax = fmaxf(amax, fabsf(__uint_as_float(sv[c])));
                const uint32_t wmax = __reduce_max_sync(0xffffffffu, __float_as_uint(amax));    // non-negative floats order as integers
                se::mma::cap_scores_by<64>(reinterpret_cast<float*>(sv), __uint_as_float(wmax) * opt.cap_in, opt.cap_in, opt.cap_out);
            }
            const bool first = j < kept_tiles;
            const int key0 = first ? j * kKeys : k_begin + (j - kept_tiles) * kKeys;
            // the distance bias slope * (key - pos): its part within the tile joins the scores here, the tile's first
            // key's (log2 units) joins the maximum and the exponents below
            float tile_bias = 0.f;
            if (opt.slopes != nullptr) {
                tile_bias = slope * (float)(key0 - pos) * scale_log2;
#pragma unroll
                for (int c = 1; c < 64; ++c) sv[c] = __float_as_uint(fmaf(slope, (float)c, __uint_as_float(sv[c])));
            }
            // A tile every row of the warp sees in full needs no masking (rows ascend with the
            // lane: lane 0 has the smallest position, lane 31 the largest window start).  A tile of kept first keys
            // is seen by every row as far as it holds such keys; in a window's tile a key before the row's window is
            // seen if it is a kept one that no tile of kept keys has brought.
            const bool full = first ? key0 + kKeys <= kept
                                    : key0 + kKeys - 1 <= pos_first && key0 >= lo_last && key0 >= kept;
            if (!full) {
                // a bit per key, so that a key costs a test and a select: compared key by key a tile took 1.7 us more than a full one
                const int shown = first ? kept - key0 : pos + 1 - key0;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t bits = low_bits(shown - 32 * h);
                    if (!first) bits &= (~low_bits(lo - key0 - 32 * h) | low_bits(keep_first - key0 - 32 * h)) & ~low_bits(kept - key0 - 32 * h);
#pragma unroll
                    for (int c = 0; c < 32; ++c)
                        if (!(bits & (1u << c))) sv[32 * h + c] = 0xff800000u;      // -inf
                }
            }
            float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};  // four chains instead of one of 64
#pragma unroll
            for (int c = 0; c < 64; c += 4) {
                m4[0] = fmaxf(m4[0], __uint_as_float(sv[c]));
                m4[1] = fmaxf(m4[1], __uint_as_float(sv[c + 1]));
                m4[2] = fmaxf(m4[2], __uint_as_float(sv[c + 2]));
                m4[3] = fmaxf(m4[3], __uint_as_float(sv[c + 3]));
            }
            float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
            mx = fmaf(mx, scale_log2, tile_bias);                        // log2 units (scale > 0)
            // move the reference maximum only on the first visible keys or a large jump
            float factor = 1.f;
            bool need = false;
            if (mx > m_ref + kRescaleThreshold || (m_ref == -INFINITY && mx != -INFINITY)) {
                factor = m_ref == -INFINITY ? 0.f : exp2f(m_ref - mx);
                need = m_ref != -INFINITY;
                m_ref = mx;
                l *= factor;
            }
            if (__any_sync(0xffffffffu, need)) {
                // O must be at rest: P·V of the previous tile has finished.  (Only then: a warp whose
                // rows keep their reference maximum runs on, up to a tile ahead of the others, which
                // is why P's barrier exists once per S buffer.)
                if (i >= 1 && !mbar_wait(bar(&bars.p_empty[x]), (i - 1) & 1, &abort_s)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
                for (int c0 = 0; c0 < DV; c0 += 32) {
                    uint32_t ov[32];
                    tmem_ld32(tmem_o(x) + c0 + lane_addr, ov);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int c = 0; c < 32; ++c) ov[c] = __float_as_uint(__uint_as_float(ov[c]) * (need ? factor : 1.f));
                    tmem_st32(tmem_o(x) + c0 + lane_addr, ov);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            }
            const float m_use = m_ref == -INFINITY ? 0.f : m_ref;
            float sum4[4] = {0.f, 0.f, 0.f, 0.f};
            const float neg_m = tile_bias - m_use;
            // P goes back to tensor memory, over the row's own scores (which are in registers now):
            // two bfloat16 per column, the A operand of P·V.
            uint32_t packed[32];
#pragma unroll
            for (int c8 = 0; c8 < 8; ++c8) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    // p = 2^(s * scale - m): one fused multiply-add and one ex2 per element
                    const float p0 = ex2(fmaf(__uint_as_float(sv[c8 * 8 + 2 * i]), scale_log2, neg_m));
                    const float p1 = ex2(fmaf(__uint_as_float(sv[c8 * 8 + 2 * i + 1]), scale_log2, neg_m));
                    sum4[i] += p0 + p1;
                    packed[c8 * 4 + i] = se::mma::pack_bf16(p0, p1);
                }
            }
            tmem_st32(tmem_s(x, b) + lane_addr, packed);
            l += (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(&bars.p_full[x][b]));
        }
        if (ok && mbar_wait(bar(&bars.o_done[x]), 0, &abort_s)) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // the sink's term 2^(0 - m): it grows beyond the type only where the keys hold nothing (the output is 0 then)
            if (opt.sink) l += exp2f(se::mma::sink_log2(opt, kvh * group + rr % group) - m_ref);
            const float inv = 1.f / l;
            __nv_bfloat16* dst = out + ((size_t)(tok0 + rr / group) * hq + kvh * group + rr % group) * DV;
            const bool gate_vec = opt.gate != nullptr && !opt.gate_per_head && se::mma::gate_rows_aligned(opt, 16);
            const __nv_bfloat16* gp = opt.gate != nullptr
                ? se::mma::gate_of(opt, tok0 + rr / group, kvh * group + rr % group, D) : nullptr;
            const float inv_gated = gp != nullptr && opt.gate_per_head ? se::mma::gated(inv, gp) : inv;     // one gate per head: in the factor
            const bool gate_each = gp != nullptr && !opt.gate_per_head;
#pragma unroll 1
            for (int c0 = 0; c0 < DV; c0 += 32) {
                uint32_t ov[32];
                tmem_ld32(tmem_o(x) + c0 + lane_addr, ov);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (valid) {
#pragma unroll
                    for (int c = 0; c < 32; c += 8) {
                        uint32_t w[4];
                        uint4 graw = make_uint4(0u, 0u, 0u, 0u);           // eight gate values in one load where the rows allow it
                        if (gate_each && gate_vec) graw = *reinterpret_cast<const uint4*>(gp + c0 + c);
                        const __nv_bfloat162* g2 = reinterpret_cast<const __nv_bfloat162*>(&graw);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            float a = __uint_as_float(ov[c + 2 * i]) * inv_gated, b = __uint_as_float(ov[c + 2 * i + 1]) * inv_gated;
                            if (gate_each) {
                                if (gate_vec) {
                                    const float2 g = __bfloat1622float2(g2[i]);
                                    a = se::mma::gated_by(a, g.x);
                                    b = se::mma::gated_by(b, g.y);
                                } else {
                                    a = se::mma::gated(a, gp + c0 + c + 2 * i);
                                    b = se::mma::gated(b, gp + c0 + c + 2 * i + 1);
                                }
                            }
                            w[i] = se::mma::pack_bf16(a, b);
                        }
                        *reinterpret_cast<uint4*>(dst + c0 + c) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                }
            }
        } else {
            abort_s = 1;
            atomicCAS(error, 0, 13);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

}  // namespace fa
}  // namespace se

extern "C" int se_attn_prefill_tc_supported(int head_dim, int hq, int hkv) {
    return (head_dim == 128 && hkv > 0 && hq % hkv == 0) ? 1 : 0;
}

extern "C" int se_attn_prefill_tc(const void* q, const void* cache, const int* table, int table_stride,
                                  const int* seq_rows, const int* cu_q, const int* kv_len, void* out, int* error,
                                  int entries, int max_q_len, int hq, int hkv, int head_dim, int page_size, float scale,
                                  int window, int num_pages, float softcap, int sink, const void* gate, int gate_pitch,
                                  const float* sink_logits, int keep_first, const float* slopes, int gate_per_head, cudaStream_t stream) {
    using namespace se::fa;
    if (entries <= 0 || max_q_len <= 0) return 0;
    if (!se_attn_prefill_tc_supported(head_dim, hq, hkv) || entries > 65535 || hkv > 65535) return SE_ERR_UNSUPPORTED;
    if (softcap < 0.f || !(scale > 0.f) || (gate != nullptr && gate_pitch < (gate_per_head ? hq : hq * head_dim)) || keep_first < 0)
        return SE_ERR_ARGUMENT;
    const se::mma::SoftmaxOptions opt{softcap > 0.f ? scale / softcap : 0.f, softcap > 0.f ? softcap / scale : 0.f,
                                      sink || sink_logits != nullptr, (const __nv_bfloat16*)gate, gate_pitch, sink_logits,
                                      window > 0 ? keep_first : 0, slopes, 1.f / scale, gate_per_head};
    const size_t smem = (size_t)kTiles * kQBytes + kStages * kKVStageBytes + 1024;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(attn_prefill_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const int group = hq / hkv;
    const int row_tiles = se::ceil_div(max_q_len * group, kTiles * kRows);
    if (row_tiles > 65535) return SE_ERR_UNSUPPORTED;
    dim3 grid(hkv, row_tiles, entries);
    attn_prefill_tc_kernel<false><<<grid, kThreads, smem, stream>>>(
        (const __nv_bfloat16*)q, (const __nv_bfloat16*)cache, table, table_stride, seq_rows, cu_q, kv_len,
        (__nv_bfloat16*)out, error, hq, hkv, page_size, scale * 1.4426950408889634f, window, num_pages, opt, Parts{});
    return (int)cudaGetLastError();
}

// Latent attention over keys and values formed per head: heads of 64 unrotated and 64 rotated dims (q's rows: heads x 128, already
// rotated), values of 64 (the pointers as struct Parts has them); out [tokens][heads][64].  window: 0 none, else the keys a token sees.
extern "C" int se_attn_prefill_tc_parts(const void* q, int q_pitch, const void* kv, int kv_pitch, int v_off, const void* rot,
                                        int rot_pitch, int rows, const int* cu_q, const int* kv_len, const float* sink_logits, void* out,
                                        int* error, int entries, int max_q_len, int heads, float scale, int window, cudaStream_t stream) {
    using namespace se::fa;
    if (entries <= 0 || max_q_len <= 0) return 0;
    if (heads <= 0 || heads > 65535 || entries > 65535 || q_pitch % 8 || kv_pitch % 8 || v_off % 8 || rot_pitch % 8) return SE_ERR_UNSUPPORTED;
    if (!(scale > 0.f) || window < 0) return SE_ERR_ARGUMENT;
    for (const void* x : {q, kv, rot, (const void*)out})
        if (reinterpret_cast<uintptr_t>(x) & 15) return SE_ERR_UNSUPPORTED;
    const se::mma::SoftmaxOptions opt{0.f, 0.f, sink_logits != nullptr, nullptr, 0, sink_logits, 0, nullptr, 1.f / scale, 0};
    const Parts parts{q_pitch, (const __nv_bfloat16*)kv, kv_pitch, v_off, (const __nv_bfloat16*)rot, rot_pitch, rows};
    const size_t smem = (size_t)kTiles * kQBytes + kStages * kKVStageBytes + 1024;
    const cudaError_t e = cudaFuncSetAttribute(attn_prefill_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    const int row_tiles = se::ceil_div(max_q_len, kTiles * kRows);
    if (row_tiles > 65535) return SE_ERR_UNSUPPORTED;
    attn_prefill_tc_kernel<true><<<dim3(heads, row_tiles, entries), kThreads, smem, stream>>>(
        (const __nv_bfloat16*)q, nullptr, nullptr, 0, nullptr, cu_q, kv_len, (__nv_bfloat16*)out, error, heads, heads, 1,
        scale * 1.4426950408889634f, window, 0, opt, parts);
    return (int)cudaGetLastError();
}
