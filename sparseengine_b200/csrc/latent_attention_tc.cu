// Latent attention over prompt portions on 5th-generation tensor cores (bfloat16).
//
// The absorbed form has one key/value head: a cached row of rank + rot elements is the key of every head, its first `rank`
// elements the value.  A query row is one (token, head) pair, token-major, so 128 rows span a few tokens and all their heads.
// One CTA per (batch entry, 256 query rows): two query tiles of 128 rows share every 64-key tile that is loaded, and a tile of
// cached rows in shared memory serves both products: S = Q K^T reads it K-major (64 dims per 128-byte row), O += P V reads the
// first rank / 64 of the same blocks MN-major.  S, P (over its scores) and O are in tensor memory: O of two tiles takes 2 rank
// columns, which leaves two S buffers per tile up to a rank of 128 and one at 192 (then the two tiles take turns: one's
// products run while the other's softmax does).
//
// The arrangement of barriers and the softmax are those of attention_prefill_tc.cu: four softmax warps per query tile, three
// loader warps, one MMA-issuing warp, every wait bounded and reported through the error word.
//
// What bounds it: at a row of 256 and a rank of 192 a key tile takes a query tile 1,150 cycles of the tensor pipe
// (128 x 64 x (256 + 192) multiply-adds, S at the rate its operands leave shared memory) and each softmax warp about 1,700 beside
// the other tile's; with one S buffer they follow one another, so a key tile takes the pair 3,700 cycles.  Measured, 32 heads,
// row 256, rank 192: 8,192 tokens with a window of 1,024 310 us (727 TFLOP/s), four prompts of 2,048 tokens 305, one 79.  The
// mma.sync kernel (latent_attention.cu) takes 866, 894 and 183: it stays for steps of few rows, which it splits along the keys,
// and for other sizes.
#include "common.cuh"
#include "fa_util.cuh"
#include "mma_util.cuh"
#include <cuda.h>
#include <mutex>

namespace se {
namespace lat_tc {

using namespace se::fa;
using se::mma::cp_async16;
using se::mma::cp_async_commit;
using se::mma::smem_u32;

constexpr int kRows = 128, kKeys = 64, kTiles = 2;
constexpr int kMaxStages = 5;
constexpr int kLoaders = 3;                          // warp 0 and those behind the softmax warps
constexpr int kLoaderWarp2 = 2 + 4 * kTiles;
constexpr int kThreads = 32 * (kLoaderWarp2 + kLoaders - 1);
constexpr int kKeyBlock = kKeys * 128;               // [64 keys][64 dims]: rows of 128 bytes
constexpr int kRowBlock = kRows * 128;               // [128 query rows][64 dims]

struct Bars {
    uint64_t kv_full[kMaxStages], kv_empty[kMaxStages];
    uint64_t s_full[kTiles][2], s_empty[kTiles][2];
    uint64_t p_full[kTiles][2], p_empty[kTiles];
    uint64_t o_done[kTiles], q_full[kTiles], all_done;
};

// db, rb: blocks of 64 dims of a row and of its latent part; buffers: S buffers per query tile; stages: key tiles in flight
__global__ void __launch_bounds__(kThreads, 1)
latent_attention_tc_kernel(const __grid_constant__ CUtensorMap q_map, const __nv_bfloat16* __restrict__ cache,
                           const int* __restrict__ table, int table_stride, const int* __restrict__ seq_rows,
                           const int* __restrict__ cu_q, const int* __restrict__ kv_len, const float* __restrict__ sink,
                           __nv_bfloat16* __restrict__ out, int heads, int db, int rb, int buffers, int stages, int page_size,
                           float scale_log2, int window, int num_pages, int* error) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int q_bytes = db * kRowBlock, stage_bytes = db * kKeyBlock, D = db * 64, rank = rb * 64;
    uint8_t* q_s = smem;                               // [2 tiles][db][128 rows][128 B]
    uint8_t* kv_s = q_s + kTiles * q_bytes;            // [stages][db][64 keys][128 B]
    __shared__ __align__(8) Bars bars;
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int abort_s;
    __shared__ unsigned long long row_list[kLoaders][kKeys];  // per loader warp: the addresses of a tile's rows

    const int entry = blockIdx.y;
    const int tok0 = cu_q[entry], q_len = cu_q[entry + 1] - tok0;
    const long long total_rows = (long long)q_len * heads;
    const long long row_base = (long long)(gridDim.x - 1 - blockIdx.x) * (kTiles * kRows);      // the tiles with the most keys start first
    if (row_base >= total_rows) return;
    const int kv_end = kv_len[entry], q_start = kv_end - q_len;
    const int warp = uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int n_rows = (int)min((long long)kTiles * kRows, total_rows - row_base);
    const int first_pos = q_start + (int)(row_base / heads), max_pos = q_start + (int)((row_base + n_rows - 1) / heads);
    const int k_lo = first_visible(first_pos, window);
    const int k_begin = (k_lo / kKeys) * kKeys, k_end = max_pos + 1;
    const int num_tiles = (k_end - k_begin + kKeys - 1) / kKeys;

    auto bar = [&](uint64_t* b) { return smem_u32(b); };
    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) { mbar_init(bar(&bars.kv_full[s]), 32); mbar_init(bar(&bars.kv_empty[s]), kTiles); }
        for (int x = 0; x < kTiles; ++x) {
            for (int b = 0; b < 2; ++b) {
                mbar_init(bar(&bars.s_full[x][b]), 1);
                mbar_init(bar(&bars.s_empty[x][b]), 4);
                mbar_init(bar(&bars.p_full[x][b]), 4);
            }
            mbar_init(bar(&bars.p_empty[x]), 1);
            mbar_init(bar(&bars.o_done[x]), 1);
            mbar_init(bar(&bars.q_full[x]), 1);
        }
        mbar_init(bar(&bars.all_done), 1);
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base_s;
    // one S buffer: O of tile x in columns 256 x .., its S behind; two: O in 128 x .., the S buffers in 256 + 128 x + 64 b ..
    auto tmem_o = [&](int x) { return tmem + (uint32_t)((buffers == 1 ? 256 : 128) * x); };
    auto tmem_s = [&](int x, int b) { return tmem + (uint32_t)(buffers == 1 ? 256 * x + 192 : 256 + 128 * x + 64 * b); };

    if (warp == 0 || warp >= kLoaderWarp2) {
        // ---- loaders: key tiles in turn, as far ahead as stages are free ----------------------
        const int* row_table = table + (size_t)seq_rows[entry] * table_stride;
        const int lanes = db > 2 ? 32 : db > 1 ? 16 : 8, c = lane & (lanes - 1), per = 32 / lanes;      // lanes per row, rows per pass
        // Where a tile's rows live: lane l looks two of them up (while the tile before is copied), all 64 addresses go through
        // shared memory, one broadcast read per row (4,900 cycles a tile and loader; 7,000 with two 64-bit shuffles and a choice
        // per row).  0: a row that is not read but zero-filled (keys outside
        // [k_lo, k_end): a page the window has left may belong to another request by now; an entry that names no page).
        const int tile0 = warp == 0 ? 0 : warp - kLoaderWarp2 + 1;
        unsigned long long* list = row_list[tile0];
        unsigned long long mine[2];
        auto look_up = [&](int tile) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int j = k_begin + tile * kKeys + 32 * h + lane;
                mine[h] = 0ull;
                if (j >= k_lo && j < k_end) {
                    const int page = row_table[j / page_size];
                    if (page_in_pool(page, num_pages, error, SE_CODE_BAD_PAGE_LATENT_TC))
                        mine[h] = (unsigned long long)(cache + ((size_t)page * page_size + j % page_size) * D);
                }
            }
        };
        const uint32_t c_off = (uint32_t)((c >> 3) * kKeyBlock);
        bool ok = true;
        if (tile0 < num_tiles) look_up(tile0);
        for (int tile = tile0; tile < num_tiles; tile += kLoaders) {
            __syncwarp();                              // the list of the tile before has been read
            list[lane] = mine[0];
            list[32 + lane] = mine[1];
            __syncwarp();
            if (tile + kLoaders < num_tiles) look_up(tile + kLoaders);
            if (tile >= stages) ok = mbar_wait(bar(&bars.kv_empty[tile % stages]), ((tile / stages) - 1) & 1, &abort_s);
            if (!ok) break;
            const uint32_t st = smem_u32(kv_s) + (uint32_t)((tile % stages) * stage_bytes) + c_off;
            if (c < db * 8) {
#pragma unroll 8
                for (int k = 0; k < kKeys; k += per) {
                    const int r = k + lane / lanes;
                    const unsigned long long row_addr = list[r];
                    cp_async16(st + sw128(r, c & 7), reinterpret_cast<const __nv_bfloat16*>(row_addr != 0ull ? row_addr : (unsigned long long)cache) + c * 8,
                               row_addr != 0ull);
                }
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar(&bars.kv_full[tile % stages])) : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (!ok) { abort_s = 1; if (lane == 0) atomicCAS(error, 0, 15); }
    } else if (warp == 1) {
        // ---- MMA issuer: one lane for both query tiles ---------------------------------------------
        // With one S buffer P V (j) and S (j + 1) of a tile go out together as its P (j) arrives (MMAs of one thread run in their
        // order, so P is read before S overwrites it), one tile's after the other's: the tiles' products then lie apart and each
        // tile's softmax runs beside the other's products.  With two, S (j) goes ahead of P V of tile j - 1.
        // The query tiles first: 128 rows that lie one behind the other, 64 dims at a time.  Rows behind the portion's are other
        // entries' or beyond the matrix (zeros): they are computed and dropped.
        if (elect_one())
            for (int x = 0; x < kTiles; ++x) {
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar(&bars.q_full[x])), "r"(q_bytes) : "memory");
                for (int kb = 0; kb < db; ++kb)
                    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                                 ::"r"(smem_u32(q_s) + (uint32_t)(x * q_bytes + kb * kRowBlock)), "l"(&q_map), "r"(bar(&bars.q_full[x])),
                                 "r"(64 * kb), "r"((int)((long long)tok0 * heads + row_base) + x * kRows) : "memory");
            }
        __syncwarp();
        const uint32_t id_s = idesc(kKeys, 0), id_o = idesc(rank, 1);
        const int tiles = uniform(num_tiles);
        const uint32_t tm = (uint32_t)uniform((int)tmem);
        auto o_at = [&](int x) { return tm + (uint32_t)((buffers == 1 ? 256 : 128) * x); };
        auto s_at = [&](int x, int b) { return tm + (uint32_t)(buffers == 1 ? 256 * x + 192 : 256 + 128 * x + 64 * b); };
        bool ok = true;
        auto wait = [&](uint64_t* b, uint32_t parity) { ok = __all_sync(0xffffffffu, mbar_wait(bar(b), parity, &abort_s)); };
        auto keys_ready = [&](int stage, uint32_t parity) {
            wait(&bars.kv_full[stage], parity);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");         // the copies were generic-proxy writes
        };
        auto issue_pv = [&](int x, int b, int stage, bool first) {
            const uint64_t v = desc_mnmajor(smem_u32(kv_s) + (uint32_t)(stage * stage_bytes), kKeyBlock);
            const uint32_t pa = s_at(x, b), o = o_at(x);
#pragma unroll
            for (int kk = 0; kk < kKeys / 16; ++kk) umma_ts(o, pa + (uint32_t)(kk * 8), v + (uint64_t)(kk * 128), id_o, (!first || kk > 0) ? 1u : 0u);
            umma_commit(bar(&bars.p_empty[x]));
            umma_commit(bar(&bars.kv_empty[stage]));
        };
        auto issue_s = [&](int x, int b, int stage) {
            uint64_t q = desc_kmajor(smem_u32(q_s) + (uint32_t)(x * q_bytes)), k = desc_kmajor(smem_u32(kv_s) + (uint32_t)(stage * stage_bytes));
            const uint32_t to = s_at(x, b);
            for (int kb = 0; kb < db; ++kb, q += kRowBlock / 16, k += kKeyBlock / 16)
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) umma(to, q + (uint64_t)(kk * 2), k + (uint64_t)(kk * 2), id_s, (kb > 0 || kk > 0) ? 1u : 0u);
            umma_commit(bar(&bars.s_full[x][b]));
        };
        for (int x = 0; x < kTiles && ok; ++x) wait(&bars.q_full[x], 0);
        int stage = 0;                                       // of tile j
        uint32_t turn = 0;                                   // how often the stages have gone round, modulo 2
        if (buffers == 1) {
            if (ok) keys_ready(0, 0);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (ok && elect_one())
                for (int x = 0; x < kTiles; ++x) issue_s(x, 0, 0);
            __syncwarp();
            for (int j = 0; j < tiles && ok; ++j) {
                const bool more = j + 1 < tiles;
                const int next = stage + 1 == stages ? 0 : stage + 1;
                const uint32_t next_turn = next == 0 ? turn ^ 1 : turn;
                if (more) keys_ready(next, next_turn);
                for (int x = 0; x < kTiles && ok; ++x) {
                    wait(&bars.p_full[x][0], j & 1);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (ok && elect_one()) {
                        issue_pv(x, 0, stage, j == 0);
                        if (more) issue_s(x, 0, next);
                    }
                    __syncwarp();
                }
                stage = next;
                turn = next_turn;
            }
        } else {
            int before = 0;                                  // the stage of tile j - 1
            for (int j = 0; j <= tiles && ok; ++j) {
                if (j < tiles) keys_ready(stage, turn);
                for (int x = 0; x < kTiles && ok; ++x) {
                    if (j < tiles) {
                        if (j >= 2) wait(&bars.s_empty[x][j & 1], ((j >> 1) - 1) & 1);
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        if (ok && elect_one()) issue_s(x, j & 1, stage);
                        __syncwarp();
                    }
                    if (j >= 1 && ok) {
                        wait(&bars.p_full[x][(j - 1) & 1], ((j - 1) >> 1) & 1);
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        if (ok && elect_one()) issue_pv(x, (j - 1) & 1, before, j == 1);
                        __syncwarp();
                    }
                }
                before = stage;
                stage = stage + 1 == stages ? 0 : stage + 1;
                if (stage == 0) turn ^= 1;
            }
        }
        if (ok && elect_one())
            for (int x = 0; x < kTiles; ++x) umma_commit(bar(&bars.o_done[x]));
        if (!ok) {       // a wait ran out: what is on its way into the block's memory ends (or runs out, too) before that is given back
            abort_s = 1;
            if (lane == 0) atomicCAS(error, 0, 16);
            if (elect_one()) umma_commit(bar(&bars.all_done));
            for (int x = 0; x < kTiles; ++x) mbar_drain(bar(&bars.q_full[x]), 0);
            mbar_drain(bar(&bars.all_done), 0);
        }
        __syncwarp();
    } else if (warp < 2 + 4 * kTiles) {
        // ---- softmax and epilogue: four warps per query tile, one thread per row --------------------
        const int x = (warp - 2) >> 2, quarter = warp & 3;
        const int r = x * kRows + quarter * 32 + lane;     // row of the CTA
        const bool valid = r < n_rows;
        const long long row = row_base + (valid ? r : n_rows - 1);
        const int pos = q_start + (int)(row / heads), lo = first_visible(pos, window);
        const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
        float m_ref = -INFINITY, l = 0.f;                  // reference maximum (log2 units), running sum
        bool ok = true;
        for (int j = 0; j < num_tiles && ok; ++j) {
            const int b = j % buffers;
            if (!mbar_wait(bar(&bars.s_full[x][b]), (j / buffers) & 1, &abort_s)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            uint32_t sv[64];
            tmem_ld32(tmem_s(x, b) + lane_addr, sv);
            tmem_ld32(tmem_s(x, b) + 32 + lane_addr, sv + 32);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(&bars.s_empty[x][b]));
            const int key0 = k_begin + j * kKeys;
            // a tile that every row of the warp sees in full needs no mask (rows ascend with the lane)
            if (!(key0 + kKeys - 1 <= __shfl_sync(0xffffffffu, pos, 0) && key0 >= __shfl_sync(0xffffffffu, lo, 31))) {
#pragma unroll
                for (int c = 0; c < 64; ++c)
                    if (key0 + c > pos || key0 + c < lo) sv[c] = 0xff800000u;      // -inf
            }
            float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int c = 0; c < 64; ++c) m4[c & 3] = fmaxf(m4[c & 3], __uint_as_float(sv[c]));
            const float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * scale_log2;       // scale > 0
            // the reference maximum moves on the first visible keys or a large jump only
            float factor = 1.f;
            bool need = false;
            if (mx > m_ref + kRescaleThreshold || (m_ref == -INFINITY && mx != -INFINITY)) {
                factor = m_ref == -INFINITY ? 0.f : exp2f(m_ref - mx);
                need = m_ref != -INFINITY;
                m_ref = mx;
                l *= factor;
            }
            if (__any_sync(0xffffffffu, need)) {           // O at rest: P V of the tile before has finished
                if (j >= 1 && !mbar_wait(bar(&bars.p_empty[x]), (j - 1) & 1, &abort_s)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
                for (int c0 = 0; c0 < rank; c0 += 32) {
                    uint32_t ov[32];
                    tmem_ld32(tmem_o(x) + c0 + lane_addr, ov);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int c = 0; c < 32; ++c) ov[c] = __float_as_uint(__uint_as_float(ov[c]) * (need ? factor : 1.f));
                    tmem_st32(tmem_o(x) + c0 + lane_addr, ov);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            }
            const float neg_m = m_ref == -INFINITY ? 0.f : -m_ref;
            float sum4[4] = {0.f, 0.f, 0.f, 0.f};
            uint32_t packed[32];
#pragma unroll
            for (int c = 0; c < 32; ++c) {
                const float p0 = ex2(fmaf(__uint_as_float(sv[2 * c]), scale_log2, neg_m));
                const float p1 = ex2(fmaf(__uint_as_float(sv[2 * c + 1]), scale_log2, neg_m));
                sum4[c & 3] += p0 + p1;
                packed[c] = se::mma::pack_bf16(p0, p1);
            }
            tmem_st32(tmem_s(x, b) + lane_addr, packed);   // P over the row's own scores
            l += (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(&bars.p_full[x][b]));
        }
        if (ok && mbar_wait(bar(&bars.o_done[x]), 0, &abort_s)) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (sink != nullptr) l += exp2f(fmaf(sink[(int)(row % heads)], 1.4426950408889634f, -m_ref));
            const float inv = 1.f / l;
            // A warp's 32 rows go through shared memory (its query tile's, whose last product has been read) and out as one run of
            // memory: row by row from the threads that hold them they took 11,800 cycles, a seventh of a block's time.
            uint8_t* stage = q_s + x * q_bytes + quarter * (32 * 2 * rank);
            const int chunks = rank / 8;                     // 16-byte chunks of a row
#pragma unroll 1
            for (int c0 = 0; c0 < rank; c0 += 32) {
                uint32_t ov[32];
                tmem_ld32(tmem_o(x) + c0 + lane_addr, ov);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int c = 0; c < 32; c += 8) {
                    uint32_t w[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        w[i] = se::mma::pack_bf16(__uint_as_float(ov[c + 2 * i]) * inv, __uint_as_float(ov[c + 2 * i + 1]) * inv);
                    *reinterpret_cast<uint4*>(stage + (lane * chunks + (((c0 + c) / 8) ^ (lane & 7))) * 16) = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
            __syncwarp();
            const int warp_rows = min(32, n_rows - x * kRows - quarter * 32);
            uint4* dst = reinterpret_cast<uint4*>(out + ((size_t)tok0 * heads + (size_t)row_base + x * kRows + quarter * 32) * rank);
#pragma unroll 4
            for (int i = lane; i < warp_rows * chunks; i += 32) {
                const int rr = i / chunks, c = i - rr * chunks;
                dst[i] = *reinterpret_cast<const uint4*>(stage + (rr * chunks + (c ^ (rr & 7))) * 16);
            }
        } else {
            abort_s = 1;
            atomicCAS(error, 0, 17);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)f;
    });
    return fn;
}

// The cached rows that a step's entries see (each from the first key that its first token sees on), entry after entry, without the pages
// between them: what a product that forms keys and values per head reads.  A warp per row, blocks of 32 rows.
__global__ void __launch_bounds__(256)
latent_gather_kernel(const __nv_bfloat16* __restrict__ cache, const int* __restrict__ table, int table_stride, const int* __restrict__ seq_rows,
                     const int* __restrict__ cu_q, const int* __restrict__ kv_len, __nv_bfloat16* __restrict__ out, int rows,
                     int row, int page_size, int window, int num_pages, int* error) {
    __shared__ int sums[8];
    const int e = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto first_of = [&](int x) { return first_visible(kv_len[x] - (cu_q[x + 1] - cu_q[x]), window); };
    int before = 0;
    for (int x = threadIdx.x; x < e; x += 256) before += kv_len[x] - first_of(x);
    before = __reduce_add_sync(0xffffffffu, before);
    if (lane == 0) sums[warp] = before;
    __syncthreads();
    before = 0;
#pragma unroll
    for (int x = 0; x < 8; ++x) before += sums[x];
    const int first = first_of(e), n = kv_len[e] - first;
    // the workspace is as large as the lengths that the host knows: beyond its end, or beyond the grid's, nothing is written
    if (threadIdx.x == 0 && blockIdx.x == 0 && (before + n > rows || n > (int)gridDim.x * 32)) atomicCAS(error, 0, SE_CODE_LATENT_ROWS);
    const int* pages = table + (size_t)seq_rows[e] * table_stride;
    for (int i = blockIdx.x * 32 + warp; i < min(min(n, rows - before), (int)(blockIdx.x + 1) * 32); i += 8) {
        const int j = first + i, page = pages[j / page_size];
        const bool there = page_in_pool(page, num_pages, error, SE_CODE_BAD_PAGE_LATENT_TC);
        const __nv_bfloat16* src = cache + ((size_t)(there ? page : 0) * page_size + j % page_size) * row;
        for (int c = lane * 8; c < row; c += 256)
            *reinterpret_cast<uint4*>(out + (size_t)(before + i) * row + c) = there ? *reinterpret_cast<const uint4*>(src + c) : make_uint4(0u, 0u, 0u, 0u);
    }
}

}  // namespace lat_tc
}  // namespace se

// A cached row of up to 256 and its latent part of up to 192, both in blocks of 64 (tensor memory holds 2 rank + 128 columns).
extern "C" int se_latent_attention_tc_supported(int rank, int rot) {
    return rank > 0 && rank <= 192 && rank % 64 == 0 && rot >= 0 && rot % 64 == 0 && rank + rot <= 256;
}

// Arguments as se_latent_attention_tiled's (which splits the keys of steps of few rows).
extern "C" int se_latent_attention_tc(const void* qfull, const void* cache, const int* table, int table_stride, const int* seq_rows,
                                      const int* cu_q, const int* kv_len, const float* sink, void* out, int tokens, int entries,
                                      int max_q_len, int heads, int rank, int rot, int page_size, float scale, int window, int num_pages, int* error,
                                      cudaStream_t stream) {
    using namespace se::lat_tc;
    if (entries <= 0 || max_q_len <= 0) return 0;
    if (!se_latent_attention_tc_supported(rank, rot) || heads <= 0 || entries > 65535) return SE_ERR_UNSUPPORTED;
    if (!(scale > 0.f) || page_size <= 0 || window < 0) return SE_ERR_ARGUMENT;
    if ((reinterpret_cast<uintptr_t>(qfull) | reinterpret_cast<uintptr_t>(cache) | reinterpret_cast<uintptr_t>(out)) & 15) return SE_ERR_UNSUPPORTED;
    const long long row_tiles = ((long long)max_q_len * heads + kTiles * kRows - 1) / (kTiles * kRows);
    if (row_tiles > 0x7fffffffLL) return SE_ERR_UNSUPPORTED;
    const int db = (rank + rot) / 64, rb = rank / 64, buffers = rank > 128 ? 1 : 2;
    const int room = 226 * 1024 - kTiles * db * kRowBlock;
    const int fit = room / (db * kKeyBlock), stages = fit < kMaxStages ? fit : kMaxStages;
    const size_t smem = (size_t)kTiles * db * kRowBlock + (size_t)stages * db * kKeyBlock + 1024;
    const EncodeTiledFn encode = encode_fn();
    if (encode == nullptr) return (int)cudaErrorNotSupported;
    CUtensorMap q_map;                                   // [tokens * heads][rank + rot], boxes of 128 rows and 64 dims
    const cuuint64_t dims[2] = {(cuuint64_t)(db * 64), (cuuint64_t)tokens * heads}, strides[1] = {(cuuint64_t)db * 128};
    const cuuint32_t box[2] = {64, kRows}, steps[2] = {1, 1};
    if ((long long)tokens * heads > 0x7fffffffLL - kTiles * kRows) return SE_ERR_UNSUPPORTED;
    if (encode(&q_map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(qfull), dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return SE_ERR_ARGUMENT;
    const cudaError_t e = cudaFuncSetAttribute(latent_attention_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    latent_attention_tc_kernel<<<dim3((unsigned)row_tiles, entries), kThreads, smem, stream>>>(
        q_map, (const __nv_bfloat16*)cache, table, table_stride, seq_rows, cu_q, kv_len, sink,
        (__nv_bfloat16*)out, heads, db, rb, buffers, stages, page_size, scale * 1.4426950408889634f, window, num_pages, error);
    return (int)cudaGetLastError();
}

// out [rows][row]: the cached rows (row elements, a multiple of 8) that the entries see; most_keys: the most that one entry sees.  Lengths on the device that
// go beyond either leave a code in the error word.
extern "C" int se_latent_gather(const void* cache, const int* table, int table_stride, const int* seq_rows, const int* cu_q, const int* kv_len,
                                void* out, int* error, int entries, int most_keys, int rows, int row, int page_size, int window,
                                int num_pages, cudaStream_t stream) {
    if (entries <= 0 || most_keys <= 0) return 0;
    if (rows < 0 || row <= 0 || row % 8 || page_size <= 0 || entries > 65535 || ((reinterpret_cast<uintptr_t>(cache) | reinterpret_cast<uintptr_t>(out)) & 15))
        return SE_ERR_UNSUPPORTED;
    se::lat_tc::latent_gather_kernel<<<dim3(se::ceil_div(most_keys, 32), entries), 256, 0, stream>>>(
        (const __nv_bfloat16*)cache, table, table_stride, seq_rows, cu_q, kv_len, (__nv_bfloat16*)out, rows, row, page_size, window, num_pages, error);
    SE_LAUNCH_CHECK();
}
