// 32-bit products on tcgen05, in tf32 terms: dense projections and the experts' grouped products of the float32 path.
//
// An operand is hi + lo, two tf32 values (11 bits of mantissa each); the tensor cores multiply hi hi, lo hi and hi lo.  Both matrices
// stay 32-bit in memory and are split on their way: TMA brings 128 weight rows (the M side) and up to 128 activation rows (the N side),
// 32 values along K each; other warps cut the weights into hi, the nearest tf32 value, and the rest and put both into tensor memory,
// from where they are the A operand, and put the activations' rest beside them in shared memory (their hi needs no copy: the
// tensor cores read the upper 19 bits).  Activations split by a kernel ahead took as long (2,048 rows by 8,192 x 3,072 weights: 513 us, 520 so then;
// the library 1,810) and a workspace of twice their size.
//
// The tensor cores cut sums off instead of rounding them, which a long sum shows: 2.5e-7 of the result per 32 products.  So hi hi
// runs over 64 products only, into one of two accumulators in turn, and four warps add those up in registers, rounded, while the
// next ones are multiplied; the small terms have an accumulator of their own over the whole of K.  Values that are not finite leave
// their hi hi sum not finite, as multiply-adds would; the small terms are then left out.
//
// What bounds it: with few activation rows the weights' bytes; with many the waits within a step, between the split, the products and the
// adding up (experts of 100 rows: tensor pipe 47 % busy, tensor memory 52 %, shared memory 44 %, issue 41 %; three tf32 products for each of the
// result's, at half the bf16 rate, would take half of its time).
//
// Where 32 bits end: rests below the smallest normal number are lost, so that operands below 2^-112 (weights) and 2^-116 (activations) lose digits,
// 1e-6 of the result there, 1e-4 another 2^6 further down.
//
// Warp roles (512 threads): 0 copies, 1 issues the products, 4-7 and 8-11 split what every other step needs (one such group took
// 1,000 cycles a step, most of it waiting, where the products take 770), 12-15 add up and store.  One CTA per
// SM (all of tensor memory), items dealt out in turn.  Every wait is bounded and reported through the error word.
#include "common.cuh"
#include "fa_util.cuh"
#include "glu.cuh"

#include <cuda.h>

#include <mutex>
#include <type_traits>

namespace se {
namespace f32tc {

using fa::mbar_arrive;
using fa::mbar_drain;
using fa::mbar_init;
using fa::mbar_wait;
using fa::sw128;

constexpr int kThreads = 512;
constexpr int kM = 128, kN = 128, kK = 32;           // kK floats: 128 bytes, one swizzle span
constexpr int kBoxRows = 64;                         // activation rows per copy: a tile takes the copies it has rows for
constexpr int kStages = 4;
constexpr int kTile = kM * kK * 4;                   // bytes of the weights, the activations and the activations' rest
constexpr int kStageBytes = 3 * kTile;
constexpr int kChunk = 2;                            // steps that a sum takes: 64 products
constexpr int kExchange = 2 * (kN / 2) * 64 * 4;     // gate and up rows change places
constexpr int kErrorCode = 18;
constexpr uint32_t kLow = 2 * kN, kSplit = 3 * kN;   // columns of tensor memory: sums 0 and kN, small terms, split weights [2][hi, lo][kK]

enum Mode { GATE_UP = 0, DOWN = 1, DENSE = 2 };

struct Params {
    const int* sorted;
    const int* offsets;
    const int* tile_expert;      // null: dense
    const int* tile_row0;
    const int* num_tiles;
    const float* route_w;
    const float* x;              // the activations, as the tensor map has them
    long long x_stride;
    float* out;                  // [rows][n_out]
    int* error;
    int rows, n_out, k_dim, blocks;
    int act_kind;
    float act_limit, act_alpha;
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void load_box(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y) : "memory");
}
// 16 bytes of shared memory by 32-bit address (the ring's base is rounded up, which would make its pointers generic ones)
__device__ __forceinline__ uint4 lds16(uint32_t at) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ void sts16(uint32_t at, uint4 v) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint32_t lds4(uint32_t at) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
    return v;
}
// kind::tf32, 32-bit sums, both operands K-major
__device__ __forceinline__ uint32_t instr(int n) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kM >> 4) << 24);
}
__device__ __forceinline__ void multiply(uint32_t d, uint32_t a_tmem, uint64_t b, uint32_t id, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a_tmem), "l"(b), "r"(id), "r"(accumulate) : "memory");
}

// the item's tile of activation rows and its block of outputs
struct Item { int expert, row0, valid, n0; };
template <int MODE>
__device__ __forceinline__ Item item_of(const Params& p, int i, int tiles) {
    constexpr int per = MODE == GATE_UP ? 64 : 128;
    Item it;
    if (MODE == DENSE) {                             // neighbours share weights, which then come from memory once
        const int tile = i % tiles;
        it.expert = 0;
        it.row0 = tile * kN;
        it.valid = min(kN, p.rows - it.row0);
        it.n0 = (i / tiles) * per;
    } else {
        const int tile = i / p.blocks;
        it.expert = p.tile_expert[tile];
        it.row0 = p.tile_row0[tile];
        it.valid = min(kN, p.offsets[it.expert + 1] - it.row0);
        it.n0 = (i - tile * p.blocks) * per;
    }
    return it;
}

// A NaN whose set bits all lie among the 13 that the tensor cores cut off an activation is read as an infinity: an infinite sum is looked at once more, with
// its row of activations, by a whole warp.  (Weights are looked after where they are split; activations are not rewritten there, where looking
// for such a NaN took the products 1 to 3 % longer.)
__device__ __forceinline__ bool has_nan(const float* row, int k_dim) {
    bool nan = false;
#pragma unroll 1
    for (int k = threadIdx.x & 31; k < k_dim; k += 32) nan = nan || isnan(row[k]);
    return __any_sync(0xffffffffu, nan);
}

template <int MODE>
__global__ void __launch_bounds__(kThreads, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const Params p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    float* exchange = reinterpret_cast<float*>(smem + kStages * kStageBytes);
    struct Bars {
        uint64_t full[kStages], empty[kStages], split_full[2], split_empty[2], sum_full[2], sum_empty[2], low_empty, meet, all_done;
    };
    __shared__ __align__(8) Bars bars;
    __shared__ float route_s[2][kN];
    __shared__ uint32_t tmem_s;
    __shared__ volatile int abort_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto bar = [](uint64_t* b) { return smem_addr(b); };

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) { mbar_init(bar(&bars.full[s]), 1); mbar_init(bar(&bars.empty[s]), 1); }
        for (int b = 0; b < 2; ++b) {
            mbar_init(bar(&bars.split_full[b]), 4);
            mbar_init(bar(&bars.split_empty[b]), 1);
            mbar_init(bar(&bars.sum_full[b]), 1);
            mbar_init(bar(&bars.sum_empty[b]), 4);
        }
        mbar_init(bar(&bars.low_empty), 4);
        mbar_init(bar(&bars.meet), 4);
        mbar_init(bar(&bars.all_done), 1);
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_addr(&tmem_s)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_s;
    const int tiles = MODE == DENSE ? ceil_div(p.rows, kN) : p.num_tiles[0];
    const int items = tiles * p.blocks, num_kb = ceil_div(p.k_dim, kK);
    bool ok = true;

    // registers: 512 threads x 128 at launch; 128 x (56 + 2 x 104 + 208) of the 65,536 afterwards
    if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == 0) {
        // the whole warp walks the loops and one elected lane copies: under a branch that the compiler takes for divergent a copy cost
        // 160 cycles (as the products do, fa_util.cuh)
        int it = 0;
        const int end = fa::uniform(items);
        for (int i = blockIdx.x; i < end && ok; i += gridDim.x) {
            const Item t = item_of<MODE>(p, i, tiles);
            const int boxes = fa::uniform(ceil_div(t.valid, kBoxRows)), row0 = fa::uniform(t.row0);
            const int wy = fa::uniform(t.expert * (MODE == GATE_UP ? 2 : 1) * p.n_out + t.n0);
            for (int kb = 0; kb < num_kb; ++kb, ++it) {
                const int s = it % kStages;
                if (it >= kStages && !__all_sync(0xffffffffu, mbar_wait(bar(&bars.empty[s]), ((it / kStages) - 1) & 1, &abort_s))) { ok = false; break; }
                if (fa::elect_one()) {
                    const uint32_t full = bar(&bars.full[s]), at = smem_addr(smem) + s * kStageBytes;
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full), "r"(kTile + boxes * kBoxRows * kK * 4) : "memory");
                    load_box(at, &map_w, full, kb * kK, wy);
                    if (MODE == GATE_UP) load_box(at + kTile / 2, &map_w, full, kb * kK, wy + p.n_out);
                    load_box(at + kTile, &map_x, full, kb * kK, row0);
                    if (boxes > 1) load_box(at + kTile + kBoxRows * kK * 4, &map_x, full, kb * kK, row0 + kBoxRows);
                }
                __syncwarp();
            }
        }
        if (!ok && lane == 0) { abort_s = 1; atomicCAS(p.error, 0, kErrorCode); }
        for (int k = max(0, it - kStages); k < it; ++k) mbar_drain(bar(&bars.full[k % kStages]), (k / kStages) & 1);
    } else if (warp == 1) {
        int it = 0, chunk = 0, done = 0;             // steps, sums and items so far
        const int last = fa::uniform(items);
        const uint32_t tm = (uint32_t)fa::uniform((int)tmem);
        auto wait = [&](uint64_t* b, uint32_t parity) {
            ok = __all_sync(0xffffffffu, mbar_wait(bar(b), parity, &abort_s));
            return ok;
        };
        auto wait_step = [&](int it, int kb, int chunk) {
            if (kb % kChunk == 0 && chunk >= 2) wait(&bars.sum_empty[chunk & 1], ((chunk >> 1) - 1) & 1);
            if (ok) wait(&bars.split_full[it & 1], (it >> 1) & 1);          // who arrives there has seen the copies land
        };
        for (int i = blockIdx.x; i < last && ok; i += gridDim.x, ++done) {
            const int valid = fa::uniform(item_of<MODE>(p, i, tiles).valid);
            const uint32_t id = instr(max(16, (valid + 15) & ~15));
            // With more than 64 activation rows the waits of a step come between the two halves of the products of the step before it, which
            // run meanwhile (the tensor cores hold some five products ahead, less than the waits take).  Few rows make short
            // products, whose buffers are better freed early, and so are those of the experts' first product, whose weights come from
            // memory.  2,048 rows by 8,192 x 3,072 weights 511 -> 479 us; experts of 105 rows, first product 3,682 (3,760 so), second 1,811 -> 1,780.
            const bool apart = MODE != GATE_UP && valid > 64;
            if (done > 0) wait(&bars.low_empty, (done - 1) & 1);
            if (ok) wait_step(it, 0, chunk);
            for (int kb = 0; kb < num_kb && ok; ++kb, ++it) {
                const int s = it % kStages, x = it & 1, b = chunk & 1;
                const bool first = kb % kChunk == 0, ends = kb % kChunk == kChunk - 1 || kb == num_kb - 1;
                const uint32_t at = smem_addr(smem) + s * kStageBytes, wh = tm + kSplit + x * 2 * kK, wl = wh + kK, to = tm + b * kN;
                const uint64_t bh = fa::desc_kmajor(at + kTile), bl = fa::desc_kmajor(at + 2 * kTile);
                auto half = [&](int k0) {
#pragma unroll
                    for (int k = k0; k < k0 + kK / 16; ++k) {    // steps of 8: 32 bytes along K, 8 columns of A
                        multiply(to, wh + 8 * k, bh + 2 * k, id, !first || k != 0);
                        multiply(tm + kLow, wl + 8 * k, bh + 2 * k, id, kb != 0 || k != 0);
                        multiply(tm + kLow, wh + 8 * k, bl + 2 * k, id, 1);
                    }
                };
                auto free = [&]() {
                    fa::umma_commit(bar(&bars.empty[s]));
                    fa::umma_commit(bar(&bars.split_empty[x]));
                    if (ends) fa::umma_commit(bar(&bars.sum_full[b]));
                };
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                chunk += ends;
                if (apart) {
                    if (fa::elect_one()) half(0);
                    __syncwarp();
                    if (kb + 1 < num_kb) wait_step(it + 1, kb + 1, chunk);
                    if (fa::elect_one()) {                       // also after a failed wait: what waits for this step ends
                        half(kK / 16);
                        free();
                    }
                    __syncwarp();
                } else {
                    if (fa::elect_one()) {
                        half(0);
                        half(kK / 16);
                        free();
                    }
                    __syncwarp();
                    if (kb + 1 < num_kb) wait_step(it + 1, kb + 1, chunk);
                }
            }
        }
        if (!ok && lane == 0) { abort_s = 1; atomicCAS(p.error, 0, kErrorCode); }
        __syncwarp();
        if (fa::elect_one()) fa::umma_commit(bar(&bars.all_done));   // what was issued ends before its memory is given back
        __syncwarp();
        mbar_drain(bar(&bars.all_done), 0);
    }
    } else if (warp < 12) {                          // steps of even and of odd number in turn
        asm volatile("setmaxnreg.dec.sync.aligned.u32 104;");
        const int x = warp >= 8, quarter = warp & 3, row = quarter * 32 + lane;
        const uint32_t to = tmem + ((uint32_t)(quarter * 32) << 16) + kSplit + x * 2 * kK;
        int it = 0;
        for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
            const bool mine = quarter * 32 < item_of<MODE>(p, i, tiles).valid;
            for (int kb = 0; kb < num_kb; ++kb, ++it) {
                if ((it & 1) != x) continue;
                const int s = it % kStages;
                if (!__all_sync(0xffffffffu, mbar_wait(bar(&bars.full[s]), (it / kStages) & 1, &abort_s))) { ok = false; break; }
                const uint32_t tile = smem_addr(smem) + s * kStageBytes;
                // every read ahead of the first write, which the compiler would not move reads across
                uint4 values[kK / 4], rows[kK / 4];
#pragma unroll
                for (int c = 0; c < kK / 4; ++c) {
                    if (mine) values[c] = lds16(tile + kTile + sw128(row, c));
                    rows[c] = lds16(tile + sw128(row, c));
                }
                if (mine)
#pragma unroll
                    for (int c = 0; c < kK / 4; ++c) {           // rounded: the tensor cores read 11 of its up to 13 bits
                        const uint32_t v4[4] = {values[c].x, values[c].y, values[c].z, values[c].w};
                        uint32_t lo[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) lo[j] = __float_as_uint(__uint_as_float(v4[j]) - __uint_as_float(v4[j] & 0xffffe000u)) + 0x1000u;
                        sts16(tile + 2 * kTile + sw128(row, c), make_uint4(lo[0], lo[1], lo[2], lo[3]));
                    }
                uint32_t hi[kK], lo[kK];
                float rest[4] = {};
#pragma unroll
                for (int c = 0; c < kK / 4; ++c) {
                    const uint32_t v4[4] = {rows[c].x, rows[c].y, rows[c].z, rows[c].w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint32_t h = (v4[j] + 0x1000u) & 0xffffe000u;
                        const float l = __uint_as_float(v4[j]) - __uint_as_float(h);
                        rest[j] += l;
                        hi[4 * c + j] = h;
                        lo[4 * c + j] = __float_as_uint(l);
                    }
                }
                if (mine) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                // only now: the products of two steps ago may still read these columns
                if (it >= 2 && !__all_sync(0xffffffffu, mbar_wait(bar(&bars.split_empty[x]), ((it >> 1) - 1) & 1, &abort_s))) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                fa::tmem_st32(to, hi);
                fa::tmem_st32(to + kK, lo);
                if (__any_sync(0xffffffffu, !isfinite((rest[0] + rest[1]) + (rest[2] + rest[3])))) {
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");         // stores to one place have no order of their own
#pragma unroll 1
                    for (int j = 0; j < kK; ++j) {               // a value without a finite nearest tf32 value: cut off, or kept as it is
                        const uint32_t v = lds4(tile + sw128(row, j / 4) + (j & 3) * 4), h = (v + 0x1000u) & 0xffffe000u;
                        const bool odd = (h & 0x7f800000u) == 0x7f800000u || (v & 0x7f800000u) == 0x7f800000u;
                        const uint32_t upper = !odd ? h : isnan(__uint_as_float(v)) ? v | 0x400000u : v & 0xffffe000u;
                        const uint32_t rest_of = isfinite(__uint_as_float(v)) ? __float_as_uint(__uint_as_float(v) - __uint_as_float(upper)) : 0u;
                        asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(to + j), "r"(upper) : "memory");
                        asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(to + kK + j), "r"(rest_of) : "memory");
                    }
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(&bars.split_full[x]));
            }
        }
        if (!ok && lane == 0) { abort_s = 1; atomicCAS(p.error, 0, kErrorCode); }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
        const int quarter = warp & 3, et = threadIdx.x - 384;
        const uint32_t from = tmem + ((uint32_t)(quarter * 32) << 16);
        const int chunks = ceil_div(num_kb, kChunk);
        int chunk = 0, done = 0, met = 0;
        auto meet = [&]() { return ok = fa::warps_meet(bar(&bars.meet), met++, &abort_s); };
        for (int i = blockIdx.x; i < items && ok; i += gridDim.x, ++done) {
            const Item t = item_of<MODE>(p, i, tiles);
            if (MODE == DOWN) {
                route_s[done & 1][et] = et < t.valid ? p.route_w[p.sorted[t.row0 + et]] : 0.f;
                if (!meet()) break;
            }
            float sum[kN];
#pragma unroll
            for (int c = 0; c < kN; ++c) sum[c] = 0.f;
            for (int k = 0; k < chunks; ++k, ++chunk) {
                const int b = chunk & 1;
                if (!__all_sync(0xffffffffu, mbar_wait(bar(&bars.sum_full[b]), (chunk >> 1) & 1, &abort_s))) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int c0 = 0; c0 < kN; c0 += 64) {
                    if (c0 >= t.valid) break;
                    uint32_t v[64];
                    fa::tmem_ld32(from + b * kN + c0, v);
                    fa::tmem_ld32(from + b * kN + c0 + 32, v + 32);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int c = 0; c < 64; ++c) sum[c0 + c] += __uint_as_float(v[c]);
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(&bars.sum_empty[b]));
            }
            if (!ok) break;
            float zeros[8] = {};                     // 0, or NaN after a sum that is not finite
#pragma unroll
            for (int c = 0; c < kN; ++c) zeros[c & 7] = fmaf(sum[c], 0.f, zeros[c & 7]);
#pragma unroll
            for (int c = 4; c > 0; c >>= 1)
#pragma unroll
                for (int j = 0; j < c; ++j) zeros[j] += zeros[j + c];
            const bool odd = __any_sync(0xffffffffu, zeros[0] != 0.f);
#pragma unroll
            for (int c0 = 0; c0 < kN; c0 += 32) {
                if (c0 >= t.valid) break;
                uint32_t v[32];
                fa::tmem_ld32(from + kLow + c0, v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (!odd) {
#pragma unroll
                    for (int c = 0; c < 32; ++c) sum[c0 + c] += __uint_as_float(v[c]);
                    continue;
                }
                uint32_t rows = 0, nans = 0;
#pragma unroll
                for (int c = 0; c < 32; ++c) {
                    if (isfinite(sum[c0 + c])) sum[c0 + c] += __uint_as_float(v[c]);
                    if (__any_sync(0xffffffffu, isinf(sum[c0 + c])) && c0 + c < t.valid) rows |= 1u << c;
                }
#pragma unroll 1
                for (; rows; rows &= rows - 1) {
                    const int c = __ffs(rows) - 1;
                    if (has_nan(p.x + (size_t)(t.row0 + c0 + c) * p.x_stride, p.k_dim)) nans |= 1u << c;
                }
#pragma unroll
                for (int c = 0; c < 32; ++c)
                    if (nans & (1u << c)) sum[c0 + c] = __int_as_float(0x7fffffff);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(&bars.low_empty));

            if (MODE == GATE_UP) {                   // lanes 0-63 hold gate rows, 64-127 the up rows of the same features
                const bool up = quarter >= 2;
                const int f = (quarter & 1) * 32 + lane, n = t.n0 + f;
                float* put = exchange + (up ? 0 : (kN / 2) * 64) + f;
                const float* get = exchange + (up ? (kN / 2) * 64 : 0) + f;
                if (!meet()) break;                  // the last item's values have been read
#pragma unroll
                for (int c = 0; c < kN / 2; ++c) put[c * 64] = up ? sum[c] : sum[kN / 2 + c];
                if (!meet()) break;
                // Eight rows at a time, every value computed and only the stores guarded: row by row behind a branch, an item's epilogue took
                // 35,000 cycles of its 145,000, and the products wait for it once both sums are full.
                const int rows = t.valid - (up ? kN / 2 : 0);        // of this thread's half
                float* o = p.out + (size_t)(t.row0 + (up ? kN / 2 : 0)) * p.n_out + n;
                auto store = [&](auto kind) {
#pragma unroll
                    for (int c0 = 0; c0 < kN / 2; c0 += 8) {
                        if (c0 >= rows) break;
                        float v[8];
#pragma unroll
                        for (int c = 0; c < 8; ++c) {
                            const float own = up ? sum[kN / 2 + c0 + c] : sum[c0 + c], other = get[(c0 + c) * 64];
                            v[c] = glu_value<float>(up ? other : own, up ? own : other, decltype(kind)::value, p.act_limit, p.act_alpha);
                        }
#pragma unroll
                        for (int c = 0; c < 8; ++c)
                            if (c0 + c < rows && n < p.n_out) o[(size_t)(c0 + c) * p.n_out] = v[c];
                    }
                };
                if (p.act_kind == SE_GLU_SILU) store(std::integral_constant<int, SE_GLU_SILU>{});
                else if (p.act_kind == SE_GLU_CLAMPED) store(std::integral_constant<int, SE_GLU_CLAMPED>{});
                else store(std::integral_constant<int, SE_GLU_GELU>{});
            } else {
                const int n = t.n0 + quarter * 32 + lane;
                float* o = p.out + (size_t)t.row0 * p.n_out + n;
#pragma unroll
                for (int c0 = 0; c0 < kN; c0 += 8) {
                    if (c0 >= t.valid) break;
                    if (MODE == DOWN)
#pragma unroll
                        for (int c = c0; c < c0 + 8; ++c) sum[c] *= route_s[done & 1][c];
                    if (c0 + 8 <= t.valid && t.n0 + kM <= p.n_out) {
#pragma unroll
                        for (int c = c0; c < c0 + 8; ++c) o[(size_t)c * p.n_out] = sum[c];
                    } else {
#pragma unroll
                        for (int c = c0; c < c0 + 8; ++c)
                            if (c < t.valid && n < p.n_out) o[(size_t)c * p.n_out] = sum[c];
                    }
                }
            }
        }
        if (!ok && lane == 0) { abort_s = 1; atomicCAS(p.error, 0, kErrorCode); }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
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
// floats [rows][cols], rows `stride` floats apart, boxes of box_rows x kK, 128-byte swizzle; what lies outside reads as 0
static int make_map(CUtensorMap* out, const float* ptr, uint64_t rows, uint64_t cols, uint64_t stride, uint32_t box_rows) {
    const EncodeTiledFn fn = encode_fn();
    if (fn == nullptr) return SE_ERR_UNSUPPORTED;
    const cuuint64_t dims[2] = {cols, rows}, strides[1] = {stride * 4};
    const cuuint32_t box[2] = {(cuuint32_t)kK, box_rows}, elem[2] = {1, 1};
    const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(ptr), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : SE_ERR_ARGUMENT;
}

template <int MODE>
static int launch(const float* w, uint64_t w_rows, const float* x, uint64_t x_stride, const Params& p, int most_tiles, int sms, cudaStream_t stream) {
    CUtensorMap mw, mx;
    int rc = make_map(&mw, w, w_rows, p.k_dim, p.k_dim, MODE == GATE_UP ? 64 : 128);
    if (rc == 0) rc = make_map(&mx, x, p.rows, p.k_dim, x_stride, kBoxRows);
    if (rc != 0) return rc;
    const size_t smem = kStages * kStageBytes + 1024 + (MODE == GATE_UP ? kExchange : 0);
    const cudaError_t e = cudaFuncSetAttribute(gemm_f32_tc_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    const long long items = (long long)most_tiles * p.blocks;
    if (items > 0x7fffffffLL) return SE_ERR_UNSUPPORTED;
    gemm_f32_tc_kernel<MODE><<<(int)(items < sms ? items : sms), kThreads, smem, stream>>>(mw, mx, p);
    return (int)cudaGetLastError();
}

static bool aligned(const void* a) { return (reinterpret_cast<uintptr_t>(a) & 15) == 0; }

}  // namespace f32tc
}  // namespace se

using namespace se::f32tc;

// 1 if the products take an inner dimension: TMA wants rows of whole 16-byte pieces
extern "C" int se_gemm_f32_tc_supported(int k_dim) { return k_dim >= 4 && k_dim % 4 == 0; }

// out [rows][n_out] = x [rows][k_dim] . w [n_out][k_dim]^T; x's rows `x_stride` floats apart
extern "C" int se_gemm_f32_dense(const float* x, long long x_stride, const float* w, float* out, int* error, int rows, int n_out, int k_dim,
                                 int sms, cudaStream_t stream) {
    if (rows <= 0 || n_out <= 0) return 0;
    if (x_stride < k_dim && rows > 1) return SE_ERR_ARGUMENT;
    if (!se_gemm_f32_tc_supported(k_dim) || x_stride % 4 || !aligned(x) || !aligned(w)) return SE_ERR_UNSUPPORTED;
    Params p = {};
    p.x = x; p.x_stride = x_stride;
    p.out = out; p.error = error; p.rows = rows; p.n_out = n_out; p.k_dim = k_dim; p.blocks = se::ceil_div(n_out, 128);
    return launch<DENSE>(w, n_out, x, rows > 1 ? x_stride : k_dim, p, se::ceil_div(rows, kN), sms, stream);
}

// The experts' products; rows in expert order, the tile list built with 128 rows per tile.
//   mode 0: a = x's rows in that order; w = w13 [experts][2 n_out][k_dim]; out = the gated activation
//   mode 1: a = the activation;         w = w2 [experts][n_out][k_dim];    out = the product times the routing weight
extern "C" int se_gemm_f32_grouped(int mode, const float* a, const float* w, const int* sorted, const int* offsets,
                                   const int* tile_expert, const int* tile_row0, const int* num_tiles, const float* route_w, float* out,
                                   int* error, int assignments, int experts, int max_tiles, int n_out, int k_dim, int act_kind,
                                   float act_limit, float act_alpha, int sms, cudaStream_t stream) {
    if (assignments <= 0 || max_tiles <= 0) return 0;
    if (act_kind < SE_GLU_SILU || act_kind > SE_GLU_GELU || (mode != 0 && mode != 1)) return SE_ERR_ARGUMENT;
    if (!se_gemm_f32_tc_supported(k_dim) || !aligned(a) || !aligned(w)) return SE_ERR_UNSUPPORTED;
    const Params p{sorted, offsets, tile_expert, tile_row0, num_tiles, route_w, a, k_dim, out, error, assignments, n_out, k_dim,
                   se::ceil_div(n_out, mode == 0 ? 64 : 128), act_kind, act_limit, act_alpha};
    if (mode == 0) return launch<GATE_UP>(w, (uint64_t)experts * 2 * n_out, a, k_dim, p, max_tiles, sms, stream);
    return launch<DOWN>(w, (uint64_t)experts * n_out, a, k_dim, p, max_tiles, sms, stream);
}
