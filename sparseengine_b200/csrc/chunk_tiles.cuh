// Linear recurrences over prompt portions by chunks of 128 tokens on tcgen05, side by side: what the chunks' kernels share.
//
// The walk (chunk_walk.cuh) takes a head's chunks one after another, outputs and all.  Only the state has to go that way, and of it
// only e^(B_n) S + (what the chunk adds), which needs no product with the state.  So here one kernel forms what chunks add
// (sum_s e^(B_n - B_s) k_s u_s^T, rows of the state = the M side), the states at the chunks' starts follow by multiply-adds, and another kernel
// makes the outputs e^(B_t) q_t . S_0 + sum_s P[t][s] u_s of every chunk by itself (tokens = the M side).
//
// Everything is 32-bit and multiplied as such: a value is cut into three bfloat16 terms, which together are the value (`cut`), and of the nine products of terms the six down
// to 2^-16 are summed, the smallest first, in 32-bit tensor memory; what is left out is below 2^-22 of a product, 2^-25.5 on average (root of the mean square), of
// either sign.  Values that stay 16-bit (the retention's v) are a term themselves.  bfloat16 has twice tf32's rate and half its steps into the accumulator, and an
// operand takes 96 KB for 128 x 128 values instead of 128.
//
// Tensor memory cuts off towards zero what does not fit when a step is added, so long sums come out too small.  Hence a product has two parts in columns of their own, which
// are added in registers, and first terms have 7 bits, not 8: fewer of their products reach below the sum's last bit.  Errors from 64 bits over the result's norm, 1e-7,
// 128 / 700 / 3,000 tokens, one part and terms cut off at 8 bits; now; the walk:
//   retention, rotated    outputs 2.4 / 2.7 / 2.7; 1.2 / 1.4 / 1.4; 1.6 / 1.7 / 2.3    states 1.3 / 1.4 / 1.5; 0.9 / 1.0 / 1.2; 1.0 / 1.3 / 2.3
//   state space           outputs 1.8 / 1.8 / 1.7; 0.7 / 0.8 / 0.8; 1.1 / 0.9 / 1.0    states 1.3 / 1.3 / 1.1; 1.1 / 0.9 / 0.7; 1.4 / 1.1 / 1.1
// All values of one sign, 700 tokens: retention 2.9; 1.2; 0.8, its state 1.6; 0.9; 0.8 (128 tokens 1.6; 0.8; 0.5), state space 3.0; 1.1; 1.1, its state 1.3; 0.8; 0.8.  (8 bits to the nearest, products of
// first terms in columns of their own: rotated 2.2, state space 1.3, of one sign 2.2 and 2.1.)  Time: the retention's outputs 224 us before, 214 now, the state space's 65 and 67.
//
// What is not finite leaves its outputs not finite, and those of earlier tokens too (their weights for it are 0): a tile with such an output is done
// again token by token.
#pragma once
#include "chunk_walk.cuh"
#include "fa_util.cuh"

namespace se {
namespace tiles {

using walk::chunk_of;
using walk::ld4;

constexpr int kT = 128, kD = 128, kThreads = 512;
constexpr int kHalf = 128 * 128;                     // bytes of [128 rows][64 bfloat16], a swizzled 128 bytes each
constexpr int kTerm = 2 * kHalf;                     // a term of a 128 x 128 operand
constexpr int kErrorCode = 19;

// x = the nearest value of 7 bits + the bfloat16 nearest to what is left + the rest (7 bits at most); of a pair, x in the lower half.  What is not finite, or rounds to
// infinity, leaves NaN in the second term or the last one.
__device__ __forceinline__ void cut(float x, float y, uint32_t (&t)[3]) {
    const uint32_t a = (__float_as_uint(x) + 0x10000u) & 0xfffe0000u, b = (__float_as_uint(y) + 0x10000u) & 0xfffe0000u;
    t[0] = __byte_perm(a, b, 0x7632);
    x -= __uint_as_float(a);
    y -= __uint_as_float(b);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(t[1]) : "f"(y), "f"(x));
    x -= __uint_as_float(t[1] << 16);
    y -= __uint_as_float(t[1] & 0xffff0000u);
    t[2] = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
}

// kind::f16 of bfloat16 operands, 32-bit sums, M = 128
__device__ __forceinline__ uint32_t instr(int n, bool a_mn, bool b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
// An operand in shared memory: terms `term` bytes apart.  K-major: halves of 64 along K `half` bytes apart, rows of 128 bytes; MN-major: rows along K, groups of 64
// along M or N `half` bytes apart.  The descriptor of step k of 16.
template <bool MN>
__device__ __forceinline__ uint64_t step_desc(uint32_t at, uint32_t half, int k) {
    return MN ? fa::desc_mnmajor(at, half) + (uint64_t)(128 * k) : fa::desc_kmajor(at + (k >> 2) * half) + (uint64_t)(2 * (k & 3));
}
// A . B over K = 128 in two parts, each in columns of its own: the products of later terms, the smallest first, then of first terms over the first half of K; of first
// terms over the other half.  One lane of a warp-uniform branch.
template <bool A_MN, bool B_MN, int B_TERMS>
__device__ __forceinline__ void product_first(uint32_t d, uint32_t a, uint32_t a_half, uint32_t a_term, uint32_t b, uint32_t b_half, uint32_t b_term, uint32_t id) {
    uint32_t started = 0;
#pragma unroll
    for (int sum = 2; sum >= 0; --sum)
#pragma unroll
        for (int j = 0; j <= sum && j < B_TERMS; ++j)
#pragma unroll
            for (int k = 0; k < (sum ? 8 : 4); ++k) {
                fa::umma(d, step_desc<A_MN>(a + (sum - j) * a_term, a_half, k), step_desc<B_MN>(b + j * b_term, b_half, k), id, started);
                started = 1;
            }
}
template <bool A_MN, bool B_MN>
__device__ __forceinline__ void product_second(uint32_t d, uint32_t a, uint32_t a_half, uint32_t b, uint32_t b_half, uint32_t id) {
#pragma unroll
    for (int k = 4; k < 8; ++k) fa::umma(d, step_desc<A_MN>(a, a_half, k), step_desc<B_MN>(b, b_half, k), id, k > 4);
}
template <bool A_MN, bool B_MN, int B_TERMS>
__device__ __forceinline__ void product(uint32_t first, uint32_t second, uint32_t a, uint32_t a_half, uint32_t a_term, uint32_t b, uint32_t b_half, uint32_t b_term, uint32_t id) {
    product_first<A_MN, B_MN, B_TERMS>(first, a, a_half, a_term, b, b_half, b_term, id);
    product_second<A_MN, B_MN>(second, a, a_half, b, b_half, id);
}
// The same with A in tensor memory, terms of 64 columns
template <bool B_MN, int B_TERMS>
__device__ __forceinline__ void product_ts(uint32_t first, uint32_t second, uint32_t a, uint32_t b, uint32_t b_half, uint32_t b_term, uint32_t id) {
    uint32_t started = 0;
#pragma unroll
    for (int sum = 2; sum >= 0; --sum)
#pragma unroll
        for (int j = 0; j <= sum && j < B_TERMS; ++j)
#pragma unroll
            for (int k = 0; k < (sum ? 8 : 4); ++k) {
                fa::umma_ts(first, a + (sum - j) * 64 + 8 * k, step_desc<B_MN>(b + j * b_term, b_half, k), id, started);
                started = 1;
            }
#pragma unroll
    for (int k = 4; k < 8; ++k) fa::umma_ts(second, a + 8 * k, step_desc<B_MN>(b, b_half, k), id, k > 4);
}

__device__ __forceinline__ void st4(uint32_t addr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
__device__ __forceinline__ void st8(uint32_t addr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void ld8(uint32_t addr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ld16(uint32_t addr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(addr) : "memory");
}
// 16 columns of the sum of a product's two parts
__device__ __forceinline__ void ld_sum16(uint32_t first, uint32_t second, float* v) {
    uint32_t a[16], b[16];
    ld16(first, a);
    ld16(second, b);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int x = 0; x < 16; ++x) v[x] = __uint_as_float(a[x]) + __uint_as_float(b[x]);
}
__device__ __forceinline__ void wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void sts8(uint32_t at, uint32_t x, uint32_t y) {
    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(at), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool fill) {      // 16 bytes, or zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(fill ? 16 : 0) : "memory");
}

// Four neighbours along a row in three terms, to an operand at `at` (a row is 64 bfloat16, quad = the four's place among its sixteen)
__device__ __forceinline__ void put4(uint32_t at, uint32_t term, int row, int quad, float4 v) {
    uint32_t a[3], b[3];
    cut(v.x, v.y, a);
    cut(v.z, v.w, b);
    at += fa::sw128(row, quad >> 1) + (quad & 1) * 8;
#pragma unroll
    for (int i = 0; i < 3; ++i) sts8(at + i * term, a[i], b[i]);
}

// Tensor memory, one barrier for the products of a block (each committed and waited for in turn) and the end of both.  abort_flag: a wait has run out,
// the others need not run to their limit.
struct Shared {
    uint64_t done, last;
    uint32_t tmem;
    volatile int abort_flag;
};
__device__ __forceinline__ uint32_t begin(Shared& s) {
    if (threadIdx.x == 0) {
        fa::mbar_init(smem_u32(&s.done), 1);
        fa::mbar_init(smem_u32(&s.last), 2);
        s.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 32) {
        __syncwarp();                                // its first lane comes from the branch above, the instruction is the whole warp's
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&s.tmem)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    return s.tmem;
}
__device__ __forceinline__ void end(Shared& s) {
    const uint32_t tmem = s.tmem;
    fence_before();
    __syncthreads();
    if (threadIdx.x < 64) {                          // what the first two warps issued ends before its memory is given back
        if (fa::elect_one()) fa::umma_commit(smem_u32(&s.last));
        __syncwarp();
    }
    if (threadIdx.x < 32) {
        fence_after();
        fa::mbar_drain(smem_u32(&s.last), 0);
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
}
// Until `bar` is in phase `n` (from 0); the same answer in every lane of a warp, whose lanes are together again afterwards: what reads tensor memory next
// is the whole warp's instruction.
__device__ __forceinline__ bool warp_wait(Shared& s, uint64_t& bar, uint32_t n) {
    const bool ok = __all_sync(0xffffffffu, fa::mbar_wait(smem_u32(&bar), n & 1, &s.abort_flag));
    if (!ok) s.abort_flag = 1;
    return ok;
}
// Until the products committed `n`-th (from 0) are there; the same answer in every thread.  A wait that runs out is reported.
// `so_far`: false in a thread whose earlier wait by itself ran out.
__device__ __forceinline__ bool products_done(Shared& s, uint32_t n, int* error, bool so_far = true) {
    const bool ok = warp_wait(s, s.done, n) && so_far;
    if (__syncthreads_and(ok)) {
        fence_after();
        return true;
    }
    if (threadIdx.x == 0) atomicCAS(error, 0, kErrorCode);
    return false;
}

}  // namespace tiles
}  // namespace se
