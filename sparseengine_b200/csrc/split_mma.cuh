// Products of 32-bit values with mma.sync in tf32 terms: an operand is the sum of two tf32 values (11 bits of mantissa each, hi the
// nearest one, lo what is left, of which they read 11 of its up to 12 bits), and hi hi + lo hi + hi lo leaves out lo lo, up to 2^-22 of a product.  The
// tensor cores cut off what does
// not fit when they add to an accumulator instead of rounding it, so that long sums there come out too small: the large products are
// summed by m16n8k8 steps that start from zero and are then added in 32-bit; the small ones have an accumulator of their own,
// where what is cut off does not count.  Measured against 64 bits, sums of 32 / 128 products of normal values, error over the result's
// norm: 1.0e-7 / 1.2e-7; one chain of multiply-adds 1.0e-7 / 2.0e-7, four chains 0.7e-7 / 1.1e-7, one accumulator for all three
// terms 2.5e-7 / 9.1e-7.  The walks that use them (chunk_walk.cuh; 70, 700 and 3,000 tokens), with chains of multiply-adds / now, 1e-7: outputs of
// the state space 1.00, 1.06, 1.29 / 0.95, 0.94, 1.01, its state 1.18, 1.22, 0.90 / 1.42, 1.43, 1.15; retention 2.09, 1.98, 2.56 / 1.71, 1.80, 2.33,
// state 1.11, 1.54, 2.57 / 1.15, 1.40, 2.39; delta rule per head 2.14, 2.22, 2.43 / 1.87, 1.93, 2.14, state 1.83, 2.07, 2.39 / 1.89, 2.14, 2.31; per
// channel 1.55, 1.56, 2.11 / 1.67, 1.69, 2.17, state 2.24, 2.25, 3.19 / 2.30, 2.31, 3.24.  Whole mixers in float32, whose projections count for more: outputs
// 1.5e-6 to 4.5e-6 / 0.4e-6 to 4.1e-6, states 0.8e-6 to 3.7e-6 / 0.2e-6 to 3.6e-6, none larger than before.
//
// What it buys is shared-memory reads, not arithmetic: mma.sync takes 8.4 cycles of a quarter SM for 1,024 products and, on this
// part, multiply-adds and integer instructions wait for it (0.65 to 1 cycle more for each), so three terms cost 25 cycles where
// multiply-adds cost 32; but a warp reads an operand once per tile of 16 x 8 instead of once per thread's tile.
#pragma once
#include "common.cuh"

namespace se {
namespace split {

__device__ __forceinline__ void halves(float x, uint32_t& hi, uint32_t& lo) {
    hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
    lo = __float_as_uint(x - __uint_as_float(hi));
}
__device__ __forceinline__ void mma_add(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void mma_start(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
}

// acc[i][n] += the products of tile row i and tile column n over `steps` steps of eight.  a(i, step, v) gives this lane's four
// values of tile row i: (row lane / 4, first k), (row + 8, first k), (row, second k), (row + 8, second k); b(n, step, v) its two of
// tile column n: (first k, column lane / 4), (second k, the same).  Which two of the step's eight k are a lane's is the callers' choice:
// 2 (lane % 4) and the one after it, so that rows along k are read two at a time.  acc[i][n] holds (row lane / 4, columns 2 (lane % 4)
// and the one after it), then the same of row + 8.  EXACT: b's values are tf32 values themselves (16-bit inputs): two terms.
template <int MT, int NT, int UNROLL, bool EXACT = false, typename A, typename B>
__device__ __forceinline__ void products(float (&acc)[MT][NT][4], int steps, A a, B b) {
    float low[MT][NT][4] = {};
#pragma unroll UNROLL
    for (int s = 0; s < steps; ++s) {
        uint32_t ah[MT][4], al[MT][4], bh[NT][2], bl[NT][2];
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            float v[4];
            a(i, s, v);
#pragma unroll
            for (int j = 0; j < 4; ++j) halves(v[j], ah[i][j], al[i][j]);
        }
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            float v[2];
            b(n, s, v);
            if (EXACT) {
                bh[n][0] = __float_as_uint(v[0]);
                bh[n][1] = __float_as_uint(v[1]);
            } else {
                halves(v[0], bh[n][0], bl[n][0]);
                halves(v[1], bh[n][1], bl[n][1]);
            }
        }
        float big[MT][NT][4];
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int n = 0; n < NT; ++n) mma_start(big[i][n], ah[i], bh[n]);
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int n = 0; n < NT; ++n) mma_add(low[i][n], al[i], bh[n]);
        if (!EXACT)
#pragma unroll
            for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int n = 0; n < NT; ++n) mma_add(low[i][n], ah[i], bl[n]);
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][n][j] += big[i][n][j];
    }
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][n][j] += low[i][n][j];
}

// Whether a lane of the warp holds a value that is not finite.  The terms of an infinity are not its parts (inf - inf), and a value
// near the largest one rounds up to infinity: either leaves its sums not finite, and the caller then takes them the plain way.
template <int MT, int NT>
__device__ __forceinline__ bool odd(const float (&acc)[MT][NT][4]) {
    float z = 0.f;
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int j = 0; j < 4; ++j) z = fmaf(acc[i][n][j], 0.f, z);
    return __any_sync(0xffffffffu, z != 0.f);
}

}  // namespace split
}  // namespace se
