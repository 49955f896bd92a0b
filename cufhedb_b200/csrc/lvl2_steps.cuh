// Steps of the lvl2 ring's kernels (lvl2_f64.cu, pbs02_f64.cu): decomposition
// words and digits, the inverse transform into the accumulator.
#pragma once
#include "fft1024_f64.cuh"
#include "lvl2.cuh"

namespace cfdb {

// digit d (0 = most significant) of a word x as a double: the 9-bit field
// u = digit + 256, set as the low mantissa bits of 2^52, minus 2^52 + 256 (exact).
// An int -> double conversion would wait for the far slower conversion unit.
__device__ __forceinline__ double digit2(uint64_t x, int d)
{
    const uint32_t u = (uint32_t)(x >> (64 - BGBIT2 * (d + 1))) & ((1u << BGBIT2) - 1);
    return __hiloint2double(0x43300000, (int)u) - 4503599627370752.0;
}

// digit-extraction words of (X^a - 1) * poly (or of poly when ROT is false)
// at m and m + 1024: x = c + offset + round, whose fields are the digits
template <bool ROT>
__device__ __forceinline__ void digit_word_pair2(uint64_t &x0, uint64_t &x1, const uint64_t *poly, uint32_t abar,
                                                 int m)
{
    uint64_t c0 = poly[m], c1 = poly[m + 1024];
    if (ROT) {
        c0 = rot_coef<N2>(poly, m, abar) - c0;
        c1 = rot_coef<N2>(poly, m + 1024, abar) - c1;
    }
    x0 = c0 + DEC2_OFFSET + DEC2_ROUND;
    x1 = c1 + DEC2_OFFSET + DEC2_ROUND;
}

// the words of thread t, m = t + 128 j: all four digits of a polynomial from
// one load of the accumulator
template <bool ROT>
__device__ __forceinline__ void digit_words2(uint64_t x[16], const uint64_t *poly, uint32_t abar, int t)
{
#pragma unroll
    for (int j = 0; j < 8; ++j) digit_word_pair2<ROT>(x[2 * j], x[2 * j + 1], poly, abar, t + T2 * j);
}

// digit d, twisted by W_32^j (fft8x folds the rest of the twist):
// v[j] = (dig_d(m) + i dig_d(m+1024)) * W_32^j, m = t + 128 j
__device__ __forceinline__ void digits2(double2 v[8], const uint64_t x[16], int d)
{
#pragma unroll
    for (int j = 0; j < 8; ++j)
        v[j] = cx_w32<1>(make_double2(digit2(x[2 * j], d), digit2(x[2 * j + 1], d)), j);
}

// poly[m] += round-toward-zero of the inverse transform, m = t + 128 j
__device__ __forceinline__ void add_inverse2(uint64_t *poly, const double2 v[8], int t)
{
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int m = t + T2 * j;
        const double2 y = cx_w32<-1>(v[j], j);
        poly[m] += f64_to_torus64(y.x * (1.0 / 1024.0));
        poly[m + 1024] += f64_to_torus64(y.y * (1.0 / 1024.0));
    }
}

}  // namespace cfdb
