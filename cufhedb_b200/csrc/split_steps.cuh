// Steps of the split-precision lvl01 bootstrap that its kernels share
// (pbs01_ct.cu, pbs01_split_tc.cu).
//
// Precision plan (the 32-bit torus needs products exact to well below the
// bootstrapping noise, which FP32 alone cannot give):
//   * each integer key polynomial b is split into limbs
//       hi = round(b / 2^24) in [-128, 128],  lo = b - hi * 2^24 in [-2^23, 2^23);
//     both are transformed in FP64 on the device at key-load time and stored
//     as FP32 frequency values;
//   * per CMux the 6 digit polynomials (|d| <= 32) are transformed in FP32 and
//     multiplied into four FP32 accumulators (hi/lo x 2 output polynomials);
//   * the hi accumulators' inverse transforms are rounded to integers, which is
//     exact: sum_r d_r * hi_r has rms magnitude ~2^16.7, so FP32 round-off
//     (~2^-21.5 relative) leaves an error ~0.04, a 12-sigma margin below 1/2;
//     then hi * 2^24 is taken modulo 2^32;
//   * the lo accumulators' inverse transforms (rms ~2^32.7) are rounded to
//     64-bit integers; their FP32 round-off (~2^11) is ~2^-6 of the per-CMux
//     bootstrapping noise standard deviation (~2^17.8), i.e. it adds about
//     0.03 % to the noise variance.
#pragma once
#include "fft_f32.cuh"
#include "pbs_common.cuh"

namespace cfdb {

// the decomposition words of (X^a - 1) * poly, once per polynomial:
// w[2 m2 + h] = (((X^a - 1) poly)[m + 512 h] + offset + round) ^ DEC1_XOR,
// m = lane + 32 m2; each of the l = 3 digits is then a field of these words
__device__ __forceinline__ void digit_words1(uint32_t w[32], const uint32_t *poly, uint32_t abar, int lane)
{
#pragma unroll
    for (int m2 = 0; m2 < 16; ++m2) {
        const int m = lane + 32 * m2;
        w[2 * m2] = ((rot_coef<N1>(poly, m, abar) - poly[m]) + DEC1_OFFSET + DEC1_ROUND) ^ DEC1_XOR;
        w[2 * m2 + 1] = ((rot_coef<N1>(poly, m + 512, abar) - poly[m + 512]) + DEC1_OFFSET + DEC1_ROUND) ^ DEC1_XOR;
    }
}

// round(h) * 2^24 mod 2^32 without a conversion instruction: adding
// 1.5 * 2^23 leaves round-to-nearest-even of h in the low mantissa bits
// (|h| < 2^22, ~40 standard deviations of the hi products), and the term
// needs only their low 8 bits.  Same bits as __float2int_rn(h) << 24, on the
// FMA and ALU pipes instead of the conversion unit (measured: 1,024 PBS
// 9.73 -> 9.41 ms, 1,184 in the 8-per-CTA shape 10.95 -> 10.5 ms; building
// the digits from their bits the same way measured slower in both shapes, so
// they keep the int -> float conversion)
__device__ __forceinline__ uint32_t hi_term(float h)
{
    return __float_as_uint(h + 12582912.0f) << 24;
}

// poly[m] += round(hi_m) * 2^24 + round(lo_m) (mod 2^32), one read-modify-write
// of the accumulator per polynomial.  f holds the hi and lo limbs of one
// output as pairs, inverse-transformed together.  The hi limb's products
// round exactly; the lo limb's FP32 error stays far below the bootstrapping
// noise.
__device__ __forceinline__ void add_inverse_split(uint32_t *poly, CP f[16], unsigned long long *xp, int lane,
                                                  const Fft512TablesFold &T)
{
    pfft512_inv(f, xp, T, lane);
#pragma unroll
    for (int m2 = 0; m2 < 16; ++m2) {
        const int m = lane + 32 * m2;
        const CP y = untwist_m2(f[m2], m2);
        const float2 re = unpk2(y.re), im = unpk2(y.im);   // (hi, lo) of coefficients m and m + 512
        poly[m] += hi_term(re.x) + (uint32_t)__float2ll_rn(re.y);
        poly[m + 512] += hi_term(im.x) + (uint32_t)__float2ll_rn(im.y);
    }
}

// f += v * k for both limbs of one output: k = (hi.re, lo.re, hi.im, lo.im),
// vr = (v.re, v.re), vi = (v.im, v.im), nvi = (-v.im, -v.im)
__device__ __forceinline__ void pmac(CP &f, unsigned long long vr, unsigned long long vi, unsigned long long nvi,
                                     float4 k)
{
    const unsigned long long kr = pk2(k.x, k.y), ki = pk2(k.z, k.w);
    f.re = f2(nvi, ki, f2(vr, kr, f.re));
    f.im = f2(vi, kr, f2(vr, ki, f.im));
}
__device__ __forceinline__ CP pmul_first(unsigned long long vr, unsigned long long vi, unsigned long long nvi, float4 k)
{
    const unsigned long long kr = pk2(k.x, k.y), ki = pk2(k.z, k.w);
    return CP{f2(nvi, ki, m2(vr, kr)), f2(vi, kr, m2(vr, ki))};
}

}  // namespace cfdb
