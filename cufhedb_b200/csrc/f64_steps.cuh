// Steps of the FP64 lvl01 bootstrap that its kernels share (pbs01_f64.cu,
// pbs01_wide.cu), the same operations in the same order per value.
#pragma once
#include "pbs_common.cuh"

namespace cfdb {

// digit d of (X^a - 1) * poly at coefficients m and m+512, twisted:
// v[m2] = (dig_d(m) + i dig_d(m+512)) * w^m,  m = lane + 32 m2.  The signed
// digit is the sign-extended field d of (t + offset + round) ^ DEC1_XOR.
__device__ __forceinline__ void load_digit_poly1(double2 v[16], const uint32_t *poly, uint32_t abar, int d, int lane,
                                        const Fft512Tables &T)
{
#pragma unroll
    for (int m2 = 0; m2 < 16; ++m2) {
        const int m = lane + 32 * m2;
        const uint32_t x0 = ((rot_coef<N1>(poly, m, abar) - poly[m]) + DEC1_OFFSET + DEC1_ROUND) ^ DEC1_XOR;
        const uint32_t x1 = ((rot_coef<N1>(poly, m + 512, abar) - poly[m + 512]) + DEC1_OFFSET + DEC1_ROUND) ^ DEC1_XOR;
        const int d0 = digit_field1(x0, d), d1 = digit_field1(x1, d);
        v[m2] = cmul(make_double2((double)d0, (double)d1), T.twist[m2 * 32 + lane]);
    }
}

// poly[m] += a_m, poly[m+512] += a_{m+512} from v[m2] = 512 z_m
__device__ __forceinline__ void add_inverse_poly1(uint32_t *poly, const double2 v[16], int lane,
                                                  const Fft512Tables &T)
{
#pragma unroll
    for (int m2 = 0; m2 < 16; ++m2) {
        const int m = lane + 32 * m2;
        double2 y = cmulc(v[m2], T.twist[m2 * 32 + lane]);
        poly[m] += f64_to_torus32(y.x * (1.0 / 512.0));
        poly[m + 512] += f64_to_torus32(y.y * (1.0 / 512.0));
    }
}

}  // namespace cfdb
