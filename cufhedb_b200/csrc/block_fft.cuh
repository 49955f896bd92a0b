// The lvl1 transforms of a block of warps that works on one ciphertext or product
// (pbs01_ct.cu, extprod.cu): one warp per TRGSW row or output, 16 of the 512 points
// per lane, as in fft_f64.cuh and fft_f32.cuh, but the radix-2 step across lanes at
// the end of the forward and at the start of the inverse transform is left to
// the products between them, where one thread holds both its inputs, and the
// per-lane twiddles come from tensor memory.  Every value goes through the same
// operations with the same roundings in the same order as in those transforms.
#pragma once
#include <cstddef>

#include "fft_f64.cuh"
#include "pbs_common.cuh"
#include "split_steps.cuh"
#include "tc_stage1.cuh"
#include "tmem_exchange.cuh"

namespace cfdb {

// One polynomial's share of the paired inverse (fft_f32.cuh pfft512_inv), in
// scalar form with the paired form's roundings.  The compiler fuses a packed
// product into the packed addition or subtraction that takes it (the first
// operand's product where both are products), so the fused forms are written
// out here; cufhedb_selftest_split_transforms compares both forms bit for bit.
// a * conj(c + i s)
__device__ __forceinline__ float2 fmulc_t(float2 a, float c, float s)
{
    return make_float2(fmaf(a.x, c, __fmul_rn(a.y, s)), fmaf(a.y, c, -__fmul_rn(a.x, s)));
}
// b + k a by component
__device__ __forceinline__ float2 faxpy(float k, float2 a, float2 b)
{
    return make_float2(fmaf(a.x, k, b.x), fmaf(a.y, k, b.y));
}
// the last four-point DFT of pdft16<-1>, from its sums and differences
__device__ __forceinline__ void finv4(float2 *v, float2 s02, float2 d02, float2 s13, float2 d13)
{
    const float2 t = make_float2(d13.y, -d13.x);
    v[0] = fadd2(s02, s13);
    v[2] = fsub2(s02, s13);
    v[1] = fadd2(d02, t);
    v[3] = fsub2(d02, t);
}
// pdft16<-1> of one polynomial
__device__ __forceinline__ void fdft16_inv(float2 v[16])
{
    constexpr float R2 = 0.70710678118654752440f;
#pragma unroll
    for (int n1 = 0; n1 < 4; ++n1) fdft4<-1>(v[n1], v[n1 + 4], v[n1 + 8], v[n1 + 12]);
    // the twiddles (+-1 - i) / sqrt 2 are left unscaled here
    auto e2 = [](float2 a) { return make_float2(__fadd_rn(a.x, a.y), __fsub_rn(a.y, a.x)); };
    auto e6 = [](float2 a) { return make_float2(__fsub_rn(a.y, a.x), -__fadd_rn(a.x, a.y)); };
    v[5] = fw16<-1, 1>(v[5]);
    v[7] = fw16<-1, 3>(v[7]);
    v[10] = fw16<-1, 4>(v[10]);
    v[13] = fw16<-1, 3>(v[13]);
    v[15] = fw16<-1, 9>(v[15]);
    const float2 u6 = e2(v[6]), u9 = e2(v[9]), u11 = e6(v[11]), u14 = e6(v[14]);
    finv4(v, fadd2(v[0], v[2]), fsub2(v[0], v[2]), fadd2(v[1], v[3]), fsub2(v[1], v[3]));
    finv4(v + 4, faxpy(R2, u6, v[4]), faxpy(-R2, u6, v[4]), fadd2(v[5], v[7]), fsub2(v[5], v[7]));
    const float2 p11 = make_float2(__fmul_rn(u11.x, R2), __fmul_rn(u11.y, R2));
    finv4(v + 8, fadd2(v[8], v[10]), fsub2(v[8], v[10]), faxpy(R2, u9, p11),
          faxpy(R2, u9, make_float2(-p11.x, -p11.y)));
    finv4(v + 12, faxpy(R2, u14, v[12]), faxpy(-R2, u14, v[12]), fadd2(v[13], v[15]), fsub2(v[13], v[15]));
    float2 t[16];
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2)
#pragma unroll
        for (int k1 = 0; k1 < 4; ++k1) t[k2 + 4 * k1] = v[4 * k2 + k1];
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = t[i];
}


// the warps of both limbs of output o meet
__device__ __forceinline__ void limbs_sync(int o) { asm volatile("bar.sync %0, 64;" ::"r"(1 + o) : "memory"); }

// Each path: its value type, its tables' tensor-memory columns, and the steps
// on the 16 values of a lane.  A row's buffer holds in turn its packed digits,
// the transpose, the spectrum [j][lane] before the last radix-2 step, and (rows
// < INV) the sums [j][lane] after the inverse's first.
struct SplitPath {
    using V = float2;
    using Full = Fft512TablesFold;
    struct Tab {
        float4 w32p[16];
    };
    static constexpr int TAB_WORD4 = offsetof(Full, w32p) / 16;
    static constexpr int ROW = 18;          // transpose rows of 16 values: 16-byte multiples, no bank conflicts
    static constexpr int BUF = 32 * ROW;
    static constexpr int INV = 4;           // inverse transforms: output x limb
    static constexpr uint32_t COLS = 64;    // tw512w, then (c, s) of tw512u
    struct Sum {
        CP z;
    };
    __device__ __forceinline__ static const float4 *tables(const void *t)
    {
        return reinterpret_cast<const float4 *>(&reinterpret_cast<const Fft512TablesF *>(t)->fold);
    }
    __device__ __forceinline__ static void stage_tables(uint32_t tm, const Full &T, int lane)
    {
        uint32_t x[32];
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            x[2 * q] = __float_as_uint(T.tw512w[q * 32 + lane].x);
            x[2 * q + 1] = __float_as_uint(T.tw512w[q * 32 + lane].y);
        }
        tmem_st32_nowait(tm, x);
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            x[2 * q] = __float_as_uint(T.tw512u[q * 32 + lane].x);
            x[2 * q + 1] = __float_as_uint(T.tw512u[q * 32 + lane].z);
        }
        tmem_st32_nowait(tm + 32, x);
        tmem_wait_st();
    }
    // entries 8 c .. 8 c + 7 of this lane at column tm
    __device__ __forceinline__ static void twiddles(uint32_t x[16], uint32_t tm, int c)
    {
        tmem_ld16_nowait(tm + 16 * c, x);
        tmem_wait_ld();
        tmem_landed<16>(x);
    }
    __device__ __forceinline__ static V entry(const uint32_t x[16], int k)
    {
        return make_float2(__uint_as_float(x[2 * k]), __uint_as_float(x[2 * k + 1]));
    }
    // packed digits: 2^23 + u has u in its low mantissa bits; the subtraction of
    // 2^23 + 32 is exact (the int -> float conversion has an eighth of its rate)
    __device__ __forceinline__ static V unpack(uint32_t u)
    {
        return fsub2(make_float2(__uint_as_float(0x4B000000u | (u & 0xFFFFu)), __uint_as_float(0x4B000000u | (u >> 16))),
                     make_float2(8388640.0f, 8388640.0f));
    }
    __device__ __forceinline__ static void forward(V v[16], V *xp, int lane, uint32_t tm)
    {
        const uint32_t *dig = reinterpret_cast<const uint32_t *>(xp) + lane;
#pragma unroll
        for (int m2 = 0; m2 < 16; ++m2) {
            v[m2] = cw64(unpack(dig[32 * m2]), m2);
        }
        fdft16<1>(v);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            uint32_t x[16];
            twiddles(x, tm, c);
#pragma unroll
            for (int k = 0; k < 8; ++k) v[8 * c + k] = fcmul(v[8 * c + k], entry(x, k));
        }
        forward_rest(v, xp, lane);
    }
    // the transpose and the second 16-point DFT: v[j] = X_h[j]
    __device__ __forceinline__ static void forward_rest(V v[16], V *xp, int lane)
    {
        __syncwarp();
        float4 *row = reinterpret_cast<float4 *>(xp + ROW * lane);
#pragma unroll
        for (int k = 0; k < 8; ++k) row[k] = make_float4(v[2 * k].x, v[2 * k].y, v[2 * k + 1].x, v[2 * k + 1].y);
        __syncwarp();
        const int h = lane >> 4, q2 = lane & 15;
#pragma unroll
        for (int m1p = 0; m1p < 16; ++m1p) v[m1p] = xp[ROW * (2 * m1p + h) + q2];
        fdft16<1>(v);
    }
    // W32^j, j = jl + 8 hh, as the one-warp kernels' forward and inverse use it
    __device__ __forceinline__ static V w32_fwd(const Tab &T, int jl, int hh)
    {
        const float4 w = T.w32p[jl];
        return hh ? make_float2(-w.z, w.x) : make_float2(w.x, w.z);
    }
    __device__ __forceinline__ static V w32_inv(const Tab &T, int jl, int hh)
    {
        const float4 w = T.w32p[jl + 8 * hh];
        return make_float2(w.x, w.z);
    }
    __device__ __forceinline__ static V mul(V a, V b) { return fcmul(a, b); }
    __device__ __forceinline__ static V add(V a, V b) { return fadd2(a, b); }
    __device__ __forceinline__ static V sub(V a, V b) { return fsub2(a, b); }
    __device__ __forceinline__ static void mac(Sum &f, bool first, V v, float4 k)
    {
        if (first) f.z = pmul_first(pk2(v.x, v.x), pk2(v.y, v.y), pk2(-v.y, -v.y), k);
        else pmac(f.z, pk2(v.x, v.x), pk2(v.y, v.y), pk2(-v.y, -v.y), k);
    }
    // rows 2 o and 2 o + 1 take the hi and the lo limb of output o
    __device__ __forceinline__ static void put(V *buf, int o, int at, const Sum &f0, const Sum &f1, V w)
    {
        const float2 r0 = unpk2(f0.z.re), i0 = unpk2(f0.z.im), r1 = unpk2(f1.z.re), i1 = unpk2(f1.z.im);
        const V a0 = make_float2(r0.x, i0.x), b0 = make_float2(r1.x, i1.x);
        const V a1 = make_float2(r0.y, i0.y), b1 = make_float2(r1.y, i1.y);
        V *hi = buf + 2 * o * BUF + at, *lo = hi + BUF;
        hi[0] = fadd2(a0, b0);
        hi[16] = fmulc_t(fsub2(a0, b0), w.x, w.y);
        lo[0] = fadd2(a1, b1);
        lo[16] = fmulc_t(fsub2(a1, b1), w.x, w.y);
    }
    // the first 16-point DFT and the transpose, to rows of xp
    __device__ __forceinline__ static void inverse_first(V v[16], V *xp, int lane)
    {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = xp[32 * j + lane];
        fdft16_inv(v);
        __syncwarp();
        const int h = lane >> 4, q2 = lane & 15;
#pragma unroll
        for (int m1p = 0; m1p < 16; ++m1p) xp[ROW * (2 * m1p + h) + q2] = v[m1p];
        __syncwarp();
    }
    // one limb (u & 1) of output u >> 1; sink(i, x) takes coefficient i of the
    // outputs, polynomial after polynomial
    template <class Sink>
    __device__ __forceinline__ static void inverse(V *xp, V *other, int u, int lane, uint32_t tm, Sink sink)
    {
        V v[16];
        inverse_first(v, xp, lane);
        const float4 *row = reinterpret_cast<const float4 *>(xp + ROW * lane);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            uint32_t x[16];
            twiddles(x, tm + 32, c);
#pragma unroll
            for (int k = 0; k < 8; k += 2) {
                const float4 z = row[4 * c + k / 2];
                const V t0 = entry(x, k), t1 = entry(x, k + 1);
                v[8 * c + k] = fmulc_t(make_float2(z.x, z.y), t0.x, t0.y);
                v[8 * c + k + 1] = fmulc_t(make_float2(z.z, z.w), t1.x, t1.y);
            }
        }
        fdft16_inv(v);
        uint32_t re[16], im[16];
#pragma unroll
        for (int m2 = 0; m2 < 16; ++m2) {
            const V c = cw64(make_float2(1.0f, 0.0f), m2);   // (cos, sin) of untwist_m2
            V y = m2 == 0 ? v[0] : fmulc_t(v[m2], c.x, c.y);
            // cos = sin: the paired form shares the product im cos, which is
            // then the rounded one
            if (m2 == 8) y.y = fmaf(-v[m2].x, c.x, __fmul_rn(v[m2].y, c.x));
            re[m2] = (u & 1) ? (uint32_t)__float2ll_rn(y.x) : hi_term(y.x);
            im[m2] = (u & 1) ? (uint32_t)__float2ll_rn(y.y) : hi_term(y.y);
        }
        join_limbs(re, im, xp, other, u, lane, sink);
    }
    // the hi warp takes both limbs of coefficients m, the lo warp of m + 512
    template <class Sink>
    __device__ __forceinline__ static void join_limbs(const uint32_t re[16], const uint32_t im[16], V *xp, V *other,
                                                      int u, int lane, Sink sink)
    {
        __syncwarp();
        uint32_t *mine = reinterpret_cast<uint32_t *>(xp) + lane;
        const uint32_t *theirs = reinterpret_cast<const uint32_t *>(other) + lane;
#pragma unroll
        for (int m2 = 0; m2 < 16; ++m2) mine[32 * m2] = (u & 1) ? re[m2] : im[m2];
        limbs_sync(u >> 1);
        const int base = (u >> 1) * N1 + 512 * (u & 1) + lane;
#pragma unroll
        for (int m2 = 0; m2 < 16; ++m2) sink(base + 32 * m2, ((u & 1) ? im[m2] : re[m2]) + theirs[32 * m2]);
    }
};

// The external product's split path: the plain tables (fft_f32.cuh), whose twist
// and untwist are products of their own.
struct PlainPath : SplitPath {
    using Full = Fft512TablesPlain;
    static constexpr int TAB_WORD4 = offsetof(Full, w32p) / 16;
    // tensor memory (COLS as above): tw512, then twist
    __device__ __forceinline__ static const float4 *tables(const void *t)
    {
        return reinterpret_cast<const float4 *>(&reinterpret_cast<const Fft512TablesF *>(t)->plain);
    }
    __device__ __forceinline__ static void stage_tables(uint32_t tm, const Full &T, int lane)
    {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            uint32_t x[32];
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                const V z = (c ? T.twist : T.tw512)[q * 32 + lane];
                x[2 * q] = __float_as_uint(z.x);
                x[2 * q + 1] = __float_as_uint(z.y);
            }
            tmem_st32_nowait(tm + 32 * c, x);
        }
        tmem_wait_st();
    }
    __device__ __forceinline__ static void forward(V v[16], V *xp, int lane, uint32_t tm)
    {
        const uint32_t *dig = reinterpret_cast<const uint32_t *>(xp) + lane;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            uint32_t x[16];
            twiddles(x, tm + 32, c);
#pragma unroll
            for (int k = 0; k < 8; ++k) v[8 * c + k] = fcmul(unpack(dig[32 * (8 * c + k)]), entry(x, k));
        }
        fdft16<1>(v);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            uint32_t x[16];
            twiddles(x, tm, c);
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (8 * c + k > 0) v[8 * c + k] = fcmul(v[8 * c + k], entry(x, k));
        }
        forward_rest(v, xp, lane);
    }
    __device__ __forceinline__ static V w32_fwd(const Tab &T, int jl, int hh) { return w32_inv(T, jl, hh); }
    template <class Sink>
    __device__ __forceinline__ static void inverse(V *xp, V *other, int u, int lane, uint32_t tm, Sink sink)
    {
        V v[16];
        inverse_first(v, xp, lane);
        const float4 *row = reinterpret_cast<const float4 *>(xp + ROW * lane);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            uint32_t x[16];
            twiddles(x, tm, c);
#pragma unroll
            for (int k = 0; k < 8; k += 2) {
                const float4 z = row[4 * c + k / 2];
                const V t0 = entry(x, k), t1 = entry(x, k + 1), z0 = make_float2(z.x, z.y);
                v[8 * c + k] = 8 * c + k > 0 ? fmulc_t(z0, t0.x, t0.y) : z0;
                v[8 * c + k + 1] = fmulc_t(make_float2(z.z, z.w), t1.x, t1.y);
            }
        }
        fdft16_inv(v);
        uint32_t re[16], im[16];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            uint32_t x[16];
            twiddles(x, tm + 32, c);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                // times conj(twist) / 512 (the scale is a power of two)
                const V a = v[8 * c + k], t = entry(x, k);
                const float cs = t.x * (1.0f / 512.0f), sn = -t.y * (1.0f / 512.0f);
                const float yr = fmaf(a.x, cs, -__fmul_rn(a.y, sn)), yi = fmaf(a.x, sn, __fmul_rn(a.y, cs));
                re[8 * c + k] = (u & 1) ? (uint32_t)__float2ll_rn(yr) : (uint32_t)__float2int_rn(yr) << 24;
                im[8 * c + k] = (u & 1) ? (uint32_t)__float2ll_rn(yi) : (uint32_t)__float2int_rn(yi) << 24;
            }
        }
        join_limbs(re, im, xp, other, u, lane, sink);
    }
};

struct F64Path {
    using V = double2;
    using Full = Fft512Tables;
    struct Tab {
        double2 w32[16];
    };
    static constexpr int TAB_WORD4 = offsetof(Full, w32) / 16;
    static constexpr int BUF = FFT512_XP;
    static constexpr int INV = 2;            // one inverse transform per output
    static constexpr uint32_t COLS = 128;    // tw512, then twist
    struct Sum {
        double2 z;
    };
    __device__ __forceinline__ static const float4 *tables(const void *t) { return reinterpret_cast<const float4 *>(t); }
    __device__ __forceinline__ static void stage_tables(uint32_t tm, const Full &T, int lane)
    {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const double2 *src = c < 2 ? T.tw512 : T.twist;
            uint32_t x[32];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const double2 z = src[(8 * (c & 1) + k) * 32 + lane];
                x[4 * k] = (uint32_t)__double2loint(z.x);
                x[4 * k + 1] = (uint32_t)__double2hiint(z.x);
                x[4 * k + 2] = (uint32_t)__double2loint(z.y);
                x[4 * k + 3] = (uint32_t)__double2hiint(z.y);
            }
            tmem_st32_nowait(tm + 32 * c, x);
        }
        tmem_wait_st();
    }
    // f(k, entry k) for the 16 entries of this lane at column tm
    template <class F>
    __device__ __forceinline__ static void each(uint32_t tm, F f)
    {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            uint32_t x[32];
            tmem_ld32_nowait(tm + 32 * c, x);
            tmem_wait_ld();
            tmem_landed<32>(x);
#pragma unroll
            for (int k = 0; k < 8; ++k)
                f(8 * c + k, make_double2(__hiloint2double((int)x[4 * k + 1], (int)x[4 * k]),
                                          __hiloint2double((int)x[4 * k + 3], (int)x[4 * k + 2])));
        }
    }
    __device__ __forceinline__ static void forward(V v[16], V *xp, int lane, uint32_t tm)
    {
        const uint32_t *dig = reinterpret_cast<const uint32_t *>(xp) + lane;
        each(tm + 64, [&](int m2, double2 tw) {
            // 2^52 + u, less 2^52 + 32: exact, and off the conversion unit
            const uint32_t u = dig[32 * m2];
            const double d0 = __hiloint2double(0x43300000, (int)(u & 0xFFFFu)) - 4503599627370528.0;
            const double d1 = __hiloint2double(0x43300000, (int)(u >> 16)) - 4503599627370528.0;
            v[m2] = cmul(make_double2(d0, d1), tw);
        });
        dft16<1>(v);
        each(tm, [&](int q2, double2 tw) {
            if (q2) v[q2] = cmul(v[q2], tw);
        });
        __syncwarp();
#pragma unroll
        for (int q2 = 0; q2 < 16; ++q2) xp[xp_index(lane, q2)] = v[q2];
        __syncwarp();
        const int h = lane >> 4, q2 = lane & 15;
#pragma unroll
        for (int m1p = 0; m1p < 16; ++m1p) v[m1p] = xp[xp_index(2 * m1p + h, q2)];
        dft16<1>(v);
    }
    __device__ __forceinline__ static V w32_fwd(const Tab &T, int jl, int hh) { return T.w32[jl + 8 * hh]; }
    __device__ __forceinline__ static V w32_inv(const Tab &T, int jl, int hh) { return T.w32[jl + 8 * hh]; }
    __device__ __forceinline__ static V mul(V a, V b) { return cmul(a, b); }
    __device__ __forceinline__ static V add(V a, V b) { return cadd(a, b); }
    __device__ __forceinline__ static V sub(V a, V b) { return csub(a, b); }
    __device__ __forceinline__ static void mac(Sum &f, bool first, V v, float4 k)
    {
        const double2 kd = *reinterpret_cast<const double2 *>(&k);
        if (first) f.z = cmul(v, kd);
        else cfma(f.z, v, kd);
    }
    __device__ __forceinline__ static void put(V *buf, int o, int at, const Sum &f0, const Sum &f1, V w)
    {
        V *b = buf + o * BUF + at;
        b[0] = cadd(f0.z, f1.z);
        b[16] = cmulc(csub(f0.z, f1.z), w);
    }
    template <class Sink>
    __device__ __forceinline__ static void inverse(V *xp, V *, int u, int lane, uint32_t tm, Sink sink)
    {
        V v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = xp[32 * j + lane];
        dft16<-1>(v);
        __syncwarp();
        const int h = lane >> 4, q2 = lane & 15;
#pragma unroll
        for (int m1p = 0; m1p < 16; ++m1p) xp[xp_index(2 * m1p + h, q2)] = v[m1p];
        __syncwarp();
        each(tm, [&](int k, double2 tw) {
            const double2 z = xp[xp_index(lane, k)];
            v[k] = k ? cmulc(z, tw) : z;
        });
        dft16<-1>(v);
        each(tm + 64, [&](int m2, double2 tw) {
            const int m = u * N1 + lane + 32 * m2;
            const double2 y = cmulc(v[m2], tw);
            sink(m, f64_to_torus32(y.x * (1.0 / 512.0)));
            sink(m + 512, f64_to_torus32(y.y * (1.0 / 512.0)));
        });
    }
};

// digits of one coefficient pair, packed by row: u(m) | u(m + 512) << 16 with
// u = digit + 32, into row buffers row0 .. row0 + 2 (BUF entries of P::V each)
template <class P>
__device__ __forceinline__ void put_digits(typename P::V *row0, int m, uint32_t c0, uint32_t c1)
{
    const uint32_t x0 = c0 + DEC1_OFFSET + DEC1_ROUND, x1 = c1 + DEC1_OFFSET + DEC1_ROUND;
#pragma unroll
    for (int d = 0; d < L1; ++d) {
        const int sh = 32 - BGBIT1 * (d + 1);
        reinterpret_cast<uint32_t *>(row0 + d * P::BUF)[m] = ((x0 >> sh) & 63u) | (((x1 >> sh) & 63u) << 16);
    }
}

// The products of slots jl and 8 + jl of this lane = (hh, q2): the radix-2 step
// that ends the transforms, X_0[j] +- W32^j X_1[j] with j = jl + 8 hh, at [j][q2] and
// [j][16 + q2] of each row's buffer, which no other thread reads; the
// multiply-accumulate with the TRGSW (row r, slot s, output o of this lane at
// g[1024 r + 64 s + 32 o]); the radix-2 step that begins the inverses, in place.
template <class P>
__device__ __forceinline__ void products(typename P::V *buf, const float4 *g, const typename P::Tab &T, int jl, int lane)
{
    using V = typename P::V;
    const int hh = lane >> 4, at = (jl + 8 * hh) * 32 + (lane & 15);
    const float4 *k = g + 64 * jl;
    const V wf = P::w32_fwd(T, jl, hh);
    typename P::Sum s[2][2];   // [slot][output]
#pragma unroll
    for (int r = 0; r < 2 * L1; ++r) {
        const V x = buf[r * P::BUF + at], t = P::mul(buf[r * P::BUF + at + 16], wf);
        const V v0 = P::add(x, t), v1 = P::sub(x, t);
#pragma unroll
        for (int o = 0; o < 2; ++o) {
            P::mac(s[0][o], r == 0, v0, __ldg(k + r * 1024 + 32 * o));
            P::mac(s[1][o], r == 0, v1, __ldg(k + r * 1024 + 512 + 32 * o));
        }
    }
    const V wi = P::w32_inv(T, jl, hh);
    P::put(buf, 0, at, s[0][0], s[1][0], wi);
    P::put(buf, 1, at, s[0][1], s[1][1], wi);
}

}  // namespace cfdb
