// Batched lvl0 -> lvl1 programmable bootstrapping (GateBootstrappingTLWE2TLWEFFT
// <lvl01param>, thirdparty/TFHEpp/src/gatebootstrapping.cpp:14-23: 672 x
// CMUXFFTwithPolynomialMulByXaiMinusOne, src/detwfa.cpp:20-35, then
// SampleExtractIndex(0), src/trlwe.cpp:108-118), one ciphertext per CTA, FP64 and
// split-precision FP32.
//
// A CTA of NW warps carries its ciphertext through the blind rotation; several
// CTAs share an SM and run out of step, so one's transforms fill the scheduler
// while another waits at a barrier, and a batch of any size is spread over the
// SMs as CTAs finish.  A CMux is four steps with a block barrier after each:
//   digits      all warps: the signed digits of (X^a - 1) acc, both polynomials,
//               packed two to a word per TRGSW row;
//   transforms  one warp per row: twist, 16 x 32-point transform (16 points per
//               lane), up to its last radix-2 step;
//   products    per (lane, slot pair): that radix-2 step of every row, the
//               multiply-accumulate into both outputs, and the first radix-2 step
//               of the inverse transforms, in place; the steps that cross lanes
//               in a one-warp transform need no shuffle here;
//   inverses    one warp per output and, on the split path, per limb.
// What bounds it is the shared-memory pipe, so what need not go through it does
// not: the per-lane twiddle tables sit in tensor memory (tcgen05.ld into the
// lanes that use them; from shared memory they were a seventh of the split
// path's and a fifth of the FP64 path's wavefronts), and the key is read from L2
// straight into the registers of the one thread that needs each value.
#include <cstddef>

#include "pbs_common.cuh"
#include "split_steps.cuh"
#include "tc_stage1.cuh"
#include "tmem_exchange.cuh"

namespace cfdb {

namespace {

// One polynomial's share of the paired inverse (fft_f32.cuh pfft512_inv), in
// scalar form with the paired form's roundings.  The compiler fuses a packed
// product into the packed addition or subtraction that takes it (the first
// operand's product where both are products), so the fused forms are written
// out here; the tests compare whole bootstraps of both kernels word for word.
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
    __device__ __forceinline__ static void forward(V v[16], V *xp, int lane, uint32_t tm)
    {
        const uint32_t *dig = reinterpret_cast<const uint32_t *>(xp) + lane;
#pragma unroll
        for (int m2 = 0; m2 < 16; ++m2) {
            // 2^23 + u has u in its low mantissa bits; the subtraction of 2^23 + 32
            // is exact (the int -> float conversion has an eighth of its rate)
            const uint32_t u = dig[32 * m2];
            const V d = fsub2(make_float2(__uint_as_float(0x4B000000u | (u & 0xFFFFu)),
                                          __uint_as_float(0x4B000000u | (u >> 16))),
                              make_float2(8388640.0f, 8388640.0f));
            v[m2] = cw64(d, m2);
        }
        fdft16<1>(v);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            uint32_t x[16];
            twiddles(x, tm, c);
#pragma unroll
            for (int k = 0; k < 8; ++k) v[8 * c + k] = fcmul(v[8 * c + k], entry(x, k));
        }
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
    // one limb (u & 1) of output u >> 1
    __device__ __forceinline__ static void inverse(uint32_t *acc, V *xp, V *other, int u, int lane, uint32_t tm)
    {
        V v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = xp[32 * j + lane];
        fdft16_inv(v);
        __syncwarp();
        const int h = lane >> 4, q2 = lane & 15;
#pragma unroll
        for (int m1p = 0; m1p < 16; ++m1p) xp[ROW * (2 * m1p + h) + q2] = v[m1p];
        __syncwarp();
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
        // the hi warp adds both limbs of coefficients m, the lo warp of m + 512
        __syncwarp();
        uint32_t *mine = reinterpret_cast<uint32_t *>(xp) + lane;
        const uint32_t *theirs = reinterpret_cast<const uint32_t *>(other) + lane;
#pragma unroll
        for (int m2 = 0; m2 < 16; ++m2) mine[32 * m2] = (u & 1) ? re[m2] : im[m2];
        limbs_sync(u >> 1);
        uint32_t *poly = acc + (u >> 1) * N1 + 512 * (u & 1) + lane;
#pragma unroll
        for (int m2 = 0; m2 < 16; ++m2) poly[32 * m2] += ((u & 1) ? im[m2] : re[m2]) + theirs[32 * m2];
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
    __device__ __forceinline__ static void inverse(uint32_t *acc, V *xp, V *, int u, int lane, uint32_t tm)
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
        uint32_t *poly = acc + u * N1;
        each(tm + 64, [&](int m2, double2 tw) {
            const int m = lane + 32 * m2;
            const double2 y = cmulc(v[m2], tw);
            poly[m] += f64_to_torus32(y.x * (1.0 / 512.0));
            poly[m + 512] += f64_to_torus32(y.y * (1.0 / 512.0));
        });
    }
};

template <class P>
struct CtSmem {
    static constexpr int TAB_OFF = 64;
    static constexpr int ACC_OFF = TAB_OFF + ((int)sizeof(typename P::Tab) + 63) / 64 * 64;
    static constexpr int BUF_OFF = ACC_OFF + 2 * N1 * 4;
    static constexpr int TOTAL = BUF_OFF + 2 * L1 * P::BUF * (int)sizeof(typename P::V);
};

template <class P, int NW, int OCC>
__global__ void __launch_bounds__(32 * NW, OCC) pbs01_ct_kernel(Pbs01Args a)
{
    using L = CtSmem<P>;
    using V = typename P::V;
    constexpr int NT = 32 * NW, BUF = P::BUF;
    static_assert(NW >= 2 * L1, "one warp per row");
    extern __shared__ __align__(128) unsigned char smem[];
    uint32_t *slot = reinterpret_cast<uint32_t *>(smem);
    typename P::Tab *T = reinterpret_cast<typename P::Tab *>(smem + L::TAB_OFF);
    uint32_t *acc = reinterpret_cast<uint32_t *>(smem + L::ACC_OFF);
    V *buf = reinterpret_cast<V *>(smem + L::BUF_OFF);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const float4 *tab = P::tables(a.tables);
    if (tid < (int)(sizeof(typename P::Tab) / 16)) reinterpret_cast<float4 *>(T)[tid] = tab[P::TAB_WORD4 + tid];
    if (warp == 0) tmem_alloc(slot, P::COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = *slot + ((32u * (warp & 3)) << 16);   // this sub-partition's lanes
    if (warp < 4) P::stage_tables(tm, *reinterpret_cast<const typename P::Full *>(tab), lane);

    const int ct = blockIdx.x;
    const uint32_t *in = a.in + (size_t)ct * (N0 + 1);
    uint32_t an = in[0];   // the next CMux's mask word, read one CMux ahead
    {
        const uint32_t bbar = 2 * N1 - (in[N0] >> 21);
        for (int j = tid; j < N1; j += NT) {
            acc[j] = 0;
            acc[N1 + j] = testvec_rot1(a.tv, j, bbar);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    // the key: row r, slot s, output o of this lane at [1024 r + 64 s + 32 o]
    const float4 *kg = reinterpret_cast<const float4 *>(a.bk) + lane;
    for (int i = 0; i < N0; ++i, kg += 2 * L1 * 1024) {
        const uint32_t ab = (an + (1u << 20)) >> 21;
        an = in[i + 1];
        if (ab == 0) continue;
        // digits: u(m) | u(m + 512) << 16 with u = digit + 32, m = lane + 32 m2
#pragma unroll
        for (int it = 0; it < (32 + NW - 1) / NW; ++it) {
            const int row = warp + NW * it;   // (polynomial, m2)
            if (row < 32) {
                const int pol = row >> 4, m = lane + 32 * (row & 15);
                const uint32_t *poly = acc + pol * N1;
                const uint32_t x0 = (rot_coef<N1>(poly, m, ab) - poly[m]) + DEC1_OFFSET + DEC1_ROUND;
                const uint32_t x1 = (rot_coef<N1>(poly, m + 512, ab) - poly[m + 512]) + DEC1_OFFSET + DEC1_ROUND;
#pragma unroll
                for (int d = 0; d < L1; ++d) {
                    const int sh = 32 - BGBIT1 * (d + 1);
                    reinterpret_cast<uint32_t *>(buf + (L1 * pol + d) * BUF)[m] =
                        ((x0 >> sh) & 63u) | (((x1 >> sh) & 63u) << 16);
                }
            }
        }
        __syncthreads();
        if (warp < 2 * L1) {
            V v[16];
            V *xp = buf + warp * BUF;
            P::forward(v, xp, lane, tm);
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 16; ++j) xp[32 * j + lane] = v[j];
        }
        __syncthreads();
        // lane = (hh, q2), slots jl and 8 + jl: X_0[j] +- W32^j X_1[j], j = jl + 8 hh,
        // at [j][q2] and [j][16 + q2], which no other thread reads
#pragma unroll
        for (int it = 0; it < (8 + NW - 1) / NW; ++it) {
            const int jl = warp + NW * it;
            if (jl < 8) {
                const int hh = lane >> 4, at = (jl + 8 * hh) * 32 + (lane & 15);
                const float4 *k = kg + 64 * jl;
                const V wf = P::w32_fwd(*T, jl, hh);
                typename P::Sum s[2][2];   // [slot][output]
#pragma unroll
                for (int r = 0; r < 2 * L1; ++r) {
                    const V x = buf[r * BUF + at], t = P::mul(buf[r * BUF + at + 16], wf);
                    const V v0 = P::add(x, t), v1 = P::sub(x, t);
#pragma unroll
                    for (int o = 0; o < 2; ++o) {
                        P::mac(s[0][o], r == 0, v0, __ldg(k + r * 1024 + 32 * o));
                        P::mac(s[1][o], r == 0, v1, __ldg(k + r * 1024 + 512 + 32 * o));
                    }
                }
                const V wi = P::w32_inv(*T, jl, hh);
                P::put(buf, 0, at, s[0][0], s[1][0], wi);
                P::put(buf, 1, at, s[0][1], s[1][1], wi);
            }
        }
        __syncthreads();
        if (warp < P::INV) P::inverse(acc, buf + warp * BUF, buf + (warp ^ 1) * BUF, warp, lane, tm);
        __syncthreads();
    }
    uint32_t *o = a.out + (size_t)ct * (N1 + 1);
    for (int j = tid; j < N1; j += NT) o[j] = j == 0 ? acc[0] : (uint32_t)(0u - acc[N1 - j]);
    if (tid == 0) o[N1] = acc[N1] + a.out_b_add;
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(*slot, P::COLS);
    }
}

template <class P, int NW, int OCC>
cudaError_t launch_ct_t(const Pbs01Args &a, cudaStream_t st)
{
    pbs01_ct_kernel<P, NW, OCC><<<a.B, 32 * NW, CtSmem<P>::TOTAL, st>>>(a);
    return cudaGetLastError();
}

template <class P, int NW, int OCC>
cudaError_t init_ct_t()
{
    return cudaFuncSetAttribute(pbs01_ct_kernel<P, NW, OCC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                CtSmem<P>::TOTAL);
}

}  // namespace

// Warps per CTA and CTAs per SM.  Eight warps divide the products evenly; the
// registers then leave two to four CTAs per SM on the split path: 128 registers
// let the transforms keep more loads in flight, more CTAs hide more latency, so
// the variant follows the CTAs an SM gets.  ms on 148 SMs, 2 / 3 / 4 per SM:
//   148: 1.86 / 2.08 / 2.36;  296: 2.88 / 2.86 / 2.95;  444: 4.52 / 3.86 / 3.89;
//   592: 5.74 / 5.43 / 4.97;  1,024: 9.95 / 8.86 / 8.60
// (one warp per ciphertext, 4 to 8 of them per persistent CTA: 7.50 ms up to 592,
// 9.40 ms at 1,024).
cudaError_t launch_pbs01_split(const Pbs01Args &a, int num_sms, cudaStream_t st)
{
    if (a.B <= 0) return cudaSuccess;
    if (a.B <= num_sms) return launch_ct_t<SplitPath, 8, 2>(a, st);
    if (a.B <= 3 * num_sms) return launch_ct_t<SplitPath, 8, 3>(a, st);
    return launch_ct_t<SplitPath, 8, 4>(a, st);
}

// FP64: two CTAs per SM (60 KB and 64 values' registers each).  Alone on its SM a
// ciphertext is faster with eight warps (2.28 ms against 2.51 with six); two
// of them with six warps of 168 registers (296: 3.43 ms against 3.81 with eight;
// 1,024: 12.1 against 12.9; one warp per ciphertext: 10.5 ms up to 592, 14.2 ms
// at 1,024).
cudaError_t launch_pbs01_f64(const Pbs01Args &a, int num_sms, cudaStream_t st)
{
    if (a.B <= 0) return cudaSuccess;
    return a.B <= num_sms ? launch_ct_t<F64Path, 8, 2>(a, st) : launch_ct_t<F64Path, 6, 2>(a, st);
}

cudaError_t init_pbs01_ct()
{
    cudaError_t e = init_ct_t<SplitPath, 8, 2>();
    if (e == cudaSuccess) e = init_ct_t<SplitPath, 8, 3>();
    if (e == cudaSuccess) e = init_ct_t<SplitPath, 8, 4>();
    if (e == cudaSuccess) e = init_ct_t<F64Path, 6, 2>();
    if (e == cudaSuccess) e = init_ct_t<F64Path, 8, 2>();
    return e;
}

}  // namespace cfdb
