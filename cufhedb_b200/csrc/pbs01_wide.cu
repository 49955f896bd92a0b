// Batched lvl0 -> lvl1 programmable bootstrapping with one ciphertext per CTA:
// the kernel for batches that leave SMs idle, or part of their schedulers.
//
// The persistent kernels (pbs01_f64.cu, pbs01_split.cu) give each ciphertext
// one warp, which is what a full SM wants; a small batch then lasts 672 CMux
// of one warp's latency (22,000 cycles each on the split path).  Here 24 warps
// work on one ciphertext, three steps per CMux:
//   transforms  six teams of four warps, one per TRGSW row; a thread holds 4
//               of the 512 points, so the 16 x 32 transform of the one-warp
//               kernels becomes five register steps (4-point DFTs, the last
//               radix-2 step by shuffle) with three exchanges between the
//               warps of the team;
//   products    thread t < 512 takes frequency t of every row into both
//               outputs and leaves the sums where the spectra were;
//   inverses    one team per output and, on the split path, per limb (the two
//               limbs' teams then trade halves and add into the accumulator).
// Every value goes through the same operations with the same roundings in the
// same order as in the one-warp kernels, so the output words are the same.
//
// A pass of up to 148 ciphertexts takes 2.30 ms on the split path (4-per-CTA
// shape of the one-warp kernel: 7.50 ms) and 3.18 ms in FP64 (10.58 ms).  Of the
// 6,700 cycles of a split CMux the transforms take 3,000 (1,200 of them for the
// decomposition words, which every team of a polynomial forms for itself), the
// products 1,100 (bound by the 96 KB of key read from shared memory), the
// inverses 2,300.  Sixteen points per thread, one warp per transform, measured
// 2.86 ms and 3.60 ms.
#include "f64_steps.cuh"
#include "pbs_common.cuh"
#include "split_steps.cuh"

namespace cfdb {

namespace {

constexpr int WIDE_WARPS = 24;

// The six key rows of one CMux in shared memory, one bulk copy (they are
// contiguous), refilled after the barrier that ends the products.  Waits are
// bounded; after one gives up nothing is waited for or issued any more.
struct CmuxKey {
    static constexpr uint32_t BYTES = 2 * L1 * 16384;
    uint64_t *full;
    int *abort_flag;
    unsigned char *rows;
    const unsigned char *src;
    uint32_t issued = 0;    // by the issuing thread

    __device__ __forceinline__ void init()
    {
        *abort_flag = 0;
        mbar_init(full, 1);
        fence_barrier_init();
    }
    __device__ __forceinline__ bool aborted() const { return *(volatile int *)abort_flag != 0; }
    // the rows of CMux i (one thread, after every reader's barrier)
    __device__ __forceinline__ void issue(int i)
    {
        if (aborted()) return;
        ++issued;
        fence_proxy_async_smem();
        mbar_arrive_expect_tx(full, BYTES);
        bulk_g2s(rows, src + (size_t)i * BYTES, BYTES, full);
    }
    // the rows of the CMux with running number n
    __device__ __forceinline__ const unsigned char *acquire(uint32_t n, int *err)
    {
        if (!aborted() && !mbar_wait(full, n & 1)) {
            report_error(err, DEV_TIMEOUT_FULL);
            *(volatile int *)abort_flag = 1;
        }
        return rows;
    }
    // the issuing thread, at the end: nothing may still be landing
    __device__ __forceinline__ void drain(int *err)
    {
        if (aborted() && issued != 0 && !mbar_wait(full, (issued - 1) & 1)) report_error(err, DEV_TIMEOUT_DRAIN);
    }
};

// ---- arithmetic, float2 and double2 ------------------------------------------------
__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return fadd2(a, b); }
__device__ __forceinline__ float2 vsub(float2 a, float2 b) { return fsub2(a, b); }
__device__ __forceinline__ double2 vadd(double2 a, double2 b) { return make_double2(__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y)); }
__device__ __forceinline__ double2 vsub(double2 a, double2 b) { return make_double2(__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y)); }
__device__ __forceinline__ float rfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double rfma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float rmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double rmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float radd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double radd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float2 vmake(float x, float y) { return make_float2(x, y); }
__device__ __forceinline__ double2 vmake(double x, double y) { return make_double2(x, y); }
__device__ __forceinline__ float2 vshfl(float2 v) { return shfl_xor_f2(v, 16); }
__device__ __forceinline__ double2 vshfl(double2 v) { return shfl_xor2(v, 16); }
template <class V>
using real_t = decltype(V::x);

// fcmul / cmul
template <class V>
__device__ __forceinline__ V vcmul(V a, V b)
{
    return vmake(rfma(a.x, b.x, -rmul(a.y, b.y)), rfma(a.x, b.y, rmul(a.y, b.x)));
}
// a conj(b): pmulc_t as compiled (the subtraction fused with its first
// product) and cmulc are the same operations
template <class V>
__device__ __forceinline__ V vcmulc(V a, V b)
{
    return vmake(rfma(a.x, b.x, rmul(a.y, b.y)), rfma(a.y, b.x, -rmul(a.x, b.y)));
}
// b + k a
template <class V>
__device__ __forceinline__ V vaxpy(real_t<V> k, V a, V b)
{
    return vmake(rfma(a.x, k, b.x), rfma(a.y, k, b.y));
}

template <int S, class V>
__device__ __forceinline__ void finish4(V v[4], V s02, V d02, V s13, V d13)
{
    const V t = S > 0 ? vmake(-d13.y, d13.x) : vmake(d13.y, -d13.x);
    v[0] = vadd(s02, s13);
    v[2] = vsub(s02, s13);
    v[1] = vadd(d02, t);
    v[3] = vsub(d02, t);
}

// The 16-point DFT (fdft16 / dft16 / pdft16) over four threads: thread w holds
// inputs w + 4 n in v[n] and does the first 4-point DFT and its twiddles
// W16^{w k}, ...
// FUSED: the factor 1/sqrt 2 of the twiddles W16^2 and W16^6 is applied by the
// fused multiply-add of the step that takes the product, as the compiler does
// for the one-warp kernels' FP64 and packed FP32 code; otherwise by a product
// of its own (their scalar FP32 code).
template <int S, bool FUSED, class V>
__device__ __forceinline__ void dft16_first(V v[4], int w)
{
    using R = real_t<V>;
    constexpr R C1 = (R)0.92387953251128673848, S1 = (R)0.38268343236508978178, R2 = (R)0.70710678118654752440;
    finish4<S>(v, vadd(v[0], v[2]), vsub(v[0], v[2]), vadd(v[1], v[3]), vsub(v[1], v[3]));
    auto rot = [](V a, R c, R s) { return vmake(rfma(a.x, c, -rmul(a.y, s)), rfma(a.x, s, rmul(a.y, c))); };
    auto scaled = [](V a) { return FUSED ? a : vmake(rmul(R2, a.x), rmul(R2, a.y)); };
    auto e2 = [&](V a) {
        return scaled(S > 0 ? vmake(radd(a.x, -a.y), radd(a.x, a.y)) : vmake(radd(a.x, a.y), radd(a.y, -a.x)));
    };
    auto e6 = [&](V a) {
        return scaled(S > 0 ? vmake(-radd(a.x, a.y), radd(a.x, -a.y)) : vmake(radd(a.y, -a.x), -radd(a.x, a.y)));
    };
    constexpr R sg = (R)S;
    if (w == 1) {
        v[1] = rot(v[1], C1, sg * S1);
        v[2] = e2(v[2]);
        v[3] = rot(v[3], S1, sg * C1);
    } else if (w == 2) {
        v[1] = e2(v[1]);
        v[2] = S > 0 ? vmake(-v[2].y, v[2].x) : vmake(v[2].y, -v[2].x);
        v[3] = e6(v[3]);
    } else if (w == 3) {
        v[1] = rot(v[1], S1, sg * C1);
        v[2] = e6(v[2]);
        v[3] = rot(v[3], -C1, -sg * S1);
    }
}
// ... then, holding every thread's value k = w, the second 4-point DFT:
// v[k1] = X[w + 4 k1]
template <int S, bool FUSED, class V>
__device__ __forceinline__ void dft16_second(V v[4], int w)
{
    using R = real_t<V>;
    constexpr R R2 = (R)0.70710678118654752440;
    V s02, d02, s13, d13;
    if (FUSED && (w & 1)) {
        s02 = vaxpy(R2, v[2], v[0]);
        d02 = vaxpy(-R2, v[2], v[0]);
    } else {
        s02 = vadd(v[0], v[2]);
        d02 = vsub(v[0], v[2]);
    }
    if (FUSED && w == 2) {
        const V p = vmake(rmul(v[3].x, R2), rmul(v[3].y, R2));
        s13 = vaxpy(R2, v[1], p);
        d13 = vaxpy(R2, v[1], vmake(-p.x, -p.y));
    } else {
        s13 = vadd(v[1], v[3]);
        d13 = vsub(v[1], v[3]);
    }
    finish4<S>(v, s02, d02, s13, d13);
}

// the 128 threads of a team meet (barriers 1 .. 6)
__device__ __forceinline__ void team_sync(int team) { asm volatile("bar.sync %0, 128;" ::"r"(1 + team) : "memory"); }
// the teams of both limbs of output o meet (barriers 7, 8)
__device__ __forceinline__ void limbs_sync(int o) { asm volatile("bar.sync %0, 256;" ::"r"(7 + o) : "memory"); }

// v[k] of thread w -> v[w'] of thread k, same lane
template <class V>
__device__ __forceinline__ void trade(V v[4], V *x, int team, int w, int lane)
{
#pragma unroll
    for (int k = 0; k < 4; ++k) x[(4 * k + w) * 32 + lane] = v[k];
    team_sync(team);
#pragma unroll
    for (int n = 0; n < 4; ++n) v[n] = x[(4 * w + n) * 32 + lane];
}

// Per-thread constants of the transforms (warp w of a team, lane): the
// per-register twist, both directions' stage-1 twiddles, the radix-2 ones.
struct SplitPath {
    using V = float2;
    using Tab = Fft512TablesFold;
    static constexpr bool FWD_FUSED = false;
    static constexpr int INV = 4;   // inverse transforms: output x limb
    struct Const {
        V cw[4];     // w^{32 m2}, m2 = w + 4 n
        V fwd[4];    // tw512w, q2 = w + 4 n
        V inv[4];    // tw512u, q2 = w + 4 n
        V r2f[2];    // e^{2 pi i j / 32}, j = w + 4 e
        V r2i[2];    // the same at j + 8 h
    };
    __device__ __forceinline__ static const float4 *tables(const void *t)
    {
        return reinterpret_cast<const float4 *>(&reinterpret_cast<const Fft512TablesF *>(t)->fold);
    }
    __device__ __forceinline__ static void constants(Const &c, const Tab &T, int w, int lane)
    {
        const int h = lane >> 4;
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            c.cw[n] = make_float2(1.0f, 0.0f);
#pragma unroll
            for (int m2 = 1; m2 < 16; ++m2)
                if (m2 == w + 4 * n) c.cw[n] = cw64(make_float2(1.0f, 0.0f), m2);
            c.fwd[n] = T.tw512w[(w + 4 * n) * 32 + lane];
            const float4 u = T.tw512u[(w + 4 * n) * 32 + lane];
            c.inv[n] = make_float2(u.x, u.z);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (j == w + 4 * e) c.r2f[e] = w32_const(j);
            const float4 u = T.w32p[w + 4 * e + 8 * h];
            c.r2i[e] = make_float2(u.x, u.z);
        }
    }
    // digits from their 6-bit fields u = digit + 32: 2^23 + u has u in its low
    // mantissa bits, and the subtraction is exact (an int -> float conversion
    // runs at an eighth of the rate, and 24 warps convert at once)
    __device__ __forceinline__ static V digit(uint32_t u0, uint32_t u1, const Const &c, const Tab &, int n, int, int)
    {
        const float2 d = fsub2(make_float2(__uint_as_float(0x4B000000u | u0), __uint_as_float(0x4B000000u | u1)),
                               make_float2(8388640.0f, 8388640.0f));
        return vcmul(d, c.cw[n]);
    }
    __device__ __forceinline__ static V fwd_tw(V v, const Const &c, const Tab &, int n, int, int)
    {
        return vcmul(v, c.fwd[n]);
    }
    __device__ __forceinline__ static V radix2(V b, const Const &c, const Tab &, int e, int, int h)
    {
        const V t = vcmul(b, c.r2f[e]);
        return h ? make_float2(-t.y, t.x) : t;
    }
    __device__ __forceinline__ static V radix2_inv(V b, const Const &c, const Tab &, int e, int, int)
    {
        return vcmulc(b, c.r2i[e]);
    }
    __device__ __forceinline__ static V inv_tw(V v, const Const &c, const Tab &, int n, int, int)
    {
        return vcmulc(v, c.inv[n]);
    }
    struct Sum {
        CP z;
    };
    __device__ __forceinline__ static void mac(Sum &f, bool first, V v, float4 k)
    {
        if (first) f.z = pmul_first(pk2(v.x, v.x), pk2(v.y, v.y), pk2(-v.y, -v.y), k);
        else pmac(f.z, pk2(v.x, v.x), pk2(v.y, v.y), pk2(-v.y, -v.y), k);
    }
    // buffers 2 o and 2 o + 1: the hi and the lo limb of output o
    __device__ __forceinline__ static void put(V *buf, int stride, int o, int t, const Sum &f)
    {
        const float2 re = unpk2(f.z.re), im = unpk2(f.z.im);
        buf[(2 * o) * stride + t] = make_float2(re.x, im.x);
        buf[(2 * o + 1) * stride + t] = make_float2(re.y, im.y);
    }
    // v[k1]: coefficients m = lane + 32 (w + 4 k1) and m + 512 of one limb
    __device__ __forceinline__ static void finish(uint32_t *acc, V v[4], V *buf, int stride, int u, const Const &c,
                                                  const Tab &, int w, int lane)
    {
        uint32_t re[4], im[4];
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            V y = vcmulc(v[n], c.cw[n]);
            // m2 = 8, cos = sin: the paired form shares the product im cos,
            // which is then the rounded one
            if (n == 2 && w == 0) y.y = rfma(-v[n].x, c.cw[n].x, rmul(v[n].y, c.cw[n].x));
            re[n] = (u & 1) ? (uint32_t)__float2ll_rn(y.x) : hi_term(y.x);
            im[n] = (u & 1) ? (uint32_t)__float2ll_rn(y.y) : hi_term(y.y);
        }
        // the hi team adds both limbs of coefficients m, the lo team of m + 512
        uint32_t *mine = reinterpret_cast<uint32_t *>(buf + u * stride) + 32 * w + lane;
        const uint32_t *other = reinterpret_cast<const uint32_t *>(buf + (u ^ 1) * stride) + 32 * w + lane;
#pragma unroll
        for (int n = 0; n < 4; ++n) mine[128 * n] = (u & 1) ? re[n] : im[n];
        limbs_sync(u >> 1);
        uint32_t *poly = acc + (u >> 1) * N1 + 512 * (u & 1) + 32 * w + lane;
#pragma unroll
        for (int n = 0; n < 4; ++n) poly[128 * n] += ((u & 1) ? im[n] : re[n]) + other[128 * n];
    }
};

struct F64Path {
    using V = double2;
    using Tab = Fft512Tables;
    static constexpr bool FWD_FUSED = true;
    static constexpr int INV = 2;   // one inverse transform per output
    struct Const {};
    __device__ __forceinline__ static const float4 *tables(const void *t) { return reinterpret_cast<const float4 *>(t); }
    __device__ __forceinline__ static void constants(Const &, const Tab &, int, int) {}
    __device__ __forceinline__ static V digit(uint32_t u0, uint32_t u1, const Const &, const Tab &T, int n, int w,
                                              int lane)
    {
        const double d0 = __dsub_rn(__hiloint2double(0x43300000, (int)u0), 4503599627370528.0);
        const double d1 = __dsub_rn(__hiloint2double(0x43300000, (int)u1), 4503599627370528.0);
        return vcmul(make_double2(d0, d1), T.twist[(w + 4 * n) * 32 + lane]);
    }
    __device__ __forceinline__ static V fwd_tw(V v, const Const &, const Tab &T, int n, int w, int lane)
    {
        return n == 0 && w == 0 ? v : vcmul(v, T.tw512[(w + 4 * n) * 32 + lane]);
    }
    __device__ __forceinline__ static V radix2(V b, const Const &, const Tab &T, int e, int w, int h)
    {
        return vcmul(b, T.w32[w + 4 * e + 8 * h]);
    }
    __device__ __forceinline__ static V radix2_inv(V b, const Const &, const Tab &T, int e, int w, int h)
    {
        return vcmulc(b, T.w32[w + 4 * e + 8 * h]);
    }
    __device__ __forceinline__ static V inv_tw(V v, const Const &, const Tab &T, int n, int w, int lane)
    {
        return n == 0 && w == 0 ? v : vcmulc(v, T.tw512[(w + 4 * n) * 32 + lane]);
    }
    struct Sum {
        double2 z;
    };
    __device__ __forceinline__ static void mac(Sum &f, bool first, V v, float4 k)
    {
        const double2 kd = *reinterpret_cast<const double2 *>(&k);
        if (first) f.z = cmul(v, kd);
        else cfma(f.z, v, kd);
    }
    __device__ __forceinline__ static void put(V *buf, int stride, int o, int t, const Sum &f)
    {
        buf[o * stride + t] = f.z;
    }
    __device__ __forceinline__ static void finish(uint32_t *acc, V v[4], V *, int, int u, const Const &, const Tab &T,
                                                  int w, int lane)
    {
        uint32_t *poly = acc + u * N1 + 32 * w + lane;
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            const double2 y = vcmulc(v[n], T.twist[(w + 4 * n) * 32 + lane]);
            poly[128 * n] += f64_to_torus32(y.x * (1.0 / 512.0));
            poly[128 * n + 512] += f64_to_torus32(y.y * (1.0 / 512.0));
        }
    }
};

template <class P>
struct WideSmem {
    static constexpr int BUF = FFT512_XP;   // entries of one exchange / spectrum buffer
    static constexpr int BUFS_BYTES = 2 * L1 * BUF * (int)sizeof(typename P::V);
    static constexpr int TAB_OFF = 128;
    static constexpr int RING_OFF = TAB_OFF + ((int)sizeof(typename P::Tab) + 127) / 128 * 128;
    static constexpr int ACC_OFF = RING_OFF + (int)CmuxKey::BYTES;
    static constexpr int A_OFF = ACC_OFF + 2 * N1 * 4;
    static constexpr int B_OFF = A_OFF + BUFS_BYTES;
    static constexpr int TOTAL = B_OFF + BUFS_BYTES;
    static_assert(TOTAL <= 227 * 1024, "shared memory budget");
};

template <class P>
__global__ void __launch_bounds__(WIDE_WARPS * 32, 1) pbs01_wide_kernel(Pbs01Args a)
{
    using L = WideSmem<P>;
    using V = typename P::V;
    constexpr int NT = WIDE_WARPS * 32, BUF = L::BUF;
    extern __shared__ __align__(128) unsigned char smem[];
    typename P::Tab *T = reinterpret_cast<typename P::Tab *>(smem + L::TAB_OFF);
    uint32_t *acc = reinterpret_cast<uint32_t *>(smem + L::ACC_OFF);
    V *bufA = reinterpret_cast<V *>(smem + L::A_OFF), *bufB = reinterpret_cast<V *>(smem + L::B_OFF);
    CmuxKey key{reinterpret_cast<uint64_t *>(smem), reinterpret_cast<int *>(smem + 64), smem + L::RING_OFF,
                reinterpret_cast<const unsigned char *>(a.bk)};
    const int tid = threadIdx.x, lane = tid & 31, team = tid >> 7, w = (tid >> 5) & 3;
    const int h = lane >> 4, q2 = lane & 15;
    // the key is issued by a thread of the last team, which has no inverse
    const bool issuer = tid == NT - 32;
    if (issuer) key.init();
    {
        const float4 *src = P::tables(a.tables);
        float4 *dst = reinterpret_cast<float4 *>(T);
        for (int i = tid; i < (int)(sizeof(typename P::Tab) / 16); i += NT) dst[i] = src[i];
    }
    __syncthreads();
    typename P::Const cst;
    P::constants(cst, *T, w, lane);
    uint32_t n = 0;   // running number of the CMux
    if (issuer) key.issue(0);

    for (int ct = blockIdx.x; ct < a.B; ct += gridDim.x) {
        const bool more = ct + (int)gridDim.x < a.B;
        const uint32_t *in = a.in + (size_t)ct * (N0 + 1);
        uint32_t an = in[0];   // the next CMux's mask word, read one CMux ahead
        {
            const uint32_t bbar = 2 * N1 - (in[N0] >> 21);
            for (int j = tid; j < N1; j += NT) {
                acc[j] = 0;
                acc[N1 + j] = testvec_rot1(a.tv, j, bbar);
            }
        }
        __syncthreads();

        for (int i = 0; i < N0; ++i, ++n) {
            const uint32_t ab = (an + (1u << 20)) >> 21;
            an = in[i + 1];
            if (ab) {
                // row `team`: digit polynomial team % 3 of polynomial team / 3
                const uint32_t *poly = acc + (team >= L1 ? N1 : 0);
                const int dsh = 32 - BGBIT1 * (1 + (team >= L1 ? team - L1 : team));
                V *xa = bufA + team * BUF, *xb = bufB + team * BUF;
                V v[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int m = lane + 32 * (w + 4 * k);
                    const uint32_t x0 = (rot_coef<N1>(poly, m, ab) - poly[m]) + DEC1_OFFSET + DEC1_ROUND;
                    const uint32_t x1 = (rot_coef<N1>(poly, m + 512, ab) - poly[m + 512]) + DEC1_OFFSET + DEC1_ROUND;
                    v[k] = P::digit((x0 >> dsh) & 63u, (x1 >> dsh) & 63u, cst, *T, k, w, lane);
                }
                dft16_first<1, P::FWD_FUSED>(v, w);
                trade(v, xa, team, w, lane);
                dft16_second<1, P::FWD_FUSED>(v, w);
#pragma unroll
                for (int k = 0; k < 4; ++k) xb[lane * 17 + w + 4 * k] = P::fwd_tw(v[k], cst, *T, k, w, lane);
                team_sync(team);
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] = xb[(2 * (w + 4 * k) + h) * 17 + q2];
                dft16_first<1, P::FWD_FUSED>(v, w);
                trade(v, xa, team, w, lane);
                dft16_second<1, P::FWD_FUSED>(v, w);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const V recv = vshfl(h ? v[e] : v[2 + e]);
                    const V x = h ? recv : v[e], t = P::radix2(h ? v[2 + e] : recv, cst, *T, e, w, h);
                    xb[(w + 4 * e) * 32 + lane] = vadd(x, t);
                    xb[(8 + w + 4 * e) * 32 + lane] = vsub(x, t);
                }
            }
            __syncthreads();
            if (tid < 512) {
                typename P::Sum f[2];
                // slot tid / 32, this lane: row r, output o at [1024 r + (2 slot + o) 32 + lane]
                const float4 *k = reinterpret_cast<const float4 *>(key.acquire(n, a.err)) + 64 * (tid >> 5) + lane;
#pragma unroll
                for (int r = 0; r < 2 * L1; ++r) {
                    const V v = bufB[r * BUF + tid];
                    P::mac(f[0], r == 0, v, k[1024 * r]);
                    P::mac(f[1], r == 0, v, k[1024 * r + 32]);
                }
                P::put(bufB, BUF, 0, tid, f[0]);
                P::put(bufB, BUF, 1, tid, f[1]);
            }
            __syncthreads();
            if (issuer && (i + 1 < N0 || more)) key.issue(i + 1 < N0 ? i + 1 : 0);
            if (ab && team < P::INV) {
                V *xa = bufA + team * BUF, *xb = bufB + team * BUF;
                V v[4];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const V x = xb[(w + 4 * e) * 32 + lane], y = xb[(8 + w + 4 * e) * 32 + lane];
                    const V g0 = vadd(x, y), g1 = P::radix2_inv(vsub(x, y), cst, *T, e, w, h);
                    const V recv = vshfl(h ? g0 : g1);
                    v[e] = h ? recv : g0;
                    v[2 + e] = h ? g1 : recv;
                }
                dft16_first<-1, true>(v, w);
                trade(v, xa, team, w, lane);
                dft16_second<-1, true>(v, w);
#pragma unroll
                for (int k = 0; k < 4; ++k) xb[(2 * (w + 4 * k) + h) * 17 + q2] = v[k];
                team_sync(team);
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] = P::inv_tw(xb[lane * 17 + w + 4 * k], cst, *T, k, w, lane);
                dft16_first<-1, true>(v, w);
                trade(v, xa, team, w, lane);
                dft16_second<-1, true>(v, w);
                P::finish(acc, v, bufB, BUF, team, cst, *T, w, lane);
            }
            __syncthreads();
        }
        uint32_t *o = a.out + (size_t)ct * (N1 + 1);
        for (int j = tid; j < N1; j += NT) o[j] = j == 0 ? acc[0] : (uint32_t)(0u - acc[N1 - j]);
        if (tid == 0) o[N1] = acc[N1] + a.out_b_add;
        __syncthreads();
    }
    if (issuer) key.drain(a.err);
}

template <class P>
cudaError_t launch_wide_t(const Pbs01Args &a, int num_sms, cudaStream_t st)
{
    if (a.B <= 0) return cudaSuccess;
    pbs01_wide_kernel<P><<<a.B < num_sms ? a.B : num_sms, WIDE_WARPS * 32, WideSmem<P>::TOTAL, st>>>(a);
    return cudaGetLastError();
}

template <class P>
cudaError_t init_wide_t()
{
    return cudaFuncSetAttribute(pbs01_wide_kernel<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, WideSmem<P>::TOTAL);
}

}  // namespace

cudaError_t launch_pbs01_wide_split(const Pbs01Args &a, int num_sms, cudaStream_t st)
{
    return launch_wide_t<SplitPath>(a, num_sms, st);
}

cudaError_t launch_pbs01_wide_f64(const Pbs01Args &a, int num_sms, cudaStream_t st)
{
    return launch_wide_t<F64Path>(a, num_sms, st);
}

cudaError_t init_pbs01_wide()
{
    const cudaError_t e = init_wide_t<SplitPath>();
    return e == cudaSuccess ? init_wide_t<F64Path>() : e;
}

}  // namespace cfdb
