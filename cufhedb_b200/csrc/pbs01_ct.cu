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
#include "block_fft.cuh"

namespace cfdb {

namespace {

constexpr uint32_t KEY_BYTES = 2 * L1 * 1024 * 16;   // of one CMux

template <class P>
struct CtSmem {
    static constexpr int TAB_OFF = 64;
    static constexpr int ACC_OFF = TAB_OFF + ((int)sizeof(typename P::Tab) + 63) / 64 * 64;
    static constexpr int BUF_OFF = ACC_OFF + 2 * N1 * 4;
    static constexpr int TOTAL = BUF_OFF + 2 * L1 * P::BUF * (int)sizeof(typename P::V);
};

// The first `askers` blocks ask the key of the CMux after next into L2, a share
// each.  A key switch of 5.6 GB has usually run before and left the key in DRAM,
// whose latency each CMux would then meet; ms with a cold L2, without -> with:
// split 1: 2.09 -> 1.96, 148: 1.95 -> 1.88, 1,024: 8.58 -> 8.48; FP64 1: 2.72 ->
// 2.43, 148: 2.52 -> 2.36, 1,024: 12.12 -> 12.11.  Three blocks per SM lose by it
// (444: 3.85 -> 3.90) and do without.
template <class P, int NW, int OCC>
__global__ void __launch_bounds__(32 * NW, OCC) pbs01_ct_kernel(Pbs01Args a, uint32_t askers)
{
    using L = CtSmem<P>;
    using V = typename P::V;
    constexpr int NT = 32 * NW, BUF = P::BUF;
    constexpr bool ASK = OCC != 3;
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
        if (ASK && tid == 0 && blockIdx.x < askers && i + 2 < N0) {
            const uint32_t share = (KEY_BYTES / 16 + askers - 1) / askers * 16, at = blockIdx.x * share;
            if (at < KEY_BYTES)
                bulk_prefetch_l2(reinterpret_cast<const unsigned char *>(a.bk) + (size_t)(i + 2) * KEY_BYTES + at,
                                 min(share, KEY_BYTES - at));
        }
        const uint32_t ab = (an + (1u << 20)) >> 21;
        an = in[i + 1];
        if (ab == 0) continue;
#pragma unroll
        for (int it = 0; it < (32 + NW - 1) / NW; ++it) {
            const int row = warp + NW * it;   // (polynomial, m2), m = lane + 32 m2
            if (row < 32) {
                const int pol = row >> 4, m = lane + 32 * (row & 15);
                const uint32_t *poly = acc + pol * N1;
                put_digits<P>(buf + L1 * pol * BUF, m, rot_coef<N1>(poly, m, ab) - poly[m],
                              rot_coef<N1>(poly, m + 512, ab) - poly[m + 512]);
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
#pragma unroll
        for (int it = 0; it < (8 + NW - 1) / NW; ++it)
            if (warp + NW * it < 8) products<P>(buf, kg, *T, warp + NW * it, lane);
        __syncthreads();
        if (warp < P::INV)
            P::inverse(buf + warp * BUF, buf + (warp ^ 1) * BUF, warp, lane, tm,
                       [&](int m, uint32_t x) { acc[m] += x; });
        __syncthreads();
    }
    __syncthreads();   // a row may be bootstrapped over itself, and skipped CMuxes have no barrier
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
cudaError_t launch_ct_t(const Pbs01Args &a, int num_sms, cudaStream_t st)
{
    pbs01_ct_kernel<P, NW, OCC><<<a.B, 32 * NW, CtSmem<P>::TOTAL, st>>>(a, a.B < num_sms ? a.B : num_sms);
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
    if (a.B <= num_sms) return launch_ct_t<SplitPath, 8, 2>(a, num_sms, st);
    if (a.B <= 3 * num_sms) return launch_ct_t<SplitPath, 8, 3>(a, num_sms, st);
    return launch_ct_t<SplitPath, 8, 4>(a, num_sms, st);
}

// FP64: two CTAs per SM (60 KB and 64 values' registers each).  Alone on its SM a
// ciphertext is faster with eight warps (2.28 ms against 2.51 with six); two
// of them with six warps of 168 registers (296: 3.43 ms against 3.81 with eight;
// 1,024: 12.1 against 12.9; one warp per ciphertext: 10.5 ms up to 592, 14.2 ms
// at 1,024).
cudaError_t launch_pbs01_f64(const Pbs01Args &a, int num_sms, cudaStream_t st)
{
    if (a.B <= 0) return cudaSuccess;
    return a.B <= num_sms ? launch_ct_t<F64Path, 8, 2>(a, num_sms, st) : launch_ct_t<F64Path, 6, 2>(a, num_sms, st);
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
