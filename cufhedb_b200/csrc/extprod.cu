// Batched lvl1 external products TRGSW (x) TRLWE, FP64 and split-precision
// FP32 paths, plus the conversion of integer TRGSWs into the engine's
// frequency-domain layout.
//
// Restates trgswfftExternalProduct<lvl1param> (thirdparty/TFHEpp/src/
// trgsw.cpp:77-103): res_o = sum_{k,d} IFFT(dec_d(trlwe_k)) * trgsw[k l + d][o],
// transformed back per output polynomial.
//
// A block of six or eight warps takes one product at a time through the steps of
// a CMux (block_fft.cuh, pbs01_ct.cu), several blocks per SM, each looping over
// products.  The next product's TRLWE and TRGSW are asked into L2 when one's
// products are done (a whole product ahead, the blocks' 2 x 57 MB evicted one
// another: 716 MB from DRAM instead of 450).  The TRGSW rows (one per TRGSW or one shared by the batch) are stored
// in the per-lane chunk layout the bootstrapping keys use, and each TRGSW byte is
// read once.  4,096 products: split 92 us (5.1 TB/s; DRAM floor 72), FP64 99 us,
// shared 73 and 89; one warp per product, its row staged by bulk copies, took 131,
// 144, 99 and 116.  One product: 20 us, was 31.
#include "block_fft.cuh"
#include "extprod.cuh"

namespace cfdb {

namespace {

// 96 KB per TRGSW: 6 rows of 1,024 complex FP64, or 1,024 (hi, lo) FP32 pairs
constexpr uint32_t TRGSW_BYTES = 2 * L1 * 16384;

template <class P>
struct EpSmem {
    static constexpr int TAB_OFF = 64;
    static constexpr int BUF_OFF = TAB_OFF + ((int)sizeof(typename P::Tab) + 63) / 64 * 64;
    static constexpr int TOTAL = BUF_OFF + 2 * L1 * P::BUF * (int)sizeof(typename P::V);
};

template <class P, int NW, int OCC>
__global__ void __launch_bounds__(32 * NW, OCC) extprod1_kernel(ExtProdArgs a)
{
    using L = EpSmem<P>;
    using V = typename P::V;
    constexpr int BUF = P::BUF;
    static_assert(NW >= 2 * L1, "one warp per row");
    extern __shared__ __align__(128) unsigned char smem[];
    uint32_t *slot = reinterpret_cast<uint32_t *>(smem);
    typename P::Tab *T = reinterpret_cast<typename P::Tab *>(smem + L::TAB_OFF);
    V *buf = reinterpret_cast<V *>(smem + L::BUF_OFF);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // asks the TRLWE and the TRGSW of product p into L2
    auto prefetch = [&](int p) {
        if (tid != 0 || p >= a.B) return;
        bulk_prefetch_l2_if_aligned(a.trlwe + (size_t)p * 2 * N1, 2 * N1 * sizeof(uint32_t));
        if (!a.shared) bulk_prefetch_l2(reinterpret_cast<const unsigned char *>(a.trgsw) + (size_t)p * TRGSW_BYTES, TRGSW_BYTES);
    };
    prefetch(blockIdx.x);
    const float4 *tab = P::tables(a.tables);
    if (tid < (int)(sizeof(typename P::Tab) / 16)) reinterpret_cast<float4 *>(T)[tid] = tab[P::TAB_WORD4 + tid];
    if (warp == 0) tmem_alloc(slot, P::COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = *slot + ((32u * (warp & 3)) << 16);   // this sub-partition's lanes
    if (warp < 4) P::stage_tables(tm, *reinterpret_cast<const typename P::Full *>(tab), lane);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    for (int p = blockIdx.x; p < a.B; p += gridDim.x) {
        const uint32_t *in = a.trlwe + (size_t)p * 2 * N1;
        const float4 *g = reinterpret_cast<const float4 *>(a.trgsw) + (a.shared ? 0 : (size_t)p * (TRGSW_BYTES / 16)) + lane;
#pragma unroll
        for (int it = 0; it < (32 + NW - 1) / NW; ++it) {
            const int row = warp + NW * it;   // (polynomial, m2), m = lane + 32 m2
            if (row < 32) {
                const int pol = row >> 4, m = lane + 32 * (row & 15);
                put_digits<P>(buf + L1 * pol * BUF, m, in[pol * N1 + m], in[pol * N1 + m + 512]);
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
            if (warp + NW * it < 8) products<P>(buf, g, *T, warp + NW * it, lane);
        __syncthreads();
        prefetch(p + gridDim.x);
        uint32_t *o = a.out + (size_t)p * 2 * N1;
        if (warp < P::INV)
            P::inverse(buf + warp * BUF, buf + (warp ^ 1) * BUF, warp, lane, tm, [&](int m, uint32_t x) { o[m] = x; });
        __syncthreads();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(*slot, P::COLS);
    }
}

template <class P, int NW, int OCC>
cudaError_t launch_ep_t(const ExtProdArgs &a, cudaStream_t st)
{
    const int blocks = OCC * a.num_sms;
    extprod1_kernel<P, NW, OCC><<<a.B < blocks ? a.B : blocks, 32 * NW, EpSmem<P>::TOTAL, st>>>(a);
    return cudaGetLastError();
}

template <class P, int NW, int OCC>
cudaError_t init_ep_t()
{
    return cudaFuncSetAttribute(extprod1_kernel<P, NW, OCC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                EpSmem<P>::TOTAL);
}

}  // namespace

cudaError_t launch_extprod1(const ExtProdArgs &a, int precision, cudaStream_t st)
{
    if (a.B <= 0) return cudaSuccess;
    // warps per block and blocks per SM as in pbs01_ct.cu, except that more than
    // three split blocks per SM gain nothing where DRAM is the bound (us, 2 / 3 / 4
    // per SM: 700 products 27.6 / 28.7 / 36.1; 4,096: 91.4 / 91.8 / 94.8, with a
    // shared TRGSW 80.3 / 72.8 / 71.3)
    if (precision == 0)
        return a.B <= a.num_sms ? launch_ep_t<F64Path, 8, 2>(a, st) : launch_ep_t<F64Path, 6, 2>(a, st);
    return a.B <= 2 * a.num_sms ? launch_ep_t<PlainPath, 8, 2>(a, st) : launch_ep_t<PlainPath, 8, 3>(a, st);
}

cudaError_t init_extprod1()
{
    cudaError_t e = init_ep_t<PlainPath, 8, 2>();
    if (e == cudaSuccess) e = init_ep_t<PlainPath, 8, 3>();
    if (e == cudaSuccess) e = init_ep_t<F64Path, 8, 2>();
    if (e == cudaSuccess) e = init_ep_t<F64Path, 6, 2>();
    return e;
}

}  // namespace cfdb
