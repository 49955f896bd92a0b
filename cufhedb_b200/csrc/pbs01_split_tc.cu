// Batched lvl0 -> lvl1 programmable bootstrapping, split-precision FP32 path, with
// the first step of every digit transform on the tensor cores (tc_stage1.cuh):
// CUFHEDB_SPLIT32_TC.  The precision plan is the split path's (split_steps.cuh).
// One warp per ciphertext, W per persistent CTA; the key streams through a ring
// of shared-memory slots (ring.cuh) of one TRGSW row each, (hi, lo) float pairs
// in 16 KB.
#include "fft_f32.cuh"
#include "pbs_common.cuh"
#include "ring.cuh"
#include "split_steps.cuh"
#include "tc_stage1.cuh"

#include <type_traits>

namespace cfdb {

template <int W, int S, int TBYTES>
struct Pbs01SplitSmem {
    static constexpr int RING_OFF = RING_HEADER_BYTES;
    static constexpr int CHUNK_BYTES = 16384;   // 16 slots x 2 outputs x 32 lanes x float4(hi, lo)
    static constexpr int TAB_OFF = RING_OFF + S * CHUNK_BYTES;
    static constexpr int WARP_OFF = TAB_OFF + (TBYTES + 127) / 128 * 128;
    static constexpr int XP_BYTES = FFT512_XP * 8;
    static constexpr int ACC_BYTES = 2 * N1 * 4;
    static constexpr int ABAR_BYTES = ((N0 * 2) + 127) / 128 * 128;
    static constexpr int PER_WARP = XP_BYTES + ACC_BYTES + ABAR_BYTES;
    // the two FP16 limbs of B, one mbarrier per warp, the tensor-memory base
    // address
    static constexpr int TC_OFF = (WARP_OFF + W * PER_WARP + 1023) / 1024 * 1024;
    static constexpr int TC_B_BYTES = 2 * TC_B_HALVES * 2;
    static constexpr int TC_BAR_OFF = TC_OFF + TC_B_BYTES;
    static constexpr int TC_SLOT_OFF = TC_BAR_OFF + 8 * 16;
    static constexpr int TOTAL_TC = TC_SLOT_OFF + 16;
};

// Tensor-core stage 1 (tc_stage1.cuh), shared by the warps of a group of
// four (warps 0-3 and 4-7; a producer warp takes no part), one polynomial at
// a time: when a polynomial's decomposition words are formed, each warp
// writes the A rows of all three of its digit polynomials into its own
// sub-partition's lanes of the group's A columns (the words are dead right
// after), the group meets at a named barrier, and one lane of the group's
// first warp issues the polynomial's three M = 128 products into three of the
// group's six D buffers and commits them to the polynomial's mbarrier.
// Polynomial 0's products are issued at the start of a CMux and taken at
// digit 0; polynomial 1's are issued at digit 1 (A is free again: every
// warp waited for polynomial 0's products at digit 0) and run under the
// transforms of digits 1 and 2.  Per group (256 columns): D 6 x 32 columns
// first, each on a 32-column boundary, then A 3 x 16.
// Every warp takes part in every step, active or not (a warp whose rotation
// is 0 for this CMux writes no rows and reads no result), so the barriers and
// the buffer reuse stay in step.  Addresses are recomputed from the block's
// shared memory and the warp index at each use (the kernel runs at the
// 255-register limit).
constexpr uint32_t TC_D_COLS = 6 * 32, TC_GROUP_COLS = 256;   // D at [0, 192), A at [192, 240)

template <class L, int W>
struct TcStage {
    unsigned char *smem;
    uint32_t phase;     // per polynomial (bits 0, 1): parity of its next completion

    __device__ __forceinline__ static int group(int warp) { return warp >> 2; }
    __device__ __forceinline__ uint32_t tbase() const
    {
        return *reinterpret_cast<const volatile uint32_t *>(smem + L::TC_SLOT_OFF);
    }
    __device__ __forceinline__ uint32_t lanes(int warp) const
    {
        return tbase() + TC_GROUP_COLS * group(warp) + ((32u * (warp & 3)) << 16);
    }
    __device__ __forceinline__ uint64_t *bar(int warp, int poly) const
    {
        return reinterpret_cast<uint64_t *>(smem + L::TC_BAR_OFF) + 2 * group(warp) + poly;
    }
    // A(d) <- the digit-d row of this lane, d < 3 (only when active), then the
    // group meets and its first warp issues D(3 poly + d) = A(d) (Bhi + Blo)
    __device__ __forceinline__ void put_issue(const uint32_t *w, bool active, int poly, int warp, int lane)
    {
        if (active) {
#pragma unroll 1
            for (int d = 0; d < L1; ++d) {
                uint32_t a[16];
                tc_a_row(a, w, d);
                tmem_st16(lanes(warp) + TC_D_COLS + 16 * d, a);
            }
            tmem_wait_st();
        }
        tc_fence_before();
        if (group(warp) == 0) asm volatile("bar.sync 2, %0;" ::"n"(32 * (W < 4 ? W : 4)) : "memory");
        else asm volatile("bar.sync 3, %0;" ::"n"(32 * (W > 4 ? W - 4 : 1)) : "memory");
        if ((warp & 3) == 0 && lane == 0) {
            tc_fence_after();
            const uint32_t gcol = tbase() + TC_GROUP_COLS * group(warp);
            const uint32_t b = smem_u32(smem + L::TC_OFF), limb = TC_B_HALVES * 2, kstep = 2 * TC_B_LBO;
#pragma unroll
            for (int d = 0; d < L1; ++d) {
                const uint32_t a = gcol + TC_D_COLS + 16 * d, dcol = gcol + 32 * (L1 * poly + d);
                umma_ts(dcol, a, tc_smem_desc(b, TC_B_LBO, TC_B_SBO), 0);
                umma_ts(dcol, a + 8, tc_smem_desc(b + kstep, TC_B_LBO, TC_B_SBO), 1);
                umma_ts(dcol, a, tc_smem_desc(b + limb, TC_B_LBO, TC_B_SBO), 1);
                umma_ts(dcol, a + 8, tc_smem_desc(b + limb + kstep, TC_B_LBO, TC_B_SBO), 1);
            }
            umma_commit(bar(warp, poly));
        }
        __syncwarp();
    }
    // waits for a polynomial's three products
    __device__ __forceinline__ void wait(int poly, int warp, int *err)
    {
        if (!mbar_wait(bar(warp, poly), (phase >> poly) & 1)) report_error(err, DEV_TIMEOUT_MMA);
        phase ^= 1u << poly;
        tc_fence_after();
    }
    // this lane's row of digit polynomial r's product (only when active):
    // v[q] = X[q]
    __device__ __forceinline__ void take(float2 v[16], bool active, int r, int warp)
    {
        if (active) {
            uint32_t x[32];
            tmem_ld32(lanes(warp) + 32 * r, x);
#pragma unroll
            for (int q = 0; q < 16; ++q) v[q] = make_float2(__uint_as_float(x[q]), __uint_as_float(x[16 + q]));
        }
        tc_fence_before();
        __syncwarp();
    }
};

template <int W>
constexpr uint32_t tc_cols()
{
    return ((W + 3) / 4) * TC_GROUP_COLS <= 256 ? 256u : 512u;
}
static_assert(2 * TC_GROUP_COLS <= 512 && TC_D_COLS + 3 * 16 <= TC_GROUP_COLS,
              "two groups' columns within one SM's tensor memory");

// W consumer warps, plus a producer warp when PRODUCER (ring.cuh has both
// feeds; the launch picks per shape, see launch_pbs01_split_tc)
template <int W, int S, bool PRODUCER>
__global__ void __launch_bounds__((W + (PRODUCER ? 1 : 0)) * 32, 1) pbs01_split_tc_kernel(Pbs01Args a)
{
    // the folded tables (fft_f32.cuh): the twist and untwist ride on the
    // stage-1 twiddles, so the kernel reads 12.3 KB of tables instead of 24.4
    using TT = Fft512TablesFold;
    using L = Pbs01SplitSmem<W, S, (int)sizeof(TT)>;
    extern __shared__ __align__(128) unsigned char smem[];
    TT *T = reinterpret_cast<TT *>(smem + L::TAB_OFF);
    const int ngroups = (a.B + W - 1) / W;
    constexpr int CHUNKS = N0 * 2 * L1;
    using Feed = std::conditional_t<PRODUCER, ProducerRing<S, L::CHUNK_BYTES, W>, KeyRing<S, L::CHUNK_BYTES, W>>;
    Feed ring{reinterpret_cast<RingHeader *>(smem), smem + L::RING_OFF, reinterpret_cast<const unsigned char *>(a.bk),
              (uint32_t)CHUNKS, (uint32_t)groups_of_block(ngroups, blockIdx.x, gridDim.x) * CHUNKS};

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint64_t *tc_bars = reinterpret_cast<uint64_t *>(smem + L::TC_BAR_OFF);
    uint32_t *tc_slot = reinterpret_cast<uint32_t *>(smem + L::TC_SLOT_OFF);
    if (threadIdx.x == 0) {
        ring.init_by_thread0();
        for (int k = 0; k < 4; ++k) mbar_init(&tc_bars[k], 1);   // 2 groups x 2 buffers
        fence_barrier_init();
    }
    if (warp == 0) tmem_alloc(tc_slot, tc_cols<W>());
    {
        const Fft512TablesF *all = reinterpret_cast<const Fft512TablesF *>(a.tables);
        const float4 *src = reinterpret_cast<const float4 *>(&all->fold);
        float4 *dst = reinterpret_cast<float4 *>(T);
        for (int i = threadIdx.x; i < (int)(sizeof(TT) / 16); i += blockDim.x) dst[i] = src[i];
        const float4 *bs = reinterpret_cast<const float4 *>(&all->tc_b[0][0]);
        float4 *bd = reinterpret_cast<float4 *>(smem + L::TC_OFF);
        for (int i = threadIdx.x; i < L::TC_B_BYTES / 16; i += blockDim.x) bd[i] = bs[i];
        fence_proxy_async_smem();   // B is read by the tensor cores (async proxy)
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if constexpr (PRODUCER) {
        if (warp == W) {
            ring.run_producer(lane, a.err);
            return;
        }
    } else {
        if (threadIdx.x == 0) ring.prologue_by_thread0();
    }

    TcStage<L, W> tc{smem, 0u};

    unsigned char *wb = smem + L::WARP_OFF + warp * L::PER_WARP;
    unsigned long long *xp = reinterpret_cast<unsigned long long *>(wb);
    uint32_t *acc = reinterpret_cast<uint32_t *>(wb + L::XP_BYTES);
    uint16_t *abar_s = reinterpret_cast<uint16_t *>(wb + L::XP_BYTES + L::ACC_BYTES);

    uint32_t c = 0;
    for (int g = blockIdx.x; g < ngroups; g += gridDim.x) {
        const int ct = g * W + warp;
        const bool valid = ct < a.B;
        uint32_t bbar = 2 * N1;
        if (valid) {
            const uint32_t *in = a.in + (size_t)ct * (N0 + 1);
            for (int i = lane; i < N0; i += 32) abar_s[i] = (uint16_t)((in[i] + (1u << 20)) >> 21);
            bbar = 2 * N1 - (in[N0] >> 21);
        }
        for (int j = lane; j < N1; j += 32) {
            acc[j] = 0;
            acc[N1 + j] = testvec_rot1(a.tv, j, bbar);
        }
        __syncwarp();
        {
            // polynomial 0's products of CMux 0; those of every later CMux are
            // issued between the previous CMux's two inverse transforms
            const uint32_t ab0 = valid ? abar_s[0] : 0u;
            uint32_t w0[32];
            if (ab0) digit_words1(w0, acc, ab0, lane);
            tc.put_issue(w0, ab0 != 0, 0, warp, lane);
        }

        for (int i = 0; i < N0; ++i) {
            const uint32_t ab = valid ? abar_s[i] : 0u;
            const bool active = ab != 0;
            CP f0[16], f1[16];
            uint32_t w[32];
#pragma unroll 1
            for (int r = 0; r < 2 * L1; ++r, ++c) {
                float2 v[16];
                if (r == 1) {
                    // polynomial 1's products, under the transforms of
                    // digits 1 and 2
                    if (active) digit_words1(w, acc + N1, ab, lane);
                    tc.put_issue(w, active, 1, warp, lane);
                }
                if (r % L1 == 0) tc.wait(r / L1, warp, a.err);
                tc.take(v, active, r, warp);
                const float4 *bkc = reinterpret_cast<const float4 *>(ring.acquire(c, a.err));
                if (active) {
                    ffft512_fwd_tw_rest(v, reinterpret_cast<float2 *>(xp), *T, lane);
                    if (r == 0) {
#pragma unroll
                        for (int s = 0; s < 16; ++s) {
                            const float4 k0 = bkc[(2 * s) * 32 + lane], k1 = bkc[(2 * s + 1) * 32 + lane];
                            const unsigned long long vr = pk2(v[s].x, v[s].x), vi = pk2(v[s].y, v[s].y),
                                                     nvi = pk2(-v[s].y, -v[s].y);
                            f0[s] = pmul_first(vr, vi, nvi, k0);
                            f1[s] = pmul_first(vr, vi, nvi, k1);
                        }
                    } else {
#pragma unroll
                        for (int s = 0; s < 16; ++s) {
                            const float4 k0 = bkc[(2 * s) * 32 + lane], k1 = bkc[(2 * s + 1) * 32 + lane];
                            const unsigned long long vr = pk2(v[s].x, v[s].x), vi = pk2(v[s].y, v[s].y),
                                                     nvi = pk2(-v[s].y, -v[s].y);
                            pmac(f0[s], vr, vi, nvi, k0);
                            pmac(f1[s], vr, vi, nvi, k1);
                        }
                    }
                }
                ring.release(c, lane);
            }
            if (active) {
                add_inverse_split(acc, f0, xp, lane, *T);
                __syncwarp();
            }
            if (i + 1 < N0) {
                // the next CMux's polynomial 0 is final here: its products
                // run under this CMux's second inverse transform
                const uint32_t abn = valid ? abar_s[i + 1] : 0u;
                if (abn) digit_words1(w, acc, abn, lane);
                tc.put_issue(w, abn != 0, 0, warp, lane);
            }
            if (active) {
                add_inverse_split(acc + N1, f1, xp, lane, *T);
                __syncwarp();
            }
        }
        if (valid) {
            uint32_t *o = a.out + (size_t)ct * (N1 + 1);
            for (int j = lane; j < N1; j += 32) o[j] = j == 0 ? acc[0] : (uint32_t)(0u - acc[N1 - j]);
            if (lane == 0) o[N1] = acc[N1] + a.out_b_add;
        }
        __syncwarp();
    }
    // every product of every warp was waited for; then the columns are freed
    tc_fence_before();
    asm volatile("bar.sync 1, %0;" ::"r"(W * 32) : "memory");
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(*tc_slot, tc_cols<W>());
    }
    if constexpr (!PRODUCER) {
        __syncthreads();
        if (threadIdx.x == 0) ring.drain_by_thread0(a.err);
    }
}

// key-ring depth: 7 slots with 7 (or 4) ciphertexts per CTA (more than one
// CMux of key rows in flight), 6 with 8 (shared memory)
template <int W>
constexpr int PBS01S_S = W == 8 ? 6 : 7;

template <int W>
using SplitLayout = Pbs01SplitSmem<W, PBS01S_S<W>, (int)sizeof(Fft512TablesFold)>;

// 7 and 4 ciphertexts per CTA run with a producer warp (8 or 5 warps), 8 per
// CTA without one (8 warps): at most 2 warps per SM sub-partition (up to 255
// registers); 4 per CTA leaves one consumer warp per sub-partition
template <int W>
constexpr bool PBS01S_PROD = W != 8;

template <int W>
static cudaError_t launch_pbs01_split_tc_t(const Pbs01Args &a, int grid, cudaStream_t st)
{
    constexpr bool PROD = PBS01S_PROD<W>;
    static_assert(SplitLayout<W>::TOTAL_TC <= 227 * 1024, "shared memory budget");
    pbs01_split_tc_kernel<W, PBS01S_S<W>, PROD>
        <<<grid, (W + (PROD ? 1 : 0)) * 32, SplitLayout<W>::TOTAL_TC, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_pbs01_split_tc(const Pbs01Args &a, int num_sms, int w, cudaStream_t st)
{
    if (a.B <= 0) return cudaSuccess;
    const int groups = (a.B + w - 1) / w;
    const int grid = groups < num_sms ? groups : num_sms;
    if (w == 7) return launch_pbs01_split_tc_t<7>(a, grid, st);
    if (w == 8) return launch_pbs01_split_tc_t<8>(a, grid, st);
    if (w == 4) return launch_pbs01_split_tc_t<4>(a, grid, st);
    return cudaErrorInvalidValue;
}

template <int W>
static cudaError_t init_pbs01_split_tc_t()
{
    return cudaFuncSetAttribute(pbs01_split_tc_kernel<W, PBS01S_S<W>, PBS01S_PROD<W>>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, SplitLayout<W>::TOTAL_TC);
}

cudaError_t init_pbs01_split_tc()
{
    cudaError_t e = init_pbs01_split_tc_t<7>();
    if (e == cudaSuccess) e = init_pbs01_split_tc_t<8>();
    if (e == cudaSuccess) e = init_pbs01_split_tc_t<4>();
    return e;
}

}  // namespace cfdb
