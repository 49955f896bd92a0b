// Batched lvl0 -> lvl2 programmable bootstrapping (GateBootstrappingTLWE2TLWEFFT
// <lvl02param>, thirdparty/TFHEpp/src/gatebootstrapping.cpp:14-23, BlindRotate
// at include/gatebootstrapping.hpp:15-43 with domain lvl0, target lvl2: bbar =
// 2N - (b >> 20), abar_i = (a_i + 2^19) >> 20).
//
// Two kernels: pbs02_team_kernel for batches of a few ciphertexts per SM, and
// pbs02_block_kernel (below) for larger ones.
//
// One persistent CTA per SM holds C = 1 or 2 ciphertexts and four teams of 128
// threads (8 of the 1,024 points each, fft8x.cuh), 16 warps in all; the teams of
// a ciphertext (4 or 2) divide every CMux:
//   words     the decomposition words of both polynomials, half a polynomial
//             or a whole one per team;
//   transform in rounds (2 of 4 rows, or 4 of 2 rows), each team transforms one
//             digit polynomial;
//   products  a team takes its share of the frequency slots (2 or 4 of 8) of
//             the round's rows into both outputs' accumulators, in registers;
//   inverse   one team per output.
// Thread u of every team sits in the same lane of the same SM sub-partition
// (four warps per team), so words, spectra and accumulators pass between teams
// through tensor memory (tmem_exchange.cuh) and shared memory keeps only the
// accumulators, the transposes and the key.  With C = 2 the two ciphertexts
// share nothing but the key stage, so one's transforms run under the other's
// products and conversions.
//
// What bounds it: per ciphertext and CMux about 10,300 shared-memory wavefronts
// (half of them the two transposes of each transform), 8,000 FP64-pipe cycles
// and 8,000 issue slots per scheduler; at C = 2 the wavefronts run at 65 % of
// their rate and FP64 at 49 %, the rest is the barriers and the latency between
// the stages.  Pass times on a B200 (148 SMs): C = 1 5.72 ms, C = 2 10.89 ms,
// where one team per ciphertext with both accumulators in its registers took
// 10.26, 13.80 and, with three ciphertexts, 17.65 ms (the shape-3 launch here,
// passes of two and of one: 16.6 ms).  On the way: all teams of both
// ciphertexts in lock step 12.28 ms; key chunks released by 16 warps with an
// atomic each 8.49 ms at C = 1, by a producer warp (which costs the others
// their registers) 7.06 ms; one release per team and round 6.20 ms; each thread's
// values loaded into its registers, ahead of the barrier, 5.72 ms.
#include "lvl2_steps.cuh"
#include "ring.cuh"
#include "tc_stage1.cuh"
#include "tmem_exchange.cuh"

namespace cfdb {

namespace {

constexpr int TEAMS = 4;

// C ciphertexts per CTA, TPC teams each: a round is TPC rows of each
// ciphertext (both outputs' chunks), SL frequency slots per thread in the
// products
template <int C>
struct TeamShape {
    static constexpr int TPC = TEAMS / C;
    static constexpr int ROUNDS = 2 * L2 / TPC;
    static constexpr int SL = 8 / TPC;
    static constexpr int CHUNK = 16384;                 // one (row, output): 1024 complex
    static constexpr int CHUNKS = 2 * TPC;              // per round
    // two ciphertexts share the round's key in shared memory; one reads it into
    // registers
    static constexpr bool STAGED = C == 2;
    static constexpr uint32_t BYTES = STAGED ? CHUNKS * CHUNK : 0;
    using Key = RoundKey<BYTES, TEAMS>;
    static constexpr int KEY_OFF = 128;
    static constexpr int TAB_OFF = KEY_OFF + (int)BYTES;
    static constexpr int XP_OFF = TAB_OFF + ((int)sizeof(Fft1024Tables) + 127) / 128 * 128;
    static constexpr int XP_BYTES = FFT8X_XP<T2> * 16;
    static constexpr int ACC_OFF = XP_OFF + TEAMS * XP_BYTES;
    static constexpr int ACC_BYTES = 2 * N2 * 8;
    static constexpr int TOTAL = ACC_OFF + C * ACC_BYTES;
    static_assert(TOTAL <= 227 * 1024, "shared memory budget");
};

// tensor-memory columns (of every lane; a double is two columns)
constexpr uint32_t TT_SPEC = 0;      // [round parity 2][team 4][slot 8][re im]
constexpr uint32_t TT_WORDS = 256;   // [ciphertext][polynomial 2][16 words]
constexpr uint32_t TT_ACC = 384;     // [ciphertext][output 2][slot 8][re im]

__device__ __forceinline__ void put_c(uint32_t *x, double2 z)
{
    x[0] = (uint32_t)__double2loint(z.x);
    x[1] = (uint32_t)__double2hiint(z.x);
    x[2] = (uint32_t)__double2loint(z.y);
    x[3] = (uint32_t)__double2hiint(z.y);
}
__device__ __forceinline__ double2 get_c(const uint32_t *x)
{
    return make_double2(__hiloint2double((int)x[1], (int)x[0]), __hiloint2double((int)x[3], (int)x[2]));
}

// a read-only load issued where it stands
__device__ __forceinline__ float4 ldg_here(const float4 *p)
{
    float4 v;
    asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "l"(p));
    return v;
}

// the teams of a ciphertext meet; tensor-memory stores before it (waited for)
// are visible to loads after it
template <int C>
__device__ __forceinline__ void ct_sync(int q)
{
    tc_fence_before();
    asm volatile("bar.sync %0, %1;" ::"r"(1 + TEAMS + q), "n"(TEAMS * T2 / C) : "memory");
    tc_fence_after();
}

template <int C>
__global__ void __launch_bounds__(TEAMS * T2, 1) pbs02_team_kernel(Pbs02Args a)
{
    using S = TeamShape<C>;
    constexpr int TPC = S::TPC, SL = S::SL, ROUNDS = S::ROUNDS;
    extern __shared__ __align__(128) unsigned char smem[];
    Fft1024Tables *T = reinterpret_cast<Fft1024Tables *>(smem + S::TAB_OFF);
    const int ngroups = (a.B + C - 1) / C;
    typename S::Key key{smem, smem + S::KEY_OFF, reinterpret_cast<const unsigned char *>(a.bk), N0 * ROUNDS,
                        (uint32_t)groups_of_block(ngroups, blockIdx.x, gridDim.x) * N0 * ROUNDS};
    uint32_t *slot = reinterpret_cast<uint32_t *>(smem + 64);

    const int warp = threadIdx.x >> 5;
    const int team = threadIdx.x / T2, t = threadIdx.x % T2, bar = 1 + team;
    const int q = team / TPC, h = team % TPC;   // the ciphertext, and the team's place in it
    if (S::STAGED && threadIdx.x == 0) key.init();
    if (warp == 0) tmem_alloc(slot, 512);
    {
        const double2 *src = reinterpret_cast<const double2 *>(a.tables);
        double2 *dst = reinterpret_cast<double2 *>(T);
        for (int i = threadIdx.x; i < (int)(sizeof(Fft1024Tables) / 16); i += blockDim.x) dst[i] = src[i];
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (S::STAGED && threadIdx.x == 0) key.issue(0);
    const uint32_t tm = *slot + ((32u * (warp & 3)) << 16);

    double2 *xp = reinterpret_cast<double2 *>(smem + S::XP_OFF + team * S::XP_BYTES);
    uint64_t *acc = reinterpret_cast<uint64_t *>(smem + S::ACC_OFF + q * S::ACC_BYTES);

    uint32_t n = 0;   // running number of the round
    for (int g = blockIdx.x; g < ngroups; g += gridDim.x) {
        const int ct = g * C + q;
        const bool valid = ct < a.B;
        const uint32_t *in = a.in + (size_t)(valid ? ct : 0) * (N0 + 1);
        uint32_t an = in[0];   // the next CMux's mask word, read one CMux ahead
        if (h == 0) {
            for (int m = t; m < N2; m += T2) acc[m] = 0;
        } else if (h == 1) {
            const uint32_t bbar = 2 * N2 - (in[N0] >> 20);
            for (int m = t; m < N2; m += T2) acc[N2 + m] = testvec_rot2(a.tv, m, bbar);
        }
        ct_sync<C>(q);

        for (int i = 0; i < N0; ++i) {
            const uint32_t ab = valid ? (an + (1u << 19)) >> 20 : 0u;
            an = in[i + 1];
            if (ab == 0) {
                if constexpr (S::STAGED) {
                    // One thread takes part in the skipped rounds for its team, which
                    // does not read them: a warp that waited here as well could be held
                    // up while the rounds run on, and would then meet the parity of a
                    // later one.  The others' next acquire follows a ct_sync with this
                    // thread, and their round cannot be replaced before they release it.
                    if (t == 0)
                        for (int k = 0; k < ROUNDS; ++k) {
                            key.acquire(n + k, a.err);
                            key.release(n + k);
                        }
                    __syncwarp();
                    n += ROUNDS;
                }
                continue;
            }
            {
                // the decomposition words of polynomial h % 2: all 16 with two
                // teams per ciphertext, one half of them with four
                constexpr int NW = C == 2 ? 8 : 4;
                const int j0 = C == 2 ? 0 : 4 * (h >> 1);
                const uint64_t *poly = acc + (h & 1) * N2;
                uint32_t x[4 * NW];
#pragma unroll
                for (int j = 0; j < NW; ++j) {
                    uint64_t w0, w1;
                    digit_word_pair2<true>(w0, w1, poly, ab, t + T2 * (j0 + j));
                    x[4 * j] = (uint32_t)w0;
                    x[4 * j + 1] = (uint32_t)(w0 >> 32);
                    x[4 * j + 2] = (uint32_t)w1;
                    x[4 * j + 3] = (uint32_t)(w1 >> 32);
                }
                const uint32_t col = tm + TT_WORDS + 64 * q + 32 * (h & 1);
                if constexpr (C == 2) tmem_st32_nowait(col, x);
                else tmem_st16_nowait(col + 4 * j0, x);
                tmem_wait_st();
            }
            ct_sync<C>(q);
            double2 f[2][SL];   // [output][slot SL h + s]
#pragma unroll 1
            for (int k = 0; k < ROUNDS; ++k, ++n) {
                {
                    const int r = TPC * k + h;
                    uint32_t x[32];
                    tmem_ld32_nowait(tm + TT_WORDS + 64 * q + 32 * (r / L2), x);
                    tmem_wait_ld();
                    tmem_landed<32>(x);
                    uint64_t w[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) w[j] = ((uint64_t)x[2 * j + 1] << 32) | x[2 * j];
                    double2 v[8];
                    digits2(v, w, r % L2);
                    // every thread of the team is past its products of the
                    // round before when it reaches the transform's first barrier
                    fft8x_fwd<double2, T2>(v, xp, *T, t, bar, [&] {
                        if (S::STAGED && k > 0 && t == 0) key.release(n - 1);
                    });
#pragma unroll
                    for (int s = 0; s < 8; ++s) put_c(x + 4 * s, v[s]);
                    tmem_st32_nowait(tm + TT_SPEC + 128 * (k & 1) + 32 * team, x);
                    tmem_wait_st();
                }
                // chunk e of the round: row TPC k + e / 2, output e % 2; this
                // thread's values at [slot][t].  Read into registers they are
                // asked for before the barrier, so the memory's latency runs
                // under the wait for the slowest team.
                float4 kr[S::STAGED ? 1 : S::CHUNKS][SL];
                if constexpr (!S::STAGED) {
                    const float4 *kg = reinterpret_cast<const float4 *>(a.bk) +
                                       ((size_t)(i * ROUNDS + k) * S::CHUNKS) * 1024 + SL * h * T2 + t;
#pragma unroll
                    for (int e = 0; e < S::CHUNKS; ++e)
#pragma unroll
                        for (int s = 0; s < SL; ++s) kr[e][s] = ldg_here(kg + e * 1024 + s * T2);
                }
                ct_sync<C>(q);
                if constexpr (S::STAGED) key.acquire(n, a.err);
                const double2 *ks = reinterpret_cast<const double2 *>(smem + S::KEY_OFF) + SL * h * T2 + t;
#pragma unroll
                for (int rr = 0; rr < TPC; ++rr) {
                    uint32_t y[4 * SL];
                    const uint32_t col = tm + TT_SPEC + 128 * (k & 1) + 32 * (TPC * q + rr) + 4 * SL * h;
                    if constexpr (SL == 4) tmem_ld16_nowait(col, y);
                    else tmem_ld8_nowait(col, y);
                    tmem_wait_ld();
                    tmem_landed<4 * SL>(y);
#pragma unroll
                    for (int o = 0; o < 2; ++o) {
                        const int e = 2 * rr + o;
#pragma unroll
                        for (int s = 0; s < SL; ++s) {
                            double2 kv;
                            if constexpr (S::STAGED) kv = ks[e * 1024 + s * T2];
                            else kv = *reinterpret_cast<const double2 *>(&kr[e][s]);
                            const double2 v = get_c(y + 4 * s);
                            if (k == 0 && rr == 0) f[o][s] = cx_mul(v, kv);
                            else cx_fma(f[o][s], v, kv);
                        }
                    }
                }
            }
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                uint32_t x[4 * SL];
#pragma unroll
                for (int s = 0; s < SL; ++s) put_c(x + 4 * s, f[o][s]);
                const uint32_t col = tm + TT_ACC + 64 * q + 32 * o + 4 * SL * h;
                if constexpr (SL == 4) tmem_st16_nowait(col, x);
                else tmem_st8_nowait(col, x);
            }
            tmem_wait_st();
            ct_sync<C>(q);
            if (S::STAGED && t == 0) key.release(n - 1);
            if (h < 2) {
                uint32_t x[32];
                tmem_ld32_nowait(tm + TT_ACC + 64 * q + 32 * h, x);
                tmem_wait_ld();
                tmem_landed<32>(x);
                double2 v[8];
#pragma unroll
                for (int s = 0; s < 8; ++s) v[s] = get_c(x + 4 * s);
                fft8x_inv<double2, T2>(v, xp, *T, t, bar);
                add_inverse2(acc + h * N2, v, t);
            }
            ct_sync<C>(q);
        }
        ct_sync<C>(q);   // a row may be bootstrapped over itself, and skipped CMuxes have no barrier
        if (valid) {
            uint64_t *o = a.out + (size_t)ct * (N2 + 1);
            for (int m = t + h * T2; m < N2; m += TPC * T2) o[m] = m == 0 ? acc[0] : 0ull - acc[N2 - m];
            if (h == 0 && t == 0) o[N2] = acc[N2] + a.out_b_add;
        }
        ct_sync<C>(q);
    }
    tc_fence_before();
    __syncthreads();
    if (S::STAGED && threadIdx.x == 0) key.drain(a.err);
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(*slot, 512);
    }
}

// ---- one team per ciphertext and block ---------------------------------------------
// For batches that fill the SMs many times over: four blocks of four warps per SM,
// out of step, where the teams of one block wait for one another.  The team does
// all rows of a CMux itself; its digits' words, its accumulators and its twiddle
// steps are in tensor memory, the key's values come from L2 into registers, asked
// for in the middle of the transform before their products.  Shared memory holds
// the accumulator polynomials and the transpose.  Bound by the transposes and
// FP64 latency: L1 data pipe at 61 %, FP64 at 50 %, issue 53 % (1,184).  ms per
// 2,048: 72.4, two ciphertexts per persistent CTA 76.0; key asked for after the
// transform 79.3, twiddle steps in shared memory 73.1, three blocks of 144
// registers 73.6 (four have 128 and spill 68 bytes), two teams per block and three
// blocks 80.1.
struct BlockSmem {
    static constexpr int XP_OFF = 16;
    static constexpr int ACC_OFF = XP_OFF + FFT8X_XP<T2> * 16;
    static constexpr int TOTAL = ACC_OFF + 2 * N2 * 8;
};
static_assert(BlockSmem::XP_OFF % 16 == 0 && 4 * (BlockSmem::TOTAL + 1024) <= 228 * 1024, "four blocks per SM");
constexpr uint32_t BT_ACC = 0;       // [output 2][slot 8][re im]
constexpr uint32_t BT_WORDS = 64;    // [16 words] of the polynomial in work
constexpr uint32_t BT_TAB = 96;      // twA0, twAs and twB1 of this thread
constexpr uint32_t BT_COLS = 128;    // of 512 per SM

__device__ __forceinline__ void tmem_ld4_nowait(uint32_t taddr, uint32_t *v)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                 : "r"(taddr)
                 : "memory");
}
struct TmemTables {
    uint32_t tm;
    __device__ __forceinline__ void stage_a(int, double2 &a0, double2 &as) const
    {
        uint32_t x[8];
        tmem_ld8_nowait(tm, x);
        tmem_wait_ld();
        tmem_landed<8>(x);
        a0 = get_c(x);
        as = get_c(x + 4);
    }
    __device__ __forceinline__ double2 stage_b(int) const
    {
        uint32_t x[4];
        tmem_ld4_nowait(tm + 8, x);
        tmem_wait_ld();
        tmem_landed<4>(x);
        return get_c(x);
    }
};

__global__ void __launch_bounds__(T2, 4) pbs02_block_kernel(Pbs02Args a)
{
    using S = BlockSmem;
    extern __shared__ __align__(128) unsigned char smem[];
    uint32_t *slot = reinterpret_cast<uint32_t *>(smem);
    double2 *xp = reinterpret_cast<double2 *>(smem + S::XP_OFF);
    uint64_t *acc = reinterpret_cast<uint64_t *>(smem + S::ACC_OFF);
    const int t = threadIdx.x, warp = t >> 5, bar = 1;
    if (warp == 0) tmem_alloc(slot, BT_COLS);
    const uint32_t *in = a.in + (size_t)blockIdx.x * (N0 + 1);
    uint32_t an = in[0];   // the next CMux's mask word, read one CMux ahead
    {
        const uint32_t bbar = 2 * N2 - (in[N0] >> 20);
        for (int m = t; m < N2; m += T2) {
            acc[m] = 0;
            acc[N2 + m] = testvec_rot2(a.tv, m, bbar);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = *slot + ((32u * warp) << 16);
    const TmemTables T{tm + BT_TAB};
    {
        const Fft1024Tables *src = reinterpret_cast<const Fft1024Tables *>(a.tables);
        uint32_t x[16];
        put_c(x, src->twA0[t]);
        put_c(x + 4, src->twAs[t]);
        put_c(x + 8, src->twB1[t & 15]);
        put_c(x + 12, src->twB1[t & 15]);
        tmem_st16_nowait(tm + BT_TAB, x);
        tmem_wait_st();
    }

    // the key: row r, output o, slot s of this thread at [(2 r + o) 1024 + 128 s]
    const float4 *kg = reinterpret_cast<const float4 *>(a.bk) + t;
    for (int i = 0; i < N0; ++i, kg += 2 * L2 * 2 * 1024) {
        const uint32_t ab = (an + (1u << 19)) >> 20;
        an = in[i + 1];
        if (ab == 0) continue;
#pragma unroll 1
        for (int r = 0; r < 2 * L2; ++r) {
            uint32_t x[32];
            uint64_t w[16];
            if (r % L2 == 0) {
                digit_words2<true>(w, acc + (r / L2) * N2, ab, t);
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    x[2 * j] = (uint32_t)w[j];
                    x[2 * j + 1] = (uint32_t)(w[j] >> 32);
                }
                tmem_st32_nowait(tm + BT_WORDS, x);
                tmem_wait_st();
            } else {
                tmem_ld32_nowait(tm + BT_WORDS, x);
                tmem_wait_ld();
                tmem_landed<32>(x);
#pragma unroll
                for (int j = 0; j < 16; ++j) w[j] = ((uint64_t)x[2 * j + 1] << 32) | x[2 * j];
            }
            double2 v[8];
            digits2(v, w, r % L2);
            float4 kv[8];
            fft8x_fwd<double2, T2>(v, xp, T, t, bar, [&] {
#pragma unroll
                for (int s = 0; s < 8; ++s) kv[s] = ldg_here(kg + 2 * r * 1024 + s * T2);
            });
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                double2 f[8];
                if (r > 0) {
                    tmem_ld32_nowait(tm + BT_ACC + 32 * o, x);
                    tmem_wait_ld();
                    tmem_landed<32>(x);
#pragma unroll
                    for (int s = 0; s < 8; ++s) {
                        f[s] = get_c(x + 4 * s);
                        cx_fma(f[s], v[s], *reinterpret_cast<const double2 *>(&kv[s]));
                    }
                } else {
#pragma unroll
                    for (int s = 0; s < 8; ++s) f[s] = cx_mul(v[s], *reinterpret_cast<const double2 *>(&kv[s]));
                }
                if (o == 0) {
#pragma unroll
                    for (int s = 0; s < 8; ++s) kv[s] = ldg_here(kg + (2 * r + 1) * 1024 + s * T2);
                }
#pragma unroll
                for (int s = 0; s < 8; ++s) put_c(x + 4 * s, f[s]);
                tmem_st32_nowait(tm + BT_ACC + 32 * o, x);
            }
            tmem_wait_st();
        }
#pragma unroll 1
        for (int o = 0; o < 2; ++o) {
            uint32_t x[32];
            tmem_ld32_nowait(tm + BT_ACC + 32 * o, x);
            tmem_wait_ld();
            tmem_landed<32>(x);
            double2 v[8];
#pragma unroll
            for (int s = 0; s < 8; ++s) v[s] = get_c(x + 4 * s);
            fft8x_inv<double2, T2>(v, xp, T, t, bar);
            add_inverse2(acc + o * N2, v, t);
        }
        group_sync<T2>(bar);
    }
    group_sync<T2>(bar);   // skipped CMuxes have no barrier
    uint64_t *o = a.out + (size_t)blockIdx.x * (N2 + 1);
    for (int m = t; m < N2; m += T2) o[m] = m == 0 ? acc[0] : 0ull - acc[N2 - m];
    if (t == 0) o[N2] = acc[N2] + a.out_b_add;
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(*slot, BT_COLS);
    }
}

template <int C>
cudaError_t launch_team_t(const Pbs02Args &a, int num_sms, cudaStream_t st)
{
    const int groups = (a.B + C - 1) / C;
    pbs02_team_kernel<C><<<groups < num_sms ? groups : num_sms, TEAMS * T2, TeamShape<C>::TOTAL, st>>>(a);
    return cudaGetLastError();
}

template <int C>
cudaError_t init_team_t()
{
    return cudaFuncSetAttribute(pbs02_team_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                TeamShape<C>::TOTAL);
}

}  // namespace

// p: ciphertexts per SM in a pass.  Three run as passes of two for two thirds
// of the batch, then passes of one.
cudaError_t launch_pbs02_f64(const Pbs02Args &a, int num_sms, int p, cudaStream_t st)
{
    if (a.B <= 0) return cudaSuccess;
    if (p == 1) return launch_team_t<1>(a, num_sms, st);
    if (p == 2) return launch_team_t<2>(a, num_sms, st);
    if (p != 3) return cudaErrorInvalidValue;
    const int passes = (a.B + 3 * num_sms - 1) / (3 * num_sms), two = 2 * num_sms * passes;
    Pbs02Args r = a;
    r.B = a.B < two ? a.B : two;
    cudaError_t e = launch_team_t<2>(r, num_sms, st);
    if (e != cudaSuccess || r.B == a.B) return e;
    r.in += (size_t)r.B * (N0 + 1);
    r.out += (size_t)r.B * (N2 + 1);
    r.B = a.B - r.B;
    return launch_team_t<1>(r, num_sms, st);
}

// one ciphertext per block, four blocks per SM
cudaError_t launch_pbs02_blocks(const Pbs02Args &a, cudaStream_t st)
{
    if (a.B <= 0) return cudaSuccess;
    pbs02_block_kernel<<<a.B, T2, BlockSmem::TOTAL, st>>>(a);
    return cudaGetLastError();
}

cudaError_t init_pbs02_f64()
{
    cudaError_t e = init_team_t<1>();
    if (e == cudaSuccess) e = init_team_t<2>();
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(pbs02_block_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, BlockSmem::TOTAL);
    return e;
}

}  // namespace cfdb
