// Self-test of the bounded waits: a key ring, and a staged round (ring.cuh), whose
// first chunk is never issued, so every consumer's wait for it runs out.  Each
// kernel must then record DEV_TIMEOUT_FULL in the context's error word, raise its
// abort flag so that no other warp waits, skip the refill, skip the drain
// (nothing was issued) and return; the host reads the code through
// cufhedb_sync and the context stays usable.  No copy is issued and no
// memory outside the block's own shared memory is touched.
#include "block_fft.cuh"
#include "ctx.cuh"
#include "ring.cuh"

namespace cfdb {

namespace {

constexpr int ST_S = 2, ST_CHUNK = 16, ST_W = 2;

__global__ void __launch_bounds__(ST_W * 32) ring_timeout_selftest_kernel(int *err, uint32_t limit)
{
    __shared__ __align__(128) unsigned char smem[RING_HEADER_BYTES + ST_S * ST_CHUNK];
    KeyRing<ST_S, ST_CHUNK, ST_W> ring{reinterpret_cast<RingHeader *>(smem), smem + RING_HEADER_BYTES, nullptr, 1u,
                                       2u, limit};
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) ring.init_by_thread0();
    __syncthreads();
    // no prologue: chunk 0 never lands
    ring.acquire(0, err);
    ring.release(0, lane);
    __syncthreads();
    if (threadIdx.x == 0) ring.drain_by_thread0(err);
}

// the staged round: both warps are teams.  `src` is never read; it is valid memory
// all the same.
__global__ void __launch_bounds__(ST_W * 32) round_timeout_selftest_kernel(int *err, uint32_t limit, const void *src)
{
    using Key = RoundKey<ST_CHUNK, ST_W>;
    __shared__ __align__(128) unsigned char smem[128 + ST_CHUNK];
    static_assert(Key::HEAD_BYTES <= 128, "head");
    Key key{smem, smem + 128, reinterpret_cast<const unsigned char *>(src), 1u, 2u, limit};
    if (threadIdx.x == 0) key.init();
    __syncthreads();
    // round 0 never lands
    key.acquire(0, err);
    __syncwarp();
    if ((threadIdx.x & 31) == 0) key.release(0);
    __syncthreads();
    if (threadIdx.x == 0) key.drain(err);
}

// The block transforms of the split path (block_fft.cuh) against the one-warp forms
// (fft_f32.cuh, split_steps.cuh) on the same values: random digits forward, random
// spectra of a bootstrap's size back into words.  Two warps, one limb each, as in
// a bootstrap; warp 0 also runs the one-warp forms.  diff counts forward values and
// inverse words that differ.
__device__ __forceinline__ uint32_t st_random(uint32_t x)
{
    x = (x ^ (x >> 16)) * 0x7feb352du;
    x = (x ^ (x >> 15)) * 0x846ca68bu;
    return x ^ (x >> 16);
}

__global__ void __launch_bounds__(64) split_transforms_selftest_kernel(const Fft512TablesFold *T, uint32_t seed, int *diff)
{
    using P = SplitPath;
    __shared__ __align__(16) float2 buf[2 * P::BUF];
    __shared__ unsigned long long xp[FFT512_XP];
    __shared__ uint32_t want[N1], got[N1];
    __shared__ uint32_t slot;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, hh = lane >> 4;
    if (warp == 0) tmem_alloc(&slot, P::COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = slot + ((32u * warp) << 16);
    P::stage_tables(tm, *T, lane);
    const P::Tab &W = *reinterpret_cast<const P::Tab *>(T->w32p);
    const uint32_t salt = st_random(seed + 0x9e3779b9u * (blockIdx.x + 1));
    if (warp == 0) {
        float2 r[16], v[16];
#pragma unroll
        for (int m2 = 0; m2 < 16; ++m2) {
            const uint32_t x = st_random(salt + lane + 32 * m2), u0 = x & 63u, u1 = (x >> 6) & 63u;
            r[m2] = cw64(make_float2((float)((int)u0 - 32), (float)((int)u1 - 32)), m2);
            reinterpret_cast<uint32_t *>(buf)[lane + 32 * m2] = u0 | (u1 << 16);
        }
        fdft16<1>(r);
        ffft512_fwd_tw_rest(r, reinterpret_cast<float2 *>(xp), *T, lane);
        P::forward(v, buf, lane, tm);
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 16; ++j) buf[32 * j + lane] = v[j];
        __syncwarp();
        int n = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int at = (j + 8 * hh) * 32 + (lane & 15);
            const float2 a = buf[at], t = P::mul(buf[at + 16], P::w32_fwd(W, j, hh));
            const float2 v0 = P::add(a, t), v1 = P::sub(a, t);
            n += (v0.x != r[j].x) + (v0.y != r[j].y) + (v1.x != r[8 + j].x) + (v1.y != r[8 + j].y);
        }
        if (n) atomicAdd(diff, n);
    }
    __syncthreads();
    // spectra whose inverse transforms have the sizes of the hi and lo limbs' sums
    auto freq = [&](int s, int c) {
        const float u = (float)(int)st_random(salt ^ (0x51ed270bu * (uint32_t)(64 * s + 2 * lane + c + 1)));
        const float w = (float)(int)st_random(salt ^ (0x2545f491u * (uint32_t)(64 * s + 2 * lane + c + 1)));
        return pk2(ldexpf(u, -9), ldexpf(w, 7));   // up to 2^22 and 2^38
    };
    for (int j = tid; j < N1; j += 64) want[j] = got[j] = 0;
    __syncthreads();
    if (warp == 0) {
        CP f[16];
#pragma unroll
        for (int s = 0; s < 16; ++s) f[s] = CP{freq(s, 0), freq(s, 1)};
#pragma unroll
        for (int j = 0; j < 8; ++j)
            P::put(buf, 0, (j + 8 * hh) * 32 + (lane & 15), P::Sum{f[j]}, P::Sum{f[8 + j]}, P::w32_inv(W, j, hh));
        add_inverse_split(want, f, xp, lane, *T);
    }
    __syncthreads();
    P::inverse(buf + warp * P::BUF, buf + (warp ^ 1) * P::BUF, warp, lane, tm, [&](int m, uint32_t x) { got[m] += x; });
    __syncthreads();
    for (int j = tid; j < N1; j += 64)
        if (want[j] != got[j]) atomicAdd(diff + 1, 1);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(slot, P::COLS);
    }
}

}  // namespace

}  // namespace cfdb

using namespace cfdb;

int cufhedb_selftest_wait_timeout(cufhedb_ctx *ctx, uint32_t polls)
{
    if (!ctx) return set_error(CUFHEDB_ERR_ARG, "ctx is null");
    if (polls == 0 || polls > (1u << 20)) return set_error(CUFHEDB_ERR_ARG, "polls must be in [1, 2^20]");
    DeviceGuard guard(ctx->device);
    ring_timeout_selftest_kernel<<<1, ST_W * 32>>>(ctx->err, polls);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_error(e, "wait self-test launch");
    const int rc = cufhedb_sync(ctx, nullptr);
    if (rc != CUFHEDB_ERR_DEVICE) return rc;
    round_timeout_selftest_kernel<<<1, ST_W * 32>>>(ctx->err, polls, ctx->tab512);
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_error(e, "wait self-test launch");
    return cufhedb_sync(ctx, nullptr);
}

int cufhedb_selftest_split_transforms(cufhedb_ctx *ctx, uint32_t seed, int blocks, int *forward_differ, int *inverse_differ)
{
    if (!ctx || !forward_differ || !inverse_differ) return set_error(CUFHEDB_ERR_ARG, "null argument");
    if (blocks <= 0 || blocks > 65536) return set_error(CUFHEDB_ERR_ARG, "blocks must be in [1, 65536]");
    DeviceGuard guard(ctx->device);
    int *diff = nullptr, host[2] = {0, 0};
    cudaError_t e = cudaMalloc((void **)&diff, sizeof host);
    if (e == cudaSuccess) e = cudaMemset(diff, 0, sizeof host);
    if (e == cudaSuccess) {
        // 8 KB more than it uses: at most seven blocks per SM, whose tensor memory fits
        split_transforms_selftest_kernel<<<blocks, 64, 8192>>>(&ctx->tab512f->fold, seed, diff);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(host, diff, sizeof host, cudaMemcpyDeviceToHost);
    cudaFree(diff);
    if (e != cudaSuccess) return cuda_error(e, "split transform self-test");
    *forward_differ = host[0];
    *inverse_differ = host[1];
    return CUFHEDB_OK;
}
