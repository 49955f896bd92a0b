// Standalone batched negacyclic transforms in TFHEpp's frequency layout:
// TwistIFFT (torus -> frequency) and TwistFFT (frequency -> torus) for the
// 32-bit torus, N = 1024 (thirdparty/TFHEpp/include/mulfft.hpp:57-121).
// One warp per polynomial, using the same warp transform as the PBS kernel.
#include "fftops.cuh"

namespace cfdb {

namespace {

__device__ __forceinline__ int bitrev9(int x) { return (int)(__brev((unsigned)x) >> 23); }

// Frequencies in TFHEpp's layout (bit-reversed, real half then imaginary half):
// slots s and s + 8 of a lane are neighbours there, but a warp's pairs lie 256
// bytes apart.  They are put in order in shared memory, in 16-byte chunks (real
// parts 0 .. 255, imaginary 256 .. 511) swizzled against bank conflicts, and cross
// memory in whole lines: stored one by one, 32 lines to an instruction, they
// bound the kernel (8,000 polynomials: 53.6 -> 30.3 us in, 52.6 -> 30.7 us back).
// VEC: the array is 16-byte aligned.
__device__ __forceinline__ int freq_chunk1(int c) { return c ^ ((c >> 5) & 7); }

template <bool VEC>
__global__ void __launch_bounds__(128, 5) twist_ifft1_kernel(double *out, const uint32_t *in, int B, const Fft512Tables *T)
{
    __shared__ double2 xp_s[4][FFT512_XP];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int p = blockIdx.x * 4 + w;
    if (p >= B) return;
    const uint32_t *a = in + (size_t)p * N1;
    double2 v[16];
#pragma unroll
    for (int m2 = 0; m2 < 16; ++m2) {
        const int m = lane + 32 * m2;
        v[m2] = cmul(make_double2((double)(int32_t)a[m], (double)(int32_t)a[m + 512]), T->twist[m2 * 32 + lane]);
    }
    fft512_fwd(v, xp_s[w], *T, lane);
    double *o = out + (size_t)p * N1;
    double2 *xp = xp_s[w];
    __syncwarp();
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        const int c = freq_chunk1(bitrev9(fft512_freq(lane, s)) >> 1);
        xp[c] = make_double2(v[s].x, v[s + 8].x);
        xp[c + 256] = make_double2(v[s].y, v[s + 8].y);
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const int c = lane + 32 * j;
        const double2 z = xp[freq_chunk1(c & 255) + (c & 256)];
        if (VEC) {
            reinterpret_cast<double2 *>(o)[c] = z;
        } else {
            o[2 * c] = z.x;
            o[2 * c + 1] = z.y;
        }
    }
}

template <bool VEC>
__global__ void __launch_bounds__(128, 5) twist_fft1_kernel(uint32_t *out, const double *in, int B, const Fft512Tables *T)
{
    __shared__ double2 xp_s[4][FFT512_XP];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int p = blockIdx.x * 4 + w;
    if (p >= B) return;
    const double *x = in + (size_t)p * N1;
    double2 v[16];
    double2 *xp = xp_s[w];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const int c = lane + 32 * j;
        v[j] = VEC ? reinterpret_cast<const double2 *>(x)[c] : make_double2(x[2 * c], x[2 * c + 1]);
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const int c = lane + 32 * j;
        xp[freq_chunk1(c & 255) + (c & 256)] = v[j];
    }
    __syncwarp();
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        const int c = freq_chunk1(bitrev9(fft512_freq(lane, s)) >> 1);
        const double2 re = xp[c], im = xp[c + 256];
        v[s] = make_double2(re.x, im.x);
        v[s + 8] = make_double2(re.y, im.y);
    }
    __syncwarp();   // before the transform writes xp
    fft512_inv(v, xp_s[w], *T, lane);
    uint32_t *o = out + (size_t)p * N1;
#pragma unroll
    for (int m2 = 0; m2 < 16; ++m2) {
        const int m = lane + 32 * m2;
        const double2 y = cmulc(v[m2], T->twist[m2 * 32 + lane]);
        o[m] = f64_to_torus32(y.x * (1.0 / 512.0));
        o[m + 512] = f64_to_torus32(y.y * (1.0 / 512.0));
    }
}

}  // namespace

cudaError_t launch_twist_ifft1(double *out, const uint32_t *in, int B, const Fft512Tables *T, cudaStream_t st)
{
    if (B <= 0) return cudaSuccess;
    if (((uintptr_t)out & 15) == 0) twist_ifft1_kernel<true><<<(B + 3) / 4, 128, 0, st>>>(out, in, B, T);
    else twist_ifft1_kernel<false><<<(B + 3) / 4, 128, 0, st>>>(out, in, B, T);
    return cudaGetLastError();
}

cudaError_t launch_twist_fft1(uint32_t *out, const double *in, int B, const Fft512Tables *T, cudaStream_t st)
{
    if (B <= 0) return cudaSuccess;
    if (((uintptr_t)in & 15) == 0) twist_fft1_kernel<true><<<(B + 3) / 4, 128, 0, st>>>(out, in, B, T);
    else twist_fft1_kernel<false><<<(B + 3) / 4, 128, 0, st>>>(out, in, B, T);
    return cudaGetLastError();
}

}  // namespace cfdb
