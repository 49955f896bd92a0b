// The lvl2 ring (N = 2048, 64-bit torus, l = 4, Bg = 2^9) in FP64: batched lvl2
// external products, standalone TwistIFFT / TwistFFT<lvl2param>, and key
// preparation (bootstrapping: pbs02_f64.cu).
//
// The external product restates trgswfftExternalProduct<lvl2param> (thirdparty/
// TFHEpp/src/trgsw.cpp:77-103).  The conversions follow TFHEpp's 64-bit torus
// FFT: int64 -> double rounding on the way in, truncation toward zero modulo
// 2^64 on the way out; FP64 keeps ~53 bits of a 64-bit torus value, the
// intrinsic precision of this path (TFHEpp's own round trip error bound is
// 2^14, test/polymul.cpp:57-68).
//
// Four warps (T2 = 128 threads, 8 complex values each) per polynomial.  Keys and
// prepared TRGSWs are stored in 16 KB chunks, one per (TRGSW row, output), as
// [slot s][thread u], so each thread reads exactly the frequencies it owns.
#include "fft1024_f64.cuh"
#include "lvl2.cuh"
#include "lvl2_steps.cuh"

namespace cfdb {

namespace {

// integer polynomials [rows][2][2048] (64-bit torus) -> chunk layout
// [rows][2 o][8 s][128 u] complex (one 1024-complex chunk per (row, o))
__global__ void __launch_bounds__(T2) bk_fft2_kernel(double2 *dst, const uint64_t *src, const Fft1024Tables *T)
{
    __shared__ double2 xp_s[FFT8X_XP<T2>];
    const int t = threadIdx.x;
    const size_t poly = blockIdx.x;
    const uint64_t *p = src + poly * N2;
    double2 v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int m = t + T2 * j;
        v[j] = cx_w32<1>(make_double2(__ll2double_rn((long long)p[m]), __ll2double_rn((long long)p[m + 1024])), j);
    }
    fft8x_fwd<double2, T2>(v, xp_s, *T, t, 1);
    double2 *d = dst + poly * 1024;
#pragma unroll
    for (int s = 0; s < 8; ++s) d[s * T2 + t] = v[s];
}

__device__ __forceinline__ int bitrev10(int x) { return (int)(__brev((unsigned)x) >> 22); }

// TFHEpp BootstrappingKeyFFT<lvl02param> / TRGSWFFT<lvl2param> rows (re | im
// halves, bit-reversed order) -> chunk layout
__global__ void bk_permute2_kernel(double2 *dst, const double *src, int rows)
{
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;   // (poly, s, u)
    if (e >= (size_t)rows * 2 * 1024) return;
    const int u = (int)(e & (T2 - 1)), s = (int)((e >> 7) & 7);
    const size_t poly = e >> 10;
    const int idx = bitrev10(fft1024_freq(u, s));
    const double *p = src + poly * N2;
    dst[e] = make_double2(p[idx], p[idx + 1024]);
}

// Frequencies in TFHEpp's layout (bit-reversed, real half then imaginary half):
// slots s and s + 4 of a thread are neighbours there, but a warp's pairs lie 128
// bytes apart, one line each.  They are put in order in shared memory, in 16-byte
// chunks (real parts 0 .. 511, imaginary 512 .. 1023) swizzled against bank
// conflicts, and cross memory in whole lines (8,000 polynomials: 70.6 -> 50.3 us
// in, 5.2 TB/s, 62.5 -> 52.6 us back).  VEC: the array is 16-byte aligned.
__device__ __forceinline__ int freq_chunk2(int c) { return c ^ ((c >> 3) & 7); }

template <bool VEC>
__device__ __forceinline__ void put_freq2(double *o, const double2 v[8], double2 *xp, int t)
{
    group_sync<T2>(1);   // every warp is done with xp
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const int c = bitrev10(fft1024_freq(t, s)) >> 1;
        xp[freq_chunk2(c)] = make_double2(v[s].x, v[s + 4].x);
        xp[freq_chunk2(c) + 512] = make_double2(v[s].y, v[s + 4].y);
    }
    group_sync<T2>(1);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int c = t + T2 * j;
        const double2 z = xp[freq_chunk2(c & 511) + (c & 512)];
        if (VEC) {
            reinterpret_cast<double2 *>(o)[c] = z;
        } else {
            o[2 * c] = z.x;
            o[2 * c + 1] = z.y;
        }
    }
}
template <bool VEC>
__device__ __forceinline__ void get_freq2(double2 v[8], const double *x, double2 *xp, int t)
{
    double2 z[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int c = t + T2 * j;
        z[j] = VEC ? reinterpret_cast<const double2 *>(x)[c] : make_double2(x[2 * c], x[2 * c + 1]);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int c = t + T2 * j;
        xp[freq_chunk2(c & 511) + (c & 512)] = z[j];
    }
    group_sync<T2>(1);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const int c = bitrev10(fft1024_freq(t, s)) >> 1;
        const double2 re = xp[freq_chunk2(c)], im = xp[freq_chunk2(c) + 512];
        v[s] = make_double2(re.x, im.x);
        v[s + 4] = make_double2(re.y, im.y);
    }
    group_sync<T2>(1);   // before the transform writes xp
}

template <bool VEC>
__global__ void __launch_bounds__(T2) twist_ifft2_kernel(double *out, const uint64_t *in, const Fft1024Tables *T)
{
    __shared__ double2 xp_s[FFT8X_XP<T2>];
    const int t = threadIdx.x;
    const size_t p = blockIdx.x;
    const uint64_t *x = in + p * N2;
    double2 v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int m = t + T2 * j;
        v[j] = cx_w32<1>(make_double2(__ll2double_rn((long long)x[m]), __ll2double_rn((long long)x[m + 1024])), j);
    }
    fft8x_fwd<double2, T2>(v, xp_s, *T, t, 1);
    put_freq2<VEC>(out + p * N2, v, xp_s, t);
}

template <bool VEC>
__global__ void __launch_bounds__(T2) twist_fft2_kernel(uint64_t *out, const double *in, const Fft1024Tables *T)
{
    __shared__ double2 xp_s[FFT8X_XP<T2>];
    const int t = threadIdx.x;
    const size_t p = blockIdx.x;
    const double *x = in + p * N2;
    double2 v[8];
    get_freq2<VEC>(v, x, xp_s, t);
    fft8x_inv<double2, T2>(v, xp_s, *T, t, 1);
    uint64_t *o = out + p * N2;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int m = t + T2 * j;
        const double2 y = cx_w32<-1>(v[j], j);
        o[m] = f64_to_torus64(y.x * (1.0 / 1024.0));
        o[m + 1024] = f64_to_torus64(y.y * (1.0 / 1024.0));
    }
}

// one product per 128-thread block; trgsw prepared: [8 rows][2 o][1024] complex
__global__ void __launch_bounds__(T2) extprod2_kernel(ExtProd2Args a)
{
    __shared__ double2 xp_s[FFT8X_XP<T2>];
    const int t = threadIdx.x;
    const size_t p = blockIdx.x;
    const Fft1024Tables &T = *a.tables;
    const uint64_t *in = a.trlwe + p * 2 * N2;
    const double2 *g = a.trgsw + (a.shared ? 0 : p * 2 * L2 * 2 * 1024);
    // the TRGSW rows two ahead of the one in use are fetched into L2 (32 KB
    // per row: both outputs), so the loads after each transform find them there
    constexpr uint32_t ROW_BYTES = 2 * 1024 * sizeof(double2);
    auto prefetch = [&](int r0, int n) {
        if (a.shared || t != 0) return;
        for (int k = r0; k < r0 + n && k < 2 * L2; ++k)
            bulk_prefetch_l2(reinterpret_cast<const unsigned char *>(g) + (size_t)k * ROW_BYTES, ROW_BYTES);
    };
    prefetch(0, 2);
    if (t == 0) bulk_prefetch_l2_if_aligned(in, 2 * N2 * sizeof(uint64_t));   // the TRLWE, read per digit polynomial
    double2 f0[8], f1[8];
#pragma unroll 1
    for (int r = 0; r < 2 * L2; ++r) {
        double2 v[8];
        uint64_t xw[16];
        prefetch(r + 2, 1);
        digit_words2<false>(xw, in + (r / L2) * N2, 0, t);
        digits2(v, xw, r % L2);
        fft8x_fwd<double2, T2>(v, xp_s, T, t, 1);
        const double2 *g0 = g + ((size_t)r * 2) * 1024, *g1 = g0 + 1024;
        if (r == 0) {
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                f0[s] = cx_mul(v[s], g0[s * T2 + t]);
                f1[s] = cx_mul(v[s], g1[s * T2 + t]);
            }
        } else {
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                cx_fma(f0[s], v[s], g0[s * T2 + t]);
                cx_fma(f1[s], v[s], g1[s * T2 + t]);
            }
        }
    }
    uint64_t *o = a.out + p * 2 * N2;
    fft8x_inv<double2, T2>(f0, xp_s, T, t, 1);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int m = t + T2 * j;
        const double2 y = cx_w32<-1>(f0[j], j);
        o[m] = f64_to_torus64(y.x * (1.0 / 1024.0));
        o[m + 1024] = f64_to_torus64(y.y * (1.0 / 1024.0));
    }
    fft8x_inv<double2, T2>(f1, xp_s, T, t, 1);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int m = t + T2 * j;
        const double2 y = cx_w32<-1>(f1[j], j);
        o[N2 + m] = f64_to_torus64(y.x * (1.0 / 1024.0));
        o[N2 + m + 1024] = f64_to_torus64(y.y * (1.0 / 1024.0));
    }
}

}  // namespace

cudaError_t bk02_to_fft(double2 *dst, const uint64_t *src, int rows, const Fft1024Tables *T, cudaStream_t st)
{
    if (rows <= 0) return cudaSuccess;
    bk_fft2_kernel<<<rows * 2, T2, 0, st>>>(dst, src, T);
    return cudaGetLastError();
}

cudaError_t bkfft02_permute(double2 *dst, const double *src, int rows, cudaStream_t st)
{
    const size_t n = (size_t)rows * 2 * 1024;
    bk_permute2_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(dst, src, rows);
    return cudaGetLastError();
}

cudaError_t launch_twist_ifft2(double *out, const uint64_t *in, int B, const Fft1024Tables *T, cudaStream_t st)
{
    if (B <= 0) return cudaSuccess;
    if (((uintptr_t)out & 15) == 0) twist_ifft2_kernel<true><<<B, T2, 0, st>>>(out, in, T);
    else twist_ifft2_kernel<false><<<B, T2, 0, st>>>(out, in, T);
    return cudaGetLastError();
}

cudaError_t launch_twist_fft2(uint64_t *out, const double *in, int B, const Fft1024Tables *T, cudaStream_t st)
{
    if (B <= 0) return cudaSuccess;
    if (((uintptr_t)in & 15) == 0) twist_fft2_kernel<true><<<B, T2, 0, st>>>(out, in, T);
    else twist_fft2_kernel<false><<<B, T2, 0, st>>>(out, in, T);
    return cudaGetLastError();
}

cudaError_t launch_extprod2(const ExtProd2Args &a, cudaStream_t st)
{
    if (a.B <= 0) return cudaSuccess;
    extprod2_kernel<<<a.B, T2, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace cfdb
