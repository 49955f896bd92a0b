// Batched identity key switching, lvl1->lvl0, lvl2->lvl0, lvl2->lvl1.
//
// Restates IdentityKeySwitch<P> (thirdparty/TFHEpp/src/keyswitch.cpp:11-48):
//   b' = b (same width) or round(b / 2^32) (64 -> 32 bit),
//   for each input coefficient i and digit j < t:
//     a_ij = ((a_i + prec_offset) >> (w - (j+1) basebit)) & (2^basebit - 1)
//     if a_ij != 0: res -= ksk[i][j][a_ij - 1]
// The reference runs this on the host for every GPU bootstrap
// (src/cuHEDB/gatebootstrap_gpu.cuh:42,133).  Here it is an HBM-bound gather
// over key rows padded to 16-byte multiples (ksk_pitch), read as uint4:
// one CTA per ciphertext walks the input coefficients in chunks of NT; each
// chunk's digits are decoded into a shared list of selected key rows (in key
// order), then
// every thread accumulates a fixed set of output words over those rows with
// several rows' loads in flight.  All CTAs of a batch walk the key in the same
// order, so concurrently running CTAs that select the same row share it in L2.
#include "common.cuh"
#include "iks.cuh"

namespace cfdb {

namespace {

// a 16-byte read-only load, issued where it stands (volatile: the U loads of
// a group are all in flight before the first subtraction)
__device__ __forceinline__ uint4 ldg_v4(const uint4 *p)
{
    uint4 v;
    asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}

// a -= x, placed after the group's loads (volatile, like them)
__device__ __forceinline__ void sub_v4(uint4 &a, const uint4 &x)
{
    asm volatile("sub.u32 %0, %0, %4;\n\tsub.u32 %1, %1, %5;\n\tsub.u32 %2, %2, %6;\n\tsub.u32 %3, %3, %7;"
                 : "+r"(a.x), "+r"(a.y), "+r"(a.z), "+r"(a.w)
                 : "r"(x.x), "r"(x.y), "r"(x.z), "r"(x.w));
}

// acc[p] -= row[t + p NT] (16-byte words of the padded rows) over the listed
// rows, U rows' loads in flight per thread
template <int NP4, int NT>
__device__ __forceinline__ void gather_rows(const uint4 *__restrict__ ksk, const uint32_t *rowid, int nrows,
                                            uint4 *acc)
{
    constexpr int PER = (NP4 + NT - 1) / NT;
    constexpr int U = 8;
    const int t = threadIdx.x;
    int r = 0;
    for (; r + U <= nrows; r += U) {
        uint4 v[U][PER];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint4 *row = ksk + (size_t)rowid[r + u] * NP4;
#pragma unroll
            for (int p = 0; p < PER; ++p) {
                const int k = t + p * NT;
                v[u][p] = (k < NP4) ? ldg_v4(row + k) : make_uint4(0u, 0u, 0u, 0u);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int p = 0; p < PER; ++p) sub_v4(acc[p], v[u][p]);
    }
    for (; r < nrows; ++r) {
        const uint4 *row = ksk + (size_t)rowid[r] * NP4;
#pragma unroll
        for (int p = 0; p < PER; ++p) {
            const int k = t + p * NT;
            if (k < NP4) {
                const uint4 x = ldg_v4(row + k);
                acc[p].x -= x.x;
                acc[p].y -= x.y;
                acc[p].z -= x.z;
                acc[p].w -= x.w;
            }
        }
    }
}

// input coefficient k of ciphertext `ct`; for the lvl1 gate form the input is
// sa*ca + sb*cb (TFHEpp HomGate, src/gate.cpp:50-58)
template <bool WIDE>
__device__ __forceinline__ uint64_t iks_input(const IksArgs &a, size_t base, int k)
{
    if constexpr (WIDE) {
        return a.in64[base + k];
    } else {
        uint32_t x = a.in32[base + k];
        if (a.in32b) x = (uint32_t)a.sa * x + (uint32_t)a.sb * a.in32b[base + k];
        else x = (uint32_t)a.sa * x;
        return x;
    }
}

// the output's b word before any key row: b' of the reference
template <bool WIDE, int NIN>
__device__ __forceinline__ uint32_t iks_b(const IksArgs &a, size_t base)
{
    if constexpr (WIDE) return (uint32_t)((a.in64[base + NIN] + a.offset64 + (1ull << 31)) >> 32);
    else return (uint32_t)iks_input<false>(a, base, NIN) + a.offset;
}

// (0, ..., 0, b'): what the parts of a divided switch add to
template <bool WIDE, int NIN, int NOUT>
__global__ void iks_init_kernel(IksArgs a)
{
    const int ct = blockIdx.x;
    const uint32_t b = iks_b<WIDE, NIN>(a, (size_t)ct * (NIN + 1));
    for (int k = threadIdx.x; k < NOUT; k += blockDim.x) a.out[(size_t)ct * NOUT + k] = k == NOUT - 1 ? b : 0u;
}

// one CTA per (ciphertext, part of the input coefficients).  With one part
// (PARTS false) it writes its ciphertext's output; otherwise every part adds
// its sum to the initialised output (integer sums modulo 2^32: any order gives
// the same words).
template <int NT, bool WIDE, int NIN, int BASEBIT, int TT, int NOUT, bool PARTS>
__global__ void __launch_bounds__(NT) iks_kernel(IksArgs a)
{
    static_assert(NT % 32 == 0, "whole warps");
    constexpr int NW = NT / 32;
    __shared__ uint32_t rowid[NT * TT];
    __shared__ int wsum[NW];
    constexpr int W = WIDE ? 64 : 32;
    constexpr uint64_t prec = 1ull << (W - (1 + BASEBIT * TT));
    constexpr uint32_t mask = (1u << BASEBIT) - 1;
    constexpr int NP4 = ksk_pitch(NOUT) / 4;
    constexpr int PER = (NP4 + NT - 1) / NT;
    const int ct = blockIdx.x;
    const size_t base = (size_t)ct * (NIN + 1);
    uint4 acc[PER];
#pragma unroll
    for (int p = 0; p < PER; ++p) acc[p] = make_uint4(0u, 0u, 0u, 0u);

    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int first = PARTS ? (int)((long long)NIN * blockIdx.y / gridDim.y) : 0;
    const int last = PARTS ? (int)((long long)NIN * (blockIdx.y + 1) / gridDim.y) : NIN;
    for (int i0 = first; i0 < last; i0 += NT) {
        // the chunk's selected rows, compacted in key order (ascending i, j)
        // so that every CTA of the batch walks the key the same way and rows
        // that several ciphertexts select are fetched close together in time
        const int i = i0 + threadIdx.x;
        uint32_t ids[TT];
        int n = 0;
        if (i < last) {
            const uint64_t abar = iks_input<WIDE>(a, base, i) + prec;
#pragma unroll
            for (int j = 0; j < TT; ++j) {
                const uint32_t d = (uint32_t)((WIDE ? abar : (uint32_t)abar) >> (W - (j + 1) * BASEBIT)) & mask;
                if (d) ids[n++] = ((uint32_t)i * TT + j) * mask + d - 1;
            }
        }
        int incl = n;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += y;
        }
        if (lane == 31) wsum[wid] = incl;
        __syncthreads();
        int pos = incl - n, total = 0;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            const int c = wsum[w];
            if (w < wid) pos += c;
            total += c;
        }
#pragma unroll
        for (int j = 0; j < TT; ++j)
            if (j < n) rowid[pos + j] = ids[j];
        __syncthreads();
        gather_rows<NP4, NT>(reinterpret_cast<const uint4 *>(a.ksk), rowid, total, acc);
        __syncthreads();
    }

    uint32_t *o = a.out + (size_t)ct * NOUT;
    const uint32_t bnew = PARTS ? 0u : iks_b<WIDE, NIN>(a, base);
#pragma unroll
    for (int p = 0; p < PER; ++p) {
        const int k0 = 4 * (threadIdx.x + p * NT);
        const uint32_t v[4] = {acc[p].x, acc[p].y, acc[p].z, acc[p].w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (k0 + c >= NOUT) continue;
            if constexpr (PARTS) atomicAdd(o + k0 + c, v[c]);
            else o[k0 + c] = k0 + c == NOUT - 1 ? v[c] + bnew : v[c];
        }
    }
}

// Parts per ciphertext.  One CTA keeps 8 rows (24 KB) in flight and takes 0.57 ms
// (lvl10) over its 2,048 rows however empty the GPU is, so a batch is divided
// into about 64 CTAs per SM, of at least 16 input coefficients each.  The
// undivided form is left where it is the faster one: a batch that nearly fills one
// wave of resident CTAs (10 per SM for lvl10, of 32 registers a thread, and 8 for
// lvl20, of 34), or more than one and a half, walks the key in step and shares its
// rows in L2.  So a batch is divided up to FEW ciphertexts per SM, and from one
// wave to TAIL per SM, where the undivided form runs a second, nearly empty one.
// ms on 148 SMs, undivided -> divided (lvl21: batches of 128 and more come here only
// without scratch):
//   lvl10   1: 0.213 -> 0.025;  148: 0.574 -> 0.142;  592: 0.589 -> 0.396;
//     850: 0.600 -> 0.545;  950: 0.615 -> 0.636;  1,300: 0.693 -> 0.813;
//     1,480: 0.717 -> 0.934;  1,481: 1.25 -> 0.930;  1,850: 1.27 -> 1.13;
//     2,072: 1.30 -> 1.32
//   lvl20   1: 0.395 -> 0.026;  148: 1.08 -> 0.262;  592: 1.11 -> 0.768;
//     750: 1.14 -> 1.05;  850: 1.16 -> 1.18;  1,100: 1.27 -> 1.49;  1,184: 1.30 -> 1.33;
//     1,185: 2.33 -> 1.40;  1,850: 2.45 -> 2.37;  1,900: 2.47 -> 2.56
//   lvl21   1: 3.38 -> 0.026;  148: 2.49 -> 0.60;  511: 2.26 -> 2.10
struct GatherRule {
    double few, wave, tail;   // ciphertexts per SM
};
constexpr GatherRule IKS10_RULE{5.75, 10.0, 12.8}, IKS20_RULE{5.4, 8.0, 12.5};

inline int iks_parts(int B, int num_sms, const GatherRule &r, int max_parts)
{
    const double per_sm = (double)B / num_sms;
    if (per_sm > r.tail || (per_sm > r.few && per_sm <= r.wave)) return 1;
    const int p = (int)((64ll * num_sms + B - 1) / B);
    return p < max_parts ? p : max_parts;
}

// Whether the output shares bytes with an input, as in a switch of one row in
// place.  The divided forms write the output before they have read the input, so
// these calls take the undivided gather, which reads a row first.
template <int NIN, int NOUT>
bool in_place(const IksArgs &a)
{
    const uintptr_t o = (uintptr_t)a.out, oe = o + (size_t)a.B * NOUT * sizeof(uint32_t);
    auto meets = [&](const void *in, size_t word) {
        const uintptr_t i = (uintptr_t)in;
        return in && i < oe && o < i + (size_t)a.B * (NIN + 1) * word;
    };
    return meets(a.in32, 4) || meets(a.in32b, 4) || meets(a.in64, 8);
}

template <int NT, bool WIDE, int NIN, int BASEBIT, int TT, int NOUT>
cudaError_t launch_gather(const IksArgs &a, const GatherRule &rule, cudaStream_t st)
{
    const int parts = in_place<NIN, NOUT>(a) ? 1 : iks_parts(a.B, a.num_sms, rule, NIN / 16);
    if (parts == 1) {
        iks_kernel<NT, WIDE, NIN, BASEBIT, TT, NOUT, false><<<a.B, NT, 0, st>>>(a);
        return cudaGetLastError();
    }
    iks_init_kernel<WIDE, NIN, NOUT><<<a.B, 256, 0, st>>>(a);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    iks_kernel<NT, WIDE, NIN, BASEBIT, TT, NOUT, true><<<dim3(a.B, parts), NT, 0, st>>>(a);
    return cudaGetLastError();
}

// ---- key-stationary lvl2 -> lvl1 switch --------------------------------------------
// The gather above reads each selected 4,100-byte key row once per ciphertext:
// 75 GB per 1,024 ciphertexts, served from L2 (the 0.59 GB key stays there).
// Turned around, each CTA owns 8 output words of TILE ciphertexts and walks a
// part of the key, staging those 8 words of every key row in shared memory, and
// each thread, one ciphertext, subtracts the staged words of the rows its digits
// select.  Integer sums modulo 2^32: the parts add up to the gather's words.
// Bound by the L1 data pipe (93 % busy at 200 and at 1,024), which serves the
// shared-memory reads (two of 16 bytes per digit, a wavefront per quarter-warp: 2.4 ms
// per 1,024) and, per tile, the staging (about 0.3 ms):
// so 512 ciphertexts share a tile where there are more than 256, and warps past
// the batch only stage.  The staged rows are padded to 48 bytes, so the eight
// digit values of a quarter-warp's 16-byte reads fall in eight distinct bank
// groups.  The key is divided over CTAs because 129 word blocks a tile fill the
// SMs unevenly.  ms, whole key per CTA of 256 -> divided, 256 / 512 a tile:
//   256: 0.98 -> 0.75 / 0.81;  512: 1.92 -> 1.46 / 1.38;  1,024: 3.58 -> 2.86 / 2.70;
//   2,048: 5.85 -> 5.66 / 5.35;  4,096: 11.8 -> 11.3 / 10.6
constexpr int KS_WB = 8;                              // output words per CTA
constexpr int KS_NB = (N1 + 1 + KS_WB - 1) / KS_WB;   // word blocks: 129
constexpr int KS_DIG = 1 << KS21_BASEBIT;             // digit values 0..7 (row 0: zeros)
constexpr int KS_RW4 = 3;                             // uint4 per staged row: 8 words + 4 pad
constexpr int KS_P4 = ksk_pitch(N1 + 1) / 4;          // uint4 per key row in HBM: 257
constexpr uint64_t KS_PREC = 1ull << (64 - (1 + KS21_BASEBIT * KS21_T));
constexpr int KS_SHIFT = 64 - KS21_BASEBIT * KS21_T;                    // the digits' 30 bits

// X[i][b] = the top 30 bits of a_i + prec_offset (ciphertext b's ten digits
// of coefficient i), 0 for the padding b >= B
__global__ void ks21_prep_kernel(const uint64_t *__restrict__ in, uint32_t *X, int B, int Bp)
{
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t)N2 * Bp) return;
    const int i = (int)(idx / Bp), b = (int)(idx % Bp);
    X[idx] = b < B ? (uint32_t)((in[(size_t)b * (N2 + 1) + i] + KS_PREC) >> KS_SHIFT) : 0u;
}

// TILE ciphertexts per CTA, IC input coefficients per staged chunk; the output
// holds (0, ..., 0, b') and takes every part's sum
template <int TILE, int IC>
__global__ void __launch_bounds__(TILE, 1024 / TILE) ks21_kernel(const uint32_t *__restrict__ X, int Bp,
                                                                 const uint4 *__restrict__ ksk, uint32_t *out, int B)
{
    constexpr int KS_TILE = TILE, KS_IC = IC;
    constexpr int KS_ROWS = KS_IC * KS21_T * KS_DIG;                               // staged rows per chunk
    constexpr int KS_LOADS = KS_IC * KS21_T * (KS_DIG - 1) * (KS_WB / 4);          // uint4 per chunk
    constexpr int KS_PER = (KS_LOADS + KS_TILE - 1) / KS_TILE;                     // per thread
    __shared__ uint4 stage[2][KS_ROWS * KS_RW4];
    const int t = threadIdx.x, s = blockIdx.x, ct = blockIdx.y * KS_TILE + t;
    const bool live = (ct & ~31) < B;
    // digit-0 rows are zero in both buffers (never written again)
    for (int e = t; e < 2 * KS_IC * KS21_T * KS_RW4; e += KS_TILE) {
        const int buf = e / (KS_IC * KS21_T * KS_RW4), rem = e % (KS_IC * KS21_T * KS_RW4);
        stage[buf][(rem / KS_RW4) * KS_DIG * KS_RW4 + rem % KS_RW4] = make_uint4(0u, 0u, 0u, 0u);
    }
    // this thread's share of chunk c: key row (i, j, d) words 16 s + 4 q .. + 3,
    // where they exist (the last word block holds only the padded row's word
    // 1024 and its pad: q = 0)
    uint4 r[KS_PER];
    auto load = [&](int c) {
#pragma unroll
        for (int k = 0; k < KS_PER; ++k) {
            const int e = t + k * KS_TILE;
            r[k] = make_uint4(0u, 0u, 0u, 0u);
            if (e < KS_LOADS) {
                const int q = e % (KS_WB / 4), row = e / (KS_WB / 4);   // row = (ii T + j) (2^b - 1) + d - 1
                const int w4 = (KS_WB / 4) * s + q;
                if (w4 < KS_P4) {
                    const size_t g = (size_t)c * KS_IC * KS21_T * (KS_DIG - 1) + row;
                    r[k] = __ldg(ksk + g * KS_P4 + w4);
                }
            }
        }
    };
    auto store = [&](int buf) {
#pragma unroll
        for (int k = 0; k < KS_PER; ++k) {
            const int e = t + k * KS_TILE;
            if (e < KS_LOADS) {
                const int q = e % (KS_WB / 4), row = e / (KS_WB / 4), ij = row / (KS_DIG - 1),
                          d = row % (KS_DIG - 1) + 1;
                stage[buf][(ij * KS_DIG + d) * KS_RW4 + q] = r[k];
            }
        }
    };
    uint32_t acc[KS_WB];
#pragma unroll
    for (int k = 0; k < KS_WB; ++k) acc[k] = 0u;
    constexpr int NCHUNK = N2 / KS_IC;
    const int first = NCHUNK * blockIdx.z / gridDim.z, last = NCHUNK * (blockIdx.z + 1) / gridDim.z;
    load(first);
    store(first & 1);
    __syncthreads();
#pragma unroll 1
    for (int c = first; c < last; ++c) {
        if (c + 1 < last) load(c + 1);
        const uint4 *buf = stage[c & 1];
        for (int ii = 0; live && ii < KS_IC; ++ii) {
            const uint32_t x = X[(size_t)(c * KS_IC + ii) * Bp + (size_t)blockIdx.y * KS_TILE + t];
#pragma unroll
            for (int j = 0; j < KS21_T; ++j) {
                const uint32_t d = (x >> (KS21_BASEBIT * (KS21_T - 1 - j))) & (KS_DIG - 1);
                const uint4 *row = buf + ((ii * KS21_T + j) * KS_DIG + d) * KS_RW4;
#pragma unroll
                for (int q = 0; q < KS_WB / 4; ++q) {
                    const uint4 v = row[q];
                    acc[4 * q] -= v.x;
                    acc[4 * q + 1] -= v.y;
                    acc[4 * q + 2] -= v.z;
                    acc[4 * q + 3] -= v.w;
                }
            }
        }
        if (c + 1 < last) store((c + 1) & 1);
        __syncthreads();
    }
    if (ct >= B) return;
    uint32_t *o = out + (size_t)ct * (N1 + 1) + KS_WB * s;
#pragma unroll
    for (int k = 0; k < KS_WB; ++k)
        if (KS_WB * s + k <= N1) atomicAdd(o + k, acc[k]);
}

// the key walked in `parts` parts by each word block and tile
template <int TILE, int IC>
cudaError_t launch_ks21(const IksArgs &a, uint32_t *X, int Bp, int parts, cudaStream_t st)
{
    iks_init_kernel<true, N2, N1 + 1><<<a.B, 256, 0, st>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const size_t n = (size_t)N2 * Bp;
    ks21_prep_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(a.in64, X, a.B, Bp);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    ks21_kernel<TILE, IC><<<dim3(KS_NB, Bp / TILE, parts), TILE, 0, st>>>(X, Bp, reinterpret_cast<const uint4 *>(a.ksk),
                                                                           a.out, a.B);
    return cudaGetLastError();
}

// Batches from KS21_MIN on take the key-stationary switch (ms, gather ->
// key-stationary: 96 0.39 -> 0.39, 128 0.51 -> 0.47, 200 0.77 -> 0.68, 300 1.14 ->
// 0.98).  It needs 8 KB of scratch per ciphertext; below KS21_SCRATCH the gather
// stands in where that is not to be had, and in a stream that is being captured,
// whose graph then holds no allocation of its own.
constexpr int KS21_MIN = 128, KS21_SCRATCH = 512;

// done: whether the switch was enqueued
cudaError_t ks21_key_stationary(const IksArgs &a, bool &done, cudaStream_t st)
{
    done = false;
    if (a.B < KS21_SCRATCH) {
        cudaStreamCaptureStatus cs;
        const cudaError_t e = cudaStreamIsCapturing(st, &cs);
        if (e != cudaSuccess) {
            cudaGetLastError();   // the gather's launch reports what is wrong with the stream
            return cudaSuccess;
        }
        if (cs != cudaStreamCaptureStatusNone) return cudaSuccess;
    }
    const int tile = a.B <= 256 ? 256 : 512, tiles = (a.B + tile - 1) / tile, Bp = tiles * tile;
    uint32_t *X = nullptr;
    cudaError_t e = cudaMallocAsync((void **)&X, (size_t)N2 * Bp * sizeof(uint32_t), st);
    if (e == cudaErrorMemoryAllocation && a.B < KS21_SCRATCH) {
        cudaGetLastError();   // not this call's failure: the gather needs no scratch
        return cudaSuccess;
    }
    if (e != cudaSuccess) return e;
    done = true;
    e = tile == 256 ? launch_ks21<256, 2>(a, X, Bp, 32, st)
                    : launch_ks21<512, 4>(a, X, Bp, tiles < 4 ? 16 / tiles : 4, st);
    const cudaError_t ef = cudaFreeAsync(X, st);
    return e != cudaSuccess ? e : ef;
}

}  // namespace

cudaError_t launch_iks(const IksArgs &a, int kind, cudaStream_t st)
{
    if (a.B <= 0) return cudaSuccess;
    if (kind == 21 && a.B >= KS21_MIN && !in_place<N2, N1 + 1>(a)) {
        bool done;
        const cudaError_t e = ks21_key_stationary(a, done, st);
        if (e != cudaSuccess || done) return e;
    }
    // one 16-byte word of a padded row per thread: 169 of 192 (lvl0 rows),
    // 257 of 288 (lvl1 rows)
    if (kind == 10) return launch_gather<192, false, N1, KS10_BASEBIT, KS10_T, N0 + 1>(a, IKS10_RULE, st);
    if (kind == 20) return launch_gather<192, true, N2, KS20_BASEBIT, KS20_T, N0 + 1>(a, IKS20_RULE, st);
    if (kind == 21) return launch_gather<288, true, N2, KS21_BASEBIT, KS21_T, N1 + 1>(a, IKS20_RULE, st);
    return cudaErrorInvalidValue;
}

}  // namespace cfdb
