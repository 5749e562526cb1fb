// fx_kmajor.cu -- corner turn of FP16 spectra: [sb][sig][t][chan] as the FFT F stage stores them (channel
// contiguous, one (Re, Im) half pair per channel) to the K-major layout [sb][chan][rows][T] of the
// tensor-core X stage (row 2 sig = Re, 2 sig + 1 = Im), with the FP8 form's running absmax.
//
// Memory bound: it reads and writes the spectra once, in whole 128-byte lines on both sides.  A CTA
// turns 64 channels x 64 FFTs of one signal (16 KB, eight CTAs per SM, so 128 KB in flight per SM)
// through shared memory; word (t, c) stands at 64 t + (c ^ 4 (t / 8 mod 8)), which keeps both the
// 8-byte writes along c and the reads of 8 FFTs x 4 channels per warp on distinct banks.
#include <algorithm>

#include "fx_common.cuh"
#include "fx_kernels.h"

namespace fx {

namespace {
constexpr int KC = 64, KT = 64, KTHREADS = 256;
}

// FFTs KT tx .., channels KC cx .. of spectrum row z = (subband, signal)
__device__ __forceinline__ void kmajor_tile(const __half2* __restrict__ src, int src_T, int nsig, int nchan, int rows,
                                            __half* __restrict__ dst, int dst_T, int t_off, unsigned* __restrict__ amax,
                                            int tx, int cx, int z)
{
    __shared__ __align__(16) uint32_t tile[KT * KC];
    const int t0 = tx * KT, c0 = cx * KC;
    const int sb = z / nsig, sig = z - sb * nsig;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const __half2* in = src + ((size_t)z * src_T + t0) * nchan + c0;
    uint2 v[8];
#pragma unroll
    for (int k = 0; k < 8; k++)
        v[k] = __ldcs(reinterpret_cast<const uint2*>(in + (size_t)(warp + 8 * k) * nchan) + lane);
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int t = warp + 8 * k;
        *reinterpret_cast<uint2*>(tile + t * KC + ((2 * lane) ^ (4 * (k & 7)))) = v[k];   // t / 8 = k
    }
    __syncthreads();
    const int ch = lane & 7, cc = lane >> 3;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int c = 4 * (warp + 8 * k) + cc;
        uint32_t w[8];
#pragma unroll
        for (int q = 0; q < 8; q++) w[q] = tile[(8 * ch + q) * KC + (c ^ (4 * ch))];
        uint4 re, im;
        re.x = __byte_perm(w[0], w[1], 0x5410); im.x = __byte_perm(w[0], w[1], 0x7632);
        re.y = __byte_perm(w[2], w[3], 0x5410); im.y = __byte_perm(w[2], w[3], 0x7632);
        re.z = __byte_perm(w[4], w[5], 0x5410); im.z = __byte_perm(w[4], w[5], 0x7632);
        re.w = __byte_perm(w[6], w[7], 0x5410); im.w = __byte_perm(w[6], w[7], 0x7632);
        const size_t item = (size_t)sb * nchan + c0 + c;
        __half* out = dst + (item * rows + 2 * sig) * dst_T + t_off + t0 + 8 * ch;
        *reinterpret_cast<uint4*>(out) = re;
        *reinterpret_cast<uint4*>(out + dst_T) = im;
        if (amax) {
            // max(|Re|, |Im|) of the 64 FFTs; non-negative floats order like their bit patterns
            __half2 m = __float2half2_rn(0.f);
#pragma unroll
            for (int q = 0; q < 8; q++) m = __hmax2(m, __habs2(*reinterpret_cast<const __half2*>(&w[q])));
            float f = fmaxf(__low2float(m), __high2float(m));
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) f = fmaxf(f, __shfl_xor_sync(0xffffffffu, f, o));
            if (ch == 0 && f > 0.f) atomicMax(amax + item * nsig + sig, __float_as_uint(f));
        }
    }
}

__global__ void __launch_bounds__(KTHREADS)
k_kmajor(const __half2* __restrict__ src, int src_T, int nsig, int nchan, int rows, __half* __restrict__ dst, int dst_T,
         int t_off, unsigned* __restrict__ amax)
{
    kmajor_tile(src, src_T, nsig, nchan, rows, dst, dst_T, t_off, amax, blockIdx.x, blockIdx.y, blockIdx.z);
}

// Blocks [first, next job's first) turn a job's slots.
__global__ void __launch_bounds__(KTHREADS) k_kmajor_batch(const KJob* __restrict__ jobs, int njobs)
{
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {
        const int m = (lo + hi + 1) / 2;
        if (jobs[m].first <= (int)blockIdx.x) lo = m;
        else hi = m - 1;
    }
    const KJob& j = jobs[lo];
    const int n = (int)blockIdx.x - j.first, nt = j.span / KT, nc = j.nchan / KC;
    kmajor_tile(static_cast<const __half2*>(j.src), j.src_T, j.nsig, j.nchan, j.rows, static_cast<__half*>(j.dst), j.dst_T, 0,
                nullptr, n % nt, n / nt % nc, n / nt / nc);
}

int kmajor_blocks(const KJob& j) { return j.span / KT * (j.nchan / KC) * j.nsb * j.nsig; }

cudaError_t launch_kmajor_batch(const KJob* d_jobs, int njobs, int nblocks, cudaStream_t st)
{
    if (njobs < 1 || nblocks < 1) return cudaErrorInvalidValue;
    k_kmajor_batch<<<nblocks, KTHREADS, 0, st>>>(d_jobs, njobs);
    return cudaGetLastError();
}

// Slots [0, span) of src [nsb][nsig][src_T][nchan] to slots t_off .. of dst [nsb][nchan][rows][dst_T].
cudaError_t launch_kmajor(const void* src, int src_T, int span, int nsb, int nsig, int nchan, int rows, void* dst,
                          int dst_T, int t_off, unsigned* amax, cudaStream_t st)
{
    if (span < KT || span % KT || span > src_T || t_off % 8 || t_off + span > dst_T || dst_T % 8 || nchan % KC ||
        2 * nsig > rows || nsb < 1 || nsig < 1)
        return cudaErrorInvalidValue;
    // grid.z holds at most 65535 (subband, signal) rows
    const int per = std::max(1, 65535 / nsig);
    for (int sb = 0; sb < nsb; sb += per) {
        const int n = std::min(per, nsb - sb);
        k_kmajor<<<dim3(span / KT, nchan / KC, n * nsig), KTHREADS, 0, st>>>(
            static_cast<const __half2*>(src) + (size_t)sb * nsig * src_T * nchan, src_T, nsig, nchan, rows,
            static_cast<__half*>(dst) + (size_t)sb * nchan * rows * dst_T, dst_T, t_off,
            amax ? amax + (size_t)sb * nchan * nsig : nullptr);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace fx
