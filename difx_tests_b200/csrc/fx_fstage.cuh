// fx_fstage.cuh -- pieces shared by the F-stage kernels (fx_fpair.cuh, fx_ftc.cu, fx_ftc32.cu) and the debug
// unpack export: FFT geometry, 2-bit decode, twiddles, and the bounded wait on an input copy.
#pragma once

#include <algorithm>
#include <cstdio>

#include "fx_common.cuh"
#include "fx_kernels.h"

namespace fx {

constexpr int ilog2c(int x) { return x <= 1 ? 0 : 1 + ilog2c(x / 2); }

// FFT plan of length F.  CPX: complex input (8-bit complex samples), every bin a
// channel (C = F); otherwise real input, channels below F/2 (C = F/2).  Only the
// channel-side constants (C, STRIDE, S, FS, FST, NROT) depend on CPX.
template <int F, bool CPX = false>
struct FPlan {
    static constexpr int C = CPX ? F : F / 2;
    static constexpr int NT = F / 16;                        // threads per FFT (pair)
    static constexpr int STRIDE = 1 << (ilog2c(C) / 2);      // kernel.c:31 generalised
    static constexpr int S = F / STRIDE;                      // substride (kernel.c:36)
    static constexpr int FS = STRIDE;                         // frac "sub" length
    static constexpr int FST = C / STRIDE;                    // frac "step" length
    static constexpr int NPASS = (F == 256) ? 2 : (F <= 4096 ? 3 : 4);
    static constexpr int LASTR = (F == 256) ? 16 : (F == 512) ? 2 : (F == 1024) ? 4 : (F == 2048) ? 8
                               : (F == 4096) ? 16 : 2;
    static constexpr int NSLOT = (NT >= 256) ? 1 : 256 / NT;
    static constexpr int NTHREADS = NT * NSLOT;
    static constexpr int MINB = (NTHREADS <= 256) ? 2 : 1;    // CTAs per SM the registers must allow
};

// Staged input bytes per FFT slot: the FFT's bytes (2-bit real: F*npol/4 plus the
// read-ahead byte of kernel.c:402-409; 8-bit complex: 2 bytes per sample and
// polarisation) plus up to 15 bytes of 16-byte alignment slack, rounded to 16.
template <int F, int NPOL, bool CPX>
constexpr int fstage_inb()
{
    return ((CPX ? F * NPOL * 2 : F * NPOL / 4 + 1) + 15 + 15) / 16 * 16;
}

__device__ __forceinline__ int padi(int i) { return i + (i >> 4); }

__device__ __forceinline__ float2 twiddle_exact(int m, int n)
{
    float s, c;
    sincospif(-2.0f * (float)m / (float)n, &s, &c);
    return make_float2(c, s);
}

// Stage the packed bytes of one FFT into shared memory with 128-bit loads.  The
// window starts at the 16-byte boundary at or below the FFT's first byte and
// covers the F*npol/4 (+1 when the offset is not byte-aligned, kernel.c:402-409)
// bytes the FFT spans; with the alignment slack that is <= F*npol/4 + 16 bytes.
// Returns the window's base byte index in the antenna row.
__device__ __forceinline__ int stage_fft_bytes(const uint8_t* row, int offset, int npol, int F, uint8_t* inb,
                                               int t, int nthr)
{
    const int first_byte = (npol == 2) ? (offset >> 1) : (offset >> 2);
    const int base_byte = first_byte & ~15;
    const int nvec = (F * npol / 4 + 1 + (first_byte - base_byte) + 15) >> 4;
    const uint4* src = reinterpret_cast<const uint4*>(row + base_byte);
    uint4* dst = reinterpret_cast<uint4*>(inb);
    for (int i = t; i < nvec; i += nthr) dst[i] = __ldg(src + i);
    return base_byte;
}

// Quantiser level of absolute sample s, polarisation pol (kernel.c:397-426 bit
// order for npol=2; 4 consecutive samples per byte, LSB first, for npol=1).
__device__ __forceinline__ float decode_sample(const uint8_t* inb, int base_byte, int s, int npol, int pol)
{
    uint32_t code;
    if (npol == 2) {
        const uint32_t byte = inb[(s >> 1) - base_byte];
        code = (byte >> (4 * (s & 1) + 2 * pol)) & 3u;
    } else {
        const uint32_t byte = inb[(s >> 2) - base_byte];
        code = (byte >> (2 * (s & 3))) & 3u;
    }
    return level2bit(code);
}

// ---- input staging by the bulk-copy (TMA) engine: one cp.async.bulk per FFT into the
// slot's staging buffer, completing an mbarrier phase; every wait is bounded by time.
__device__ __forceinline__ uint32_t smem_u32a(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long gtimer()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void stg_bar_init(uint64_t* bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32a(bar)) : "memory");
}

__device__ __forceinline__ bool stg_try(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32a(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// true when the phase completed, false after 1 s
__device__ __forceinline__ bool stg_wait(uint64_t* bar, uint32_t parity)
{
    if (stg_try(bar, parity)) return true;
    const unsigned long long t0 = gtimer();
    while (!stg_try(bar, parity))
        if (gtimer() - t0 > 1000000000ull) return false;
    return true;
}

}  // namespace fx
