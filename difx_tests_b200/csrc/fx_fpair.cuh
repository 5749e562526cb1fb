// fx_fpair.cuh -- fused F stage of the FX correlator for sm_100a: two FFTs at a time in packed FP32.
//
// Per FFT and polarisation, without touching HBM in between (kernel.c line numbers of the reference):
//   offset / validity / fractional delay from the delay table (733-756), 2-bit decode of F samples
//   (397-426) or 8-bit complex samples (gkernel.cu:277-296), fringe rotation (428-497), forward
//   unnormalised FFT (499-510), fractional-sample correction (512-555), store of channels [0, C).
//   The conjugation (557-568) is folded into the X stage.
//
// What bounds it: shared memory (exchanges, twiddles, sample table: 401 wavefronts per 1024 samples at 4096
// points, 73 % of the data pipe), then the FP32 pipe (53 %); HBM runs at a quarter of its rate.  A
// scalar FFT is bound by instruction issue instead (75 instructions per sample).  So a slot of NT = F / 16 threads takes a PAIR of FFTs -- both polarisations
// of one FFT, or two consecutive FFTs of a single-polarisation antenna -- and holds 16 points of
// each as (lane A, lane B) register pairs: every butterfly is a packed f32x2 instruction on two
// independent FFTs with no operand shuffles, half the issue slots of the scalar form.
//
// The FFT is radix 16 Stockham (Govindaraju et al., SC'08: 16 points per thread, exchanges in
// padded shared memory, remainder radix last), each pass as radix-2 stages with the twiddle folded
// into the butterfly (the FMA form of Linzer and Feig, IEEE TSP 41, 1993): s = a + w b in four FMAs
// and 2 a - s, here s - 2 a = -(a - w b), in two more, so the output of channel c carries the
// sign (-1)^popcount(c), which the correction factors below take out again.  A stage needs 1, 1,
// 2, 4 distinct w (the others are -i times one of them).
//
// The sums of many FFTs keep what the factors get wrong the same way every time, their magnitudes above
// all, so w is built to its last bit: rho is kept as rho - 1 (small: it is one bit's share of the
// phase) and w = W + (W_lo + W (rho - 1)), with the rounding W_lo of the constant W put back where
// there is room for it (passes 0 and 1).  Visibility errors halve against w = rho W rounded twice.
//
// Fringe rotation: its phase is lo (j / F + i stride / F) a with n = i S + j (145, 428-497), linear
// in the bits of the sample number n, and every stage contracts one bit of n, so the rotation is
// one factor rho per FFT and stage, multiplied into that stage's w: log2 F factors per FFT instead
// of a table of S + stride and a complex multiply per sample.  The constant phase lo b' and the
// fractional-sample correction, linear in the channel number c = t + NT e, are a product
// E[t] G[e] applied to the 8 (16 for complex input) channels a thread stores.
//
// Thread t = 16 d0 + u of a slot takes samples n = r NT + u NT / 16 + d0 in pass 0 and butterfly t of
// pass 1, whose inputs are then those of the 16 threads with its d0: the first exchange stays inside
// half a warp and needs no barrier.  (Complex input reads its bytes without an expansion step, in
// order of t, and exchanges across the slot.)
//
// Slots are independent workers that draw the pairs of a launch from a counter (nothing is CTA-wide after
// the constant tables are built), so one kernel serves a single job and a batch of jobs; with a
// fixed share each, the CTA an SM's schedulers favour ended early and left its partner alone
// (14 of 16 warps active on average).  Per pair i:
//   pass 0; factor tables of pair i + 1                                              | barrier
//   exchange, pass 1; sample expansion and pass 0 / 1 twiddles of pair i + 1         | barrier
//   pass 2 (and 3), correction, store
// while the slot's first thread describes pair i + 2, copies its bytes and fetches the delay
// entries of pair i + 3.
//
// Real samples at 1024 and 2048 points (PPlan::R32) take a plan with one exchange instead of two: 32 points a thread
// (32 x 32; 64 x 32 with two threads to a set of 64 samples, each of which decodes all of them and forms its half of
// stage 0's outputs), 314 wavefronts per 1024 samples (2048 points), one barrier fewer, coalesced runs of 32
// channels.  It costs 184 registers, so 8 warps per SM: too few to hide a pair's preparation, which a helper warp
// per slot does instead -- descriptors in registers, samples straight from global memory, factor
// tables three FP64 chains abreast -- and meets the slot's threads at two barriers per pair:
//   helper:  words and factors of pair i + 1                | expansion, pass 0 twiddles of i + 1, entries of i + 2
//   others:  stage 0, pass 0 of pair i                      | exchange, pass 1, correction, store
// 23 antennas x 3 subbands x 2777 FFTs of 1024 points: 0.459 -> 0.351 ms; 64 antennas x 8 subbands x 31250 FFTs of
// 2048 points: 72 -> 65.5 ms (power-limited: 1.85 GHz).  Without the helper 0.450 and 67.9.  At 4096 points this plan
// needs a radix 2 over lanes (64 shuffles a thread) or half the warps and gains nothing.
//
// Measured (B200, against one scalar FFT per slot, fx_fscalar.cuh with FP32 spectra): 64 antennas x 8 subbands
// x 31250 FFTs of 2048 points, one polarisation: 89.7 -> 70.6 ms (464 Gsamp/s; now R32); 16 antennas x 2
// polarisations x 4 subbands x 31250 FFTs of 4096 points: 47.1 -> 32.3 ms (507 Gsamp/s).
#pragma once

#include "fx_fstage.cuh"

namespace fx {

// A complex number of both lanes: x = (re A, re B), y = (im A, im B).
struct c2 {
    float2 x, y;
};
__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ c2 as_c2(float4 f) { return c2{make_float2(f.x, f.y), make_float2(f.z, f.w)}; }
__device__ __forceinline__ float4 as_f4(c2 a) { return make_float4(a.x.x, a.x.y, a.y.x, a.y.y); }
__device__ __forceinline__ c2 cmul2(c2 a, c2 b)
{
    return c2{__ffma2_rn(a.x, b.x, neg2(__fmul2_rn(a.y, b.y))), __ffma2_rn(a.x, b.y, __fmul2_rn(a.y, b.x))};
}

// A factor of both lanes in shared memory: one (x, y) when the lanes are polarisations of one FFT, or
// (x A, x B, y A, y B).  (An (x, x, y, y) for the former saves the two moves but takes twice the
// shared-memory wavefronts, and those bound the kernel.)
// mul(r, W): W rho of r = rho - 1; with the constant's rounding Wl put back.
template <int NPOL>
struct Fac {
    using T = float4;
    static __device__ __forceinline__ c2 get(T f) { return as_c2(f); }
    static __device__ __forceinline__ T mul(T r, float2 w)
    {
        const c2 a = as_c2(r);
        const float2 wx = dup(w.x), wy = dup(w.y);
        return as_f4(c2{__ffma2_rn(a.x, wx, __ffma2_rn(neg2(a.y), wy, wx)), __ffma2_rn(a.x, wy, __ffma2_rn(a.y, wx, wy))});
    }
    static __device__ __forceinline__ T mul(T r, float2 w, float2 wl)
    {
        const c2 a = as_c2(r);
        const float2 wx = dup(w.x), wy = dup(w.y);
        return as_f4(c2{__fadd2_rn(wx, __ffma2_rn(neg2(a.y), wy, __ffma2_rn(a.x, wx, dup(wl.x)))),
                        __fadd2_rn(wy, __ffma2_rn(a.y, wx, __ffma2_rn(a.x, wy, dup(wl.y))))});
    }
    static __device__ __forceinline__ T rho(T r) { return make_float4(1.f + r.x, 1.f + r.y, r.z, r.w); }
    static __device__ __forceinline__ T by(T a, float2 k) { return as_f4(cmul2(as_c2(a), c2{dup(k.x), dup(k.y)})); }
};
template <>
struct Fac<2> {
    using T = float2;
    static __device__ __forceinline__ c2 get(T f) { return c2{dup(f.x), dup(f.y)}; }
    static __device__ __forceinline__ T mul(T r, float2 w)
    {
        return make_float2(fmaf(r.x, w.x, fmaf(-r.y, w.y, w.x)), fmaf(r.x, w.y, fmaf(r.y, w.x, w.y)));
    }
    static __device__ __forceinline__ T mul(T r, float2 w, float2 wl)
    {
        return make_float2(w.x + fmaf(-r.y, w.y, fmaf(r.x, w.x, wl.x)), w.y + fmaf(r.y, w.x, fmaf(r.x, w.y, wl.y)));
    }
    static __device__ __forceinline__ T rho(T r) { return make_float2(1.f + r.x, r.y); }
    static __device__ __forceinline__ T by(T a, float2 k) { return cmul(a, k); }
};

// a, b -> a + w b, -(a - w b)
__device__ __forceinline__ void bfly(c2& a, c2& b, const c2& w)
{
    const float2 m2 = make_float2(-2.f, -2.f);
    c2 s;
    s.x = __ffma2_rn(neg2(w.y), b.y, __ffma2_rn(w.x, b.x, a.x));
    s.y = __ffma2_rn(w.y, b.x, __ffma2_rn(w.x, b.y, a.y));
    b.x = __ffma2_rn(a.x, m2, s.x);
    b.y = __ffma2_rn(a.y, m2, s.y);
    a = s;
}
// the same for the twiddle -i w
__device__ __forceinline__ void bfly_mi(c2& a, c2& b, const c2& w)
{
    const float2 m2 = make_float2(-2.f, -2.f);
    c2 s;
    s.x = __ffma2_rn(w.y, b.x, __ffma2_rn(w.x, b.y, a.x));
    s.y = __ffma2_rn(w.y, b.y, __ffma2_rn(neg2(w.x), b.x, a.y));
    b.x = __ffma2_rn(a.x, m2, s.x);
    b.y = __ffma2_rn(a.y, m2, s.y);
    a = s;
}
// only a + w b (the last stage of a real-input FFT: channels below F / 2)
__device__ __forceinline__ void bfly_lo(c2& a, const c2& b, const c2& w)
{
    a.x = __ffma2_rn(neg2(w.y), b.y, __ffma2_rn(w.x, b.x, a.x));
    a.y = __ffma2_rn(w.y, b.x, __ffma2_rn(w.x, b.y, a.y));
}
__device__ __forceinline__ void bfly_lo_mi(c2& a, const c2& b, const c2& w)
{
    a.x = __ffma2_rn(w.y, b.x, __ffma2_rn(w.x, b.y, a.x));
    a.y = __ffma2_rn(w.y, b.y, __ffma2_rn(neg2(w.x), b.x, a.y));
}

__host__ __device__ constexpr int bitrev(int v, int bits)
{
    int r = 0;
    for (int i = 0; i < bits; i++) r |= ((v >> i) & 1) << (bits - 1 - i);
    return r;
}

// Distinct twiddles of stage q of a butterfly: first index and count in the order q = 0, 1, 2, 2, 3, 3, 3, 3.
__host__ __device__ constexpr int wfirst(int q) { return q == 0 ? 0 : 1 << (q - 1); }
__host__ __device__ constexpr int wcount(int q) { return q == 0 ? 1 : 1 << (q - 1); }

// Stages [Q0, log2 R) of one radix-R butterfly in v[0 .. R): stage q contracts the top remaining bit
// of the element number; the sub-transforms' output numbers k' stand in bit-reversed block order, so
// output k ends at v[bitrev(k)].  w(d): twiddle d (order of wfirst), including the stage's rho.
// LO: the last stage keeps outputs k < R / 2 only.
template <int R, int Q0, bool LO, typename W>
__device__ __forceinline__ void butterfly(c2* v, W&& w)
{
    constexpr int M = ilog2c(R);
#pragma unroll
    for (int q = Q0; q < M; q++) {
#pragma unroll
        for (int d = 0; d < wcount(q); d++) {
            const c2 wd = w(wfirst(q) + d);
            const int len = R >> q, half = len >> 1;
#pragma unroll
            for (int h = 0; h < half; h++) {
                c2* p = v + bitrev(d, q) * len + h;
                if (LO && q == M - 1) bfly_lo(p[0], p[half], wd);
                else bfly(p[0], p[half], wd);
            }
            if (q > 0) {
                const int kp = d + (1 << (q > 0 ? q - 1 : 0));   // k' with twiddle -i w
#pragma unroll
                for (int h = 0; h < half; h++) {
                    c2* p = v + bitrev(kp, q) * len + h;
                    if (LO && q == M - 1) bfly_lo_mi(p[0], p[half], wd);
                    else bfly_mi(p[0], p[half], wd);
                }
            }
        }
    }
}

template <int F, int NPOL, bool CPX>
struct PPlan {
    using P = FPlan<F, CPX>;
    static constexpr int C = P::C;
    // real samples at 1024 and 2048 points: one exchange, 32 points per thread, H0 threads share a sample
    static constexpr bool R32 = !CPX && (F == 1024 || F == 2048);
    static constexpr int H0 = R32 && F == 2048 ? 2 : 1;
    static constexpr int NT = R32 ? F / 32 : F / 16;
    static constexpr int LOGF = ilog2c(F);
    static constexpr int LOGS = ilog2c(P::S);
    static constexpr int NPASS = P::NPASS;
    static constexpr int LASTR = P::LASTR;
    // slots of a CTA: 256 threads (complex samples at 256 points: 14 slots, what half an SM's shared memory holds)
    static constexpr int NSLOT = R32 ? 256 / NT : CPX && F == 256 ? 14 : P::NSLOT;
    // R32: a helper warp per slot, which prepares pairs; registers of compute and helper threads (their sum is what the
    // block is launched with, 168 or 128 a thread; splits by 8 either way measured 1 to 9 % slower)
    static constexpr int NCOMP = NT * NSLOT;
    static constexpr int NTHREADS = NCOMP + (R32 ? 32 * NSLOT : 0);
    static constexpr int PN = R32 ? 32 : NT;               // threads that prepare a slot's pairs
    static constexpr int R_COMP = 184, R_HELP = F == 2048 ? 136 : 72;
    static constexpr int MINB = R32 ? 1 : P::MINB;
    static constexpr int NE = CPX || R32 ? 16 : 8;         // channels a thread stores
    static constexpr int HI = NT / 16;
    static constexpr int NTAB = LOGF + 16 + HI + NE;       // rho, E low, E high, G
    static constexpr int NLANE = NPOL == 2 ? 1 : 2;        // delay entries of a pair
    static constexpr int R2 = NPASS == 2 ? 0 : NPASS == 3 ? LASTR : 16;   // radix of pass 2
    static constexpr int D2 = R32 ? 0 : R2 / 2;
    static constexpr bool W1TAB = !R32 && F > (CPX ? 1024 : 512);  // pass 1 twiddles per pair in a table
    // factor tables kept: those of pair i + 1 are written before the barrier that ends pair i - 1's
    // reads, except where a slot is half a warp or (complex input) they are written after it
    static constexpr int NTABS = R32 || CPX || NT < 32 ? 2 : 4;
    static constexpr int BUF = R32 ? F + F / 32 : F + F / 16;   // padded exchange buffer (float4)
    // one window (and the read past its last word); R32 stages none
    static constexpr int INB = R32 ? 16 : fstage_inb<F, NPOL, CPX>() + 16;
};

// What the slot's threads need of a pair.
struct PairLoc {
    const uint8_t* row;        // packed input of the antenna
    const DelayEntry* d;       // delay entry of lane A (lane B: the next one, or the same)
    unsigned char* out;        // lane A's spectrum
    size_t out_b;              // bytes from lane A's to lane B's
    const double* plo;         // the subband's LO (Hz), and its value (copied with the delay entries)
    double lo, chalf;          // chalf: half-turns per channel and second of fractional delay
    int* err;
    int has, wr;               // bit l: lane l holds an FFT of the call / is stored
    int end;                   // no pair: the slot is done
    int valid;                 // bit l: lane l's antenna is valid (has its bytes)
    int base[2], bit[2];       // lane's staged window: first byte in the row, first sample's bit in the window
};

template <int F, int NPOL, bool CPX>
struct PairSlot {              // shared memory of one slot
    using P = PPlan<F, NPOL, CPX>;
    float4 buf[P::BUF];
    using Fe = typename Fac<NPOL>::T;
    Fe tab[P::NTABS][P::NTAB]; // by pair number
    Fe w0[P::R32 ? 16 * P::H0 : 8];   // pass 0: 1 .. 7 of the twiddle order (R32: 16 per stage 0 output)
    Fe w1[P::W1TAB ? 2 : 1][P::W1TAB ? 128 : 2];   // by pair parity
    DelayEntry dent[P::R32 ? 1 : 4][2];
    PairLoc loc[4];
    alignas(16) uint8_t inb[P::NLANE][P::INB];
    alignas(16) uint8_t xs[CPX ? 16 : F];
    alignas(16) uint64_t bar;
    uint64_t pad;
};

template <int F, int NPOL, bool CPX>
struct PairSmem {
    using P = PPlan<F, NPOL, CPX>;
    PairSlot<F, NPOL, CPX> slot[P::NSLOT];
    float4 w1c[P::R32 ? 1 : 128];      // constant part of pass 1's twiddles [8][16] and its rounding
    float2 wbc[P::R32 ? 16 * P::NT : 1];               // R32: constant part of pass 1's twiddles [16][NT]
    float2 w2c[P::D2 ? P::D2 * 256 : 2];               // constant part of pass 2's twiddles [D2][256]
    float2 lut[16];            // levels of codes (A, B)
    float4 w0c[P::R32 ? 16 * P::H0 : 8];               // as w1c, of pass 0
};

template <int NT>
__device__ __forceinline__ void pair_sync(int slot)
{
    if constexpr (NT > 32) {
        asm volatile("bar.sync %0, %1;" ::"r"(slot + 1), "r"(NT) : "memory");
    } else {
        __syncwarp();
    }
}

// (cos, sin)(pi x) of x in [-1, 1]: Taylor series on the nearest multiple of pi / 2, to about 1e-11
__device__ __forceinline__ double2 cospi_d(double x)
{
    const double k = rint(2.0 * x);
    const double y = (x - 0.5 * k) * 3.14159265358979323846;
    const double z = y * y;
    double s = -1.0 / 39916800, c = 1.0 / 479001600;
    s = fma(s, z, 1.0 / 362880);
    c = fma(c, z, -1.0 / 3628800);
    s = fma(s, z, -1.0 / 5040);
    c = fma(c, z, 1.0 / 40320);
    s = fma(s, z, 1.0 / 120);
    c = fma(c, z, -1.0 / 720);
    s = fma(s, z, -1.0 / 6);
    c = fma(c, z, 1.0 / 24);
    s = fma(s * z, y, y);
    c = fma(c, z, -0.5);
    c = fma(c, z, 1.0);
    const int q = (int)k;
    const double a = q & 1 ? s : c, b = q & 1 ? c : s;
    return make_double2((q + 1) & 2 ? -a : a, q & 2 ? -b : b);
}

// e^{-2 pi i (jm + NS k') / (NS 2^(q+1))}: constant part of twiddle d of a pass with NS sub-transforms, and
// what its rounding to FP32 left
__device__ __forceinline__ float4 pass_w(int d, int jm, int NS)
{
    const int q = d == 0 ? 0 : 32 - __clz(d);
    const int kp = d - (q == 0 ? 0 : 1 << (q - 1));
    const double inv = __hiloint2double((1023 - (31 - __clz(NS)) - (q + 1)) << 20, 0);   // 1 / (NS 2^(q+1))
    const double2 w = cospi_d(-2.0 * (jm + NS * kp) * inv);
    const float x = __double2float_rn(w.x), y = __double2float_rn(w.y);
    return make_float4(x, y, __double2float_rn(w.x - (double)x), __double2float_rn(w.y - (double)y));
}

// Table entry e of one lane: rho - 1 of stage e, then E[t & 15], E[t >> 4], G.  Its angle in half-turns (of one
// form for all entries: a warp's threads don't part):
template <int F, int NPOL, bool CPX>
__device__ __forceinline__ double pair_angle(int e, double da, double db, double frac, double lo, double chalf)
{
    using P = PPlan<F, NPOL, CPX>;
    constexpr int LOGSTRIDE = P::LOGF - P::LOGS;
    // the FFT's constant phase, kernel.c:434-466: lo b', b' = b - (int)b, and the LO's fraction
    const double whole = trunc(db);
    double ph = dmul(dsub(db, whole), lo);
    const double lofrac = dsub(lo, trunc(lo));
    if (lofrac > 1e-11) ph = dadd(ph, dmul(lofrac, whole));   // kernel.c:39
    ph = 2.0 * dsub(ph, rint(ph));
    // kernel.c:145, 434-470: bit b of n weighs 2^b / F below S, 2^b / S steps of stride / F above
    const bool rho = e < P::LOGF;
    const int b = P::LOGF - 1 - e;
    const int ex = (b < P::LOGS ? b : b - P::LOGS + LOGSTRIDE) - P::LOGF;
    const int k = e - P::LOGF;
    const int c = k < 16 ? k : k < 16 + P::HI ? 16 * (k - 16) : P::NT * (k - 16 - P::HI);
    const double w = rho ? __hiloint2double((1023 + ex) << 20, 0) : (double)c;
    double x = dmul(dmul(w, rho ? da : chalf), rho ? lo : frac);
    x = rho ? -2.0 * x : dsub(x, k >= 16 + P::HI ? ph : 0.0);
    return dsub(x, 2.0 * rint(0.5 * x));
}
// and its value, of (cos, sin) of that angle
template <int F, int NPOL, bool CPX>
__device__ __forceinline__ float2 pair_entry(int e, double2 r)
{
    using P = PPlan<F, NPOL, CPX>;
    if (e < P::LOGF) return make_float2(__double2float_rn(r.x - 1.0), __double2float_rn(r.y));
    const int k = e - P::LOGF;
    const int c = k < 16 ? k : k < 16 + P::HI ? 16 * (k - 16) : P::NT * (k - 16 - P::HI);
    // sign of the FMA-form butterflies (two threads' stage 0 outputs are plain sums)
    const float sg = __popc(c & ~(P::H0 - 1)) & 1 ? -1.f : 1.f;
    return make_float2(sg * __double2float_rn(r.x), sg * __double2float_rn(r.y));
}

template <int F, int MODE, int NPOL, bool CPX, typename Locate>
__device__ __forceinline__ void pair_worker(PairSmem<F, NPOL, CPX>& sm, int nitem, int* ctr, const Locate& locate)
{
    using P = PPlan<F, NPOL, CPX>;
    constexpr int NT = P::NT;
    constexpr int PN = P::PN;
    const bool helper = P::R32 && threadIdx.x >= P::NCOMP;
    const int slot = helper ? (threadIdx.x - P::NCOMP) / 32 : threadIdx.x / NT;
    const int t = helper ? threadIdx.x & 31 : threadIdx.x - slot * NT;
    const bool lead = t == 0 && helper == P::R32;   // of the threads that draw the slot's pairs
    PairSlot<F, NPOL, CPX>& s = sm.slot[slot];
    using Fe = typename Fac<NPOL>::T;
    auto fac = [](Fe f) { return Fac<NPOL>::get(f); };
    auto mul_hl = [](Fe r, float4 w) { return Fac<NPOL>::mul(r, make_float2(w.x, w.y), make_float2(w.z, w.w)); };

    float2 wlast = make_float2(1.f, 0.f);   // 8192 points: W8192^t of the radix-2 pass
    if constexpr (P::NPASS == 4) wlast = twiddle_exact(t, F);

    // Tickets: a slot's first three pairs (those described before its first one is done) go by its number, the
    // others come from ctr[0] (ctr[1] counts the workers that are done; the last one zeroes both for
    // the next launch).  Half-warp slots draw
    // together, two pairs a ticket, and so keep one trip count in a warp.
    constexpr int PT = NT >= 32 ? 1 : 2;                     // slots (pairs) per ticket
    const int nwork = (int)gridDim.x * (P::NSLOT / PT);
    int ticket = (int)blockIdx.x * (P::NSLOT / PT) + slot / PT;
    auto draw = [&] {   // the slot's first thread: the next ticket
        int k = 0;
        if (PT == 1 || (slot & 1) == 0) k = 3 * nwork + atomicAdd(ctr, 1);
        if constexpr (PT == 2) k = __shfl_sync(0x00010001u, k, 0);
        return k;
    };
    const bool drawn = nitem > 3 * nwork * PT;   // otherwise no slot gets a fourth pair

    // stage of twiddle d (order of wfirst)
    auto stage_of = [](int d) { return d == 0 ? 0 : 32 - __clz(d); };

    // ---- slot's first thread: descriptor and delay entries of pair i, then its bytes
    auto fetch = [&](int i) {
        PairLoc& L = s.loc[i & 3];
        L.has = L.wr = L.valid = 0;
        L.end = ticket * PT >= nitem;
        const int g = ticket * PT + slot % PT;
        if (!L.end && !P::R32) ticket = i < 2 || !drawn ? ticket + nwork : draw();   // needed one pair later
        if (g < nitem) {
            locate(g, L);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32a(&L.lo)), "l"(L.plo) : "memory");
#pragma unroll
            for (int l = 0; l < P::NLANE; l++)
                if ((L.has >> l) & 1) {
                    const unsigned dst = smem_u32a(&s.dent[i & 3][l]);
                    const DelayEntry* src = L.d + l;
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst + 16),
                                 "l"(reinterpret_cast<const char*>(src) + 16)
                                 : "memory");
                }
        }
    };
    auto entries_wait = [] { asm volatile("cp.async.wait_all;" ::: "memory"); };
    // which lanes of pair i are valid, and where their first sample lies in the staged window: the window
    // (kernel.c:402-409: F NPOL / 4 bytes and the read-ahead byte, or 2 NPOL bytes per complex
    // sample) begins at the 16-byte boundary at or below the first byte
    constexpr int SB = CPX ? 16 * NPOL : 2 * NPOL;   // bits per sample
    auto describe = [&](PairLoc& L, const DelayEntry* dent) {
        int valid = 0;
#pragma unroll
        for (int l = 0; l < P::NLANE; l++) {
            L.bit[l] = 0;
            if ((L.has >> l) & 1) {
                const DelayEntry& d = dent[l];
                if (d.valid) {
                    valid |= 1 << l;
                    const long long bit = (long long)d.offset * SB;
                    L.base[l] = (int)(bit >> 3) & ~15;
                    L.bit[l] = (int)(bit - 8LL * L.base[l]);
                }
            }
        }
        L.valid = valid;
    };
    // the windows of pair i: whole 16-byte vectors by the bulk-copy engine
    auto copy = [&](const PairLoc& L) {
        if (!L.valid) return;
        uint32_t bytes[P::NLANE], total = 0;
#pragma unroll
        for (int l = 0; l < P::NLANE; l++) {
            bytes[l] = (L.valid >> l) & 1 ? 16u * ((F * SB / 8 + (CPX ? 0 : 1) + (L.bit[l] >> 3) + 15) >> 4) : 0u;
            total += bytes[l];
        }
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32a(&s.bar)), "r"(total)
                     : "memory");
#pragma unroll
        for (int l = 0; l < P::NLANE; l++)
            if (bytes[l]) {
                size_t gsrc;
                asm volatile("cvta.to.global.u64 %0, %1;" : "=l"(gsrc) : "l"(L.row + L.base[l]));
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                        smem_u32a(s.inb[l])),
                    "l"(gsrc), "r"(bytes[l]), "r"(smem_u32a(&s.bar))
                    : "memory");
            }
    };
    // factor tables of pair i, by the slot's last threads (the first one is busy with descriptors)
    auto factors = [&](int i, const PairLoc& L, const DelayEntry* dent) {
        float* tab = reinterpret_cast<float*>(s.tab[i & (P::NTABS - 1)]);   // single polarisation: lanes interleaved
        // (a helper's few rounds side by side: each is a chain of some thirty FP64 instructions)
        constexpr int N = P::NTAB * P::NLANE, NR = P::R32 ? (N + PN - 1) / PN : 1;
        for (int u0 = PN - 1 - t; u0 < N; u0 += NR * PN) {
            double x[NR];
#pragma unroll
            for (int r = 0; r < NR; r++) {
                const int u = u0 + r * PN, e = u / P::NLANE, l = u % P::NLANE;
                constexpr int B = P::NLANE - 1;
                const double da = l ? dent[B].a : dent[0].a, db = l ? dent[B].b : dent[0].b;
                const double df = l ? dent[B].frac : dent[0].frac;
                x[r] = u < N && ((L.valid >> l) & 1) ? pair_angle<F, NPOL, CPX>(e, da, db, df, L.lo, L.chalf) : 0.0;
            }
            double2 cs[NR];
#pragma unroll
            for (int r = 0; r < NR; r++) cs[r] = cospi_d(x[r]);
#pragma unroll
            for (int r = 0; r < NR; r++) {
                const int u = u0 + r * PN, e = u / P::NLANE, l = u % P::NLANE;
                if (u >= N) break;
                float2 v = make_float2(0.f, 0.f);   // an invalid lane's spectrum is zero
                if ((L.valid >> l) & 1) v = pair_entry<F, NPOL, CPX>(e, cs[r]);
                if constexpr (NPOL == 2) {
                    s.tab[i & (P::NTABS - 1)][e] = v;
                } else {
                    tab[4 * e + l] = v.x;
                    tab[4 * e + 2 + l] = v.y;
                }
            }
        }
    };

    uint32_t phase = 0;
    bool expired = false;
    auto bytes_wait = [&](const PairLoc& L) {
        if (L.valid) {
            if (!stg_wait(&s.bar, phase)) {
                if (t == 0 && L.err) atomicCAS(L.err, 0, 6);
                expired = true;
            }
            phase ^= 1;
        }
    };
    // at the end of the slot's pairs
    auto finish = [&] {
        // after an expired wait the copy may still land: wait for it once more (bounded) so it cannot
        // write into an exited CTA's shared memory
        if (!P::R32 && expired) stg_wait(&s.bar, phase ^ 1);
        if (drawn && lead && slot % PT == 0) {
            __threadfence();   // this worker's draws come before its count
            if (atomicAdd(ctr + 1, 1) == nwork - 1) {
                ctr[0] = 0;
                ctr[1] = 0;
            }
        }
    };
    // 2-bit real samples of pair i: one byte per sample pair, the offset of its levels in the table.  The
    // words of 16 samples are permuted so that pass 0's reads, NT / 16 samples apart, hit distinct banks.
    constexpr int SWZ = P::R32 ? 0 : NT == 512 ? 3 : NT == 256 ? 1 : 0;   // bits of n >> 7 taken into the word number
    struct Words { uint32_t w[NPOL == 2 ? 3 : 4]; };
    auto load16 = [&](const PairLoc& L, int t) {   // the words with samples 16 t .. 16 t + 15
        Words a;
#pragma unroll
        for (int l = 0; l < P::NLANE; l++) {
            const uint32_t* wp = reinterpret_cast<const uint32_t*>(s.inb[l]) + NPOL * t + (L.bit[l] >> 5);
#pragma unroll
            for (int k = 0; k < NPOL + 1; k++) a.w[2 * l + k] = wp[k];
        }
        return a;
    };
    auto expand16 = [&](const int (&sh)[P::NLANE], int t, const Words& a) {   // sh: the first one's bit in its word
        uint32_t nib[2];   // 8 samples each: codes (A, B) of sample k in bits 4 k .. 4 k + 3
        if constexpr (NPOL == 2) {
            nib[0] = __funnelshift_r(a.w[0], a.w[1], sh[0]);
            nib[1] = __funnelshift_r(a.w[1], a.w[2], sh[0]);
        } else {
            uint32_t sp[2][2];
#pragma unroll
            for (int l = 0; l < 2; l++) {
                const uint32_t b = __funnelshift_r(a.w[2 * l], a.w[2 * l + 1], sh[l]);
#pragma unroll
                for (int h = 0; h < 2; h++) {   // 2-bit groups of a half word to every second group
                    uint32_t x = h ? b >> 16 : b & 0xFFFFu;
                    x = (x | (x << 8)) & 0x00FF00FFu;
                    x = (x | (x << 4)) & 0x0F0F0F0Fu;
                    sp[l][h] = (x | (x << 2)) & 0x33333333u;
                }
            }
            nib[0] = sp[0][0] | (sp[1][0] << 2);
            nib[1] = sp[0][1] | (sp[1][1] << 2);
        }
        uint32_t o[4];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint32_t ev = (nib[h] << 3) & 0x78787878u, od = (nib[h] >> 1) & 0x78787878u;
            o[2 * h] = __byte_perm(ev, od, 0x5140);
            o[2 * h + 1] = __byte_perm(ev, od, 0x7362);
        }
        const int k = (t >> 3) & SWZ;
        if constexpr (SWZ & 1)
            if (k & 1) {
                uint32_t x = o[0]; o[0] = o[1]; o[1] = x;
                x = o[2]; o[2] = o[3]; o[3] = x;
            }
        if constexpr (SWZ & 2)
            if (k & 2) {
                uint32_t x = o[0]; o[0] = o[2]; o[2] = x;
                x = o[1]; o[1] = o[3]; o[3] = x;
            }
        *reinterpret_cast<uint4*>(s.xs + 16 * t) = make_uint4(o[0], o[1], o[2], o[3]);
    };
    constexpr int NG = P::R32 ? F / 512 : 1;
    auto expand_w = [&](const PairLoc& L, const Words (&a)[NG]) {
        int sh[P::NLANE];
#pragma unroll
        for (int l = 0; l < P::NLANE; l++) sh[l] = L.bit[l] & 31;
#pragma unroll
        for (int g = 0; g < NG; g++) expand16(sh, t + g * PN, a[g]);
    };
    auto expand = [&](const PairLoc& L) {   // from the staged bytes
        const Words a[NG] = {load16(L, t)};
        expand_w(L, a);
    };
    // twiddles of passes 0 and 1 with pair i's rho
    auto twiddles = [&](int i) {
        const Fe* tab = s.tab[i & (P::NTABS - 1)];
        if constexpr (P::R32) {
            for (int e = t; e < 16 * P::H0; e += PN) s.w0[e] = mul_hl(tab[P::H0 - 1 + stage_of(e & 15)], sm.w0c[e]);
        } else if (t < 8 && t > 0) {
            const int q = t == 1 ? 1 : t < 4 ? 2 : 3;
            s.w0[t] = mul_hl(tab[q], sm.w0c[t]);
        }
        if constexpr (P::W1TAB) {
            for (int e = t; e < 128; e += NT) {
                const int d = e >> 4;
                const int q = d == 0 ? 0 : d == 1 ? 1 : d < 4 ? 2 : 3;
                s.w1[i & 1][e] = mul_hl(tab[4 + q], sm.w1c[e]);
            }
        }
    };

    // R32: the helper's lanes hold the next pair's descriptor in registers, all the same (a chain of loads from shared
    // memory takes 300 cycles a link beside the other warps), and leave the other threads what they store by
    PairLoc nxt;
    DelayEntry dnxt[P::NLANE];
    auto load = [&](int i, int k) {   // pair i of the slot: ticket k
        nxt.has = nxt.wr = 0;
        nxt.end = k >= nitem;
        if (!nxt.end) {
            locate(k, nxt);
            nxt.lo = __ldg(nxt.plo);
        }
#pragma unroll
        for (int l = 0; l < P::NLANE; l++) {
            dnxt[l].offset = dnxt[l].valid = 0;
            if ((nxt.has >> l) & 1) {
                const int4* src = reinterpret_cast<const int4*>(nxt.d + l);
                reinterpret_cast<int4*>(&dnxt[l])[0] = __ldg(src);
                reinterpret_cast<int4*>(&dnxt[l])[1] = __ldg(src + 1);
            }
        }
        if (t == 0) {
            PairLoc& S = s.loc[i & 3];
            S.out = nxt.out;
            S.out_b = nxt.out_b;
            S.wr = nxt.wr;
            S.end = nxt.end;
        }
    };
    // the words with the samples that a lane expands, from global memory: those alone that hold needed bits
    auto words = [&](Words (&a)[NG]) {
#pragma unroll
        for (int l = 0; l < P::NLANE; l++) {
            const long long bit = (long long)dnxt[l].offset * SB;
            nxt.bit[l] = (int)bit & 31;
            const uint32_t* wp = reinterpret_cast<const uint32_t*>(nxt.row) + (bit >> 5) + NPOL * t;
            const bool on = dnxt[l].valid;
#pragma unroll
            for (int g = 0; g < NG; g++)
#pragma unroll
                for (int k = 0; k < NPOL + 1; k++) {
                    uint32_t w = 0;   // (volatile: here, not where the word is used)
                    if (on && (k < NPOL || nxt.bit[l]))
                        asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(w) : "l"(wp + 32 * NPOL * g + k));
                    a[g].w[2 * l + k] = w;
                }
        }
        nxt.valid = 0;
#pragma unroll
        for (int l = 0; l < P::NLANE; l++) nxt.valid |= dnxt[l].valid ? 1 << l : 0;
    };
    if constexpr (P::R32) {
        if (helper) load(0, ticket);
    } else if (t == 0) {
        fetch(0);
        fetch(1);
    }
    // ---- constant tables of the CTA
    if constexpr (P::R32) {
        for (int e = threadIdx.x; e < 16 * NT; e += P::NTHREADS) {
            const float4 w = pass_w(e / NT, e % NT, 32 * P::H0);
            sm.wbc[e] = make_float2(w.x, w.y);
        }
    } else {
        for (int e = threadIdx.x; e < 128; e += P::NTHREADS) sm.w1c[e] = pass_w(e >> 4, e & 15, 16);
    }
    for (int e = threadIdx.x; e < P::D2 * 256; e += P::NTHREADS) {
        const float4 w = pass_w(e >> 8, e & 255, 256);
        sm.w2c[e] = make_float2(w.x, w.y);
    }
    if (threadIdx.x < 16) sm.lut[threadIdx.x] = make_float2(level2bit(threadIdx.x & 3), level2bit(threadIdx.x >> 2));
    if (threadIdx.x < (P::R32 ? 16 * P::H0 : 8)) sm.w0c[threadIdx.x] = pass_w(threadIdx.x & 15, threadIdx.x >> 4, P::H0);
    if (!P::R32 && t == 0) {
        stg_bar_init(&s.bar);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (!P::R32 && t == 0) {
        entries_wait();
        describe(s.loc[0], s.dent[0]);
        copy(s.loc[0]);
        describe(s.loc[1], s.dent[1]);
        fetch(2);
    }
    __syncthreads();
    // R32: the helper meets the slot's threads before pass 0 (a pair is prepared) and after it (the samples and the
    // twiddles of pass 0 are free)
    auto meet = [&] { asm volatile("bar.sync %0, %1;" ::"r"(slot + 1), "r"(NT + 32) : "memory"); };
    if constexpr (P::R32) {
        if (helper) {
            asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(P::R_HELP));
            const bool any = !nxt.end;
            int ahead = 0;   // lane 1: the ticket of pair i + 3, drawn one pair earlier
            for (int i = -1; !nxt.end; i++) {   // nxt is pair i + 1
                Words a[NG];
                if (i >= 0) meet();
                words(a);
                factors(i + 1, nxt, dnxt);
                if (i >= 0) meet();
                __syncwarp();
                expand_w(nxt, a);
                twiddles(i + 1);
                const int k = __shfl_sync(0xffffffffu, ahead, 1);
                if (drawn && i >= 0 && t == 1) ahead = 3 * nwork + atomicAdd(ctr, 1);
                load(i + 2, i < 1 || !drawn ? ticket + (i + 2) * nwork : k);
            }
            if (any) {   // the last pair
                meet();
                meet();
            }
            __syncwarp();   // lane 1's last draw comes before lane 0's fence
            finish();
            return;
        }
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(P::R_COMP));
    } else {
    factors(0, s.loc[0], s.dent[0]);
    pair_sync<NT>(slot);
    if constexpr (!CPX) {
        bytes_wait(s.loc[0]);
        expand(s.loc[0]);
    }
    twiddles(0);
    pair_sync<NT>(slot);
    if constexpr (!CPX)
        if (t == 0) copy(s.loc[1]);
    }

    const float4* buf_t = s.buf + padi(t);
    float4* row_t = s.buf + 272 * (t >> 4);   // exchange rows of the threads with this d0
    const int u = t & 15;
    const int n0 = CPX ? t : u * (NT / 16) + (t >> 4);   // samples n0 + r NT in pass 0
    const uint8_t* xs_t = s.xs + (n0 ^ (((n0 >> 7) & SWZ) << 2));

    for (int i = 0; !s.loc[i & 3].end; i++) {
        const PairLoc& L = s.loc[i & 3];
        const bool more = !s.loc[(i + 1) & 3].end;
        const Fe* tab = s.tab[i & (P::NTABS - 1)];
        c2 v[P::R32 ? 32 : 16];
        auto next = [&] {
            if (more) {
                if constexpr (!CPX) {
                    bytes_wait(s.loc[(i + 1) & 3]);
                    expand(s.loc[(i + 1) & 3]);
                }
                twiddles(i + 1);
            }
            pair_sync<NT>(slot);
            if constexpr (!CPX)
                if (t == 0) copy(s.loc[(i + 2) & 3]);
        };
        if constexpr (P::R32) {
            // ---- stage 0 on real samples (output h of two: x +- rho x'), stages 1 to 4 + H0 of thread tp's 32 H0
            // samples, one of its H0 sets of 32 outputs k1 = h + H0 r
            constexpr int G = NT / P::H0;
            meet();
            const int h = t / G, tp = t % G;
            const c2 r0 = fac(Fac<NPOL>::rho(tab[0]));
            const unsigned char* lut = reinterpret_cast<const unsigned char*>(sm.lut);
            const uint8_t* xp = s.xs + tp;
            auto level = [&](int n) { return *reinterpret_cast<const float2*>(lut + xp[n]); };
            if constexpr (P::H0 == 2) {
                const c2 rs = h ? c2{neg2(r0.x), neg2(r0.y)} : r0;
#pragma unroll
                for (int r = 0; r < 32; r++) {
                    const float2 x = level(r * G), x1 = level(r * G + F / 2);
                    v[r].x = __ffma2_rn(rs.x, x1, x);
                    v[r].y = __fmul2_rn(rs.y, x1);
                }
                butterfly<32, 0, false>(v, [&](int d) { return fac(s.w0[16 * h + d]); });
            } else {
                const float2 m2 = make_float2(-2.f, -2.f);
#pragma unroll
                for (int r = 0; r < 16; r++) {
                    const float2 x = level(r * G), x1 = level((r + 16) * G);
                    v[r].x = __ffma2_rn(r0.x, x1, x);
                    v[r].y = __fmul2_rn(r0.y, x1);
                    v[r + 16].x = __ffma2_rn(x, m2, v[r].x);
                    v[r + 16].y = v[r].y;
                }
                butterfly<32, 1, false>(v, [&](int d) { return fac(s.w0[d]); });
            }
            meet();
            // ---- exchange: rows k1 of G + 1; pass 1 takes row t
#pragma unroll
            for (int r = 0; r < 32; r++) s.buf[(h + P::H0 * r) * (G + 1) + tp] = as_f4(v[bitrev(r, 5)]);
            if constexpr (NT > 32) asm volatile("bar.sync %0, %1;" ::"r"(P::NSLOT + slot + 1), "n"(NT) : "memory");
            else __syncwarp();
#pragma unroll
            for (int r = 0; r < 32; r++) v[r] = as_c2(s.buf[t * (G + 1) + r]);
            butterfly<32, 0, true>(v, [&](int d) {
                return fac(Fac<NPOL>::mul(tab[4 + P::H0 + stage_of(d)], sm.wbc[NT * d + t]));
            });
        } else {
        // (not indented: the plan with an exchange per pass)
        // ---- pass 0
        {
            const c2 r0 = fac(Fac<NPOL>::rho(tab[0]));
            if constexpr (CPX) {
                bytes_wait(L);
                // int8 (re, im): bytes to floats by the 2^23 + 2^7 + value form, exact
                auto conv = [](uint32_t w, uint32_t sel) { return __uint_as_float(__byte_perm(w, 0x4B000000u, sel)); };
                const float2 off = make_float2(-8388736.f, -8388736.f);
#pragma unroll
                for (int r = 0; r < 16; r++) {
                    uint32_t w;   // (re A, im A, re B, im B)
                    if constexpr (NPOL == 2) {
                        w = *reinterpret_cast<const uint32_t*>(s.inb[0] + (L.bit[0] >> 3) + 4 * (n0 + r * NT));
                    } else {
                        const uint32_t wa = *reinterpret_cast<const uint16_t*>(s.inb[0] + (L.bit[0] >> 3) + 2 * (n0 + r * NT));
                        const uint32_t wb = *reinterpret_cast<const uint16_t*>(s.inb[1] + (L.bit[1] >> 3) + 2 * (n0 + r * NT));
                        w = wa | (wb << 16);
                    }
                    w ^= 0x80808080u;
                    v[r].x = __fadd2_rn(make_float2(conv(w, 0x7440), conv(w, 0x7442)), off);
                    v[r].y = __fadd2_rn(make_float2(conv(w, 0x7441), conv(w, 0x7443)), off);
                }
                butterfly<16, 0, false>(v, [&](int d) { return d == 0 ? r0 : fac(s.w0[d]); });
            } else {
                const unsigned char* lut = reinterpret_cast<const unsigned char*>(sm.lut);
#pragma unroll
                for (int r = 0; r < 16; r++) v[r].x = *reinterpret_cast<const float2*>(lut + xs_t[r * NT]);
                // stage 0 on real samples: x + rho x', and -(x - rho x') with the same imaginary part
                const float2 m2 = make_float2(-2.f, -2.f);
#pragma unroll
                for (int r = 0; r < 8; r++) {
                    const float2 x = v[r].x, xp = v[r + 8].x;
                    v[r].x = __ffma2_rn(r0.x, xp, x);
                    v[r].y = __fmul2_rn(r0.y, xp);
                    v[r + 8].x = __ffma2_rn(x, m2, v[r].x);
                    v[r + 8].y = v[r].y;
                }
                butterfly<16, 1, false>(v, [&](int d) { return fac(s.w0[d]); });
            }
        }
        if constexpr (!CPX)
            if (more) factors(i + 1, s.loc[(i + 1) & 3], s.dent[(i + 1) & 3]);
        pair_sync<NT>(slot);   // the exchange buffer, the samples and the twiddles of pass 0 are free
        if (t == 0) {
            entries_wait();
            describe(s.loc[(i + 2) & 3], s.dent[(i + 2) & 3]);
            fetch(i + 3);
            if constexpr (CPX) copy(s.loc[(i + 1) & 3]);
        }
        // ---- exchange and pass 1
        if constexpr (CPX) {
            if (more) factors(i + 1, s.loc[(i + 1) & 3], s.dent[(i + 1) & 3]);
#pragma unroll
            for (int r = 0; r < 16; r++) s.buf[17 * t + r] = as_f4(v[bitrev(r, 4)]);
            pair_sync<NT>(slot);
            constexpr int STEP16 = F / 16 + F / 256;
#pragma unroll
            for (int r = 0; r < 16; r++) v[r] = as_c2(buf_t[r * STEP16]);
            pair_sync<NT>(slot);
        } else {
#pragma unroll
            for (int r = 0; r < 16; r++) row_t[17 * u + r] = as_f4(v[bitrev(r, 4)]);
            __syncwarp();
#pragma unroll
            for (int r = 0; r < 16; r++) v[r] = as_c2(row_t[17 * r + u]);
            __syncwarp();
        }
        constexpr bool LAST1 = P::NPASS == 2;
        if constexpr (P::W1TAB) {
            butterfly<16, 0, LAST1 && !CPX>(v, [&](int d) { return fac(s.w1[i & 1][16 * d + u]); });
        } else {
            butterfly<16, 0, LAST1 && !CPX>(v, [&](int d) {
                const int q = d == 0 ? 0 : d == 1 ? 1 : d < 4 ? 2 : 3;
                return fac(mul_hl(tab[4 + q], sm.w1c[16 * d + u]));
            });
        }
        if constexpr (P::NPASS > 2) {
#pragma unroll
            for (int r = 0; r < 16; r++) row_t[17 * r + u] = as_f4(v[bitrev(r, 4)]);
        }
        if constexpr (P::NPASS > 2) next();
        // ---- pass 2
        constexpr int R2 = P::R2 ? P::R2 : 16;
        constexpr int NB2 = 16 / R2;
        if constexpr (P::NPASS > 2) {
            constexpr int ST = F / R2 + F / R2 / 16;
            constexpr bool LO2 = P::NPASS == 3 && !CPX;
#pragma unroll
            for (int b = 0; b < NB2; b++)
#pragma unroll
                for (int r = 0; r < R2; r++) v[b * R2 + r] = as_c2(buf_t[b * (NT + NT / 16) + r * ST]);
            if constexpr (P::NPASS > 3) pair_sync<NT>(slot);
#pragma unroll
            for (int b = 0; b < NB2; b++) {
                const int jm = (t + b * NT) & 255;
                butterfly<R2, 0, LO2>(v + b * R2, [&](int d) {
                    const int q = d == 0 ? 0 : d == 1 ? 1 : d < 4 ? 2 : 3;
                    return fac(Fac<NPOL>::mul(tab[8 + q], sm.w2c[256 * d + jm]));
                });
            }
        }
        // ---- pass 3 (8192 points): radix 2, w = rho W8192^t W16^b
        if constexpr (P::NPASS > 3) {
            float4* p = s.buf + padi((t >> 8) * 4096 + (t & 255));
#pragma unroll
            for (int r = 0; r < 16; r++) p[272 * r] = as_f4(v[bitrev(r, 4)]);
            pair_sync<NT>(slot);
            constexpr int ST = F / 2 + F / 32;
            const Fe wt = Fac<NPOL>::mul(tab[12], wlast);
#pragma unroll
            for (int b = 0; b < 4; b++) {
                const c2 w = fac(b == 0 ? wt : Fac<NPOL>::by(wt, w16(b)));
                c2 lo = as_c2(buf_t[b * (NT + NT / 16)]), hi = as_c2(buf_t[b * (NT + NT / 16) + ST]);
                bfly_lo(lo, hi, w);
                v[2 * b] = lo;
                lo = as_c2(buf_t[(b + 4) * (NT + NT / 16)]);
                hi = as_c2(buf_t[(b + 4) * (NT + NT / 16) + ST]);
                bfly_lo_mi(lo, hi, w);
                v[2 * (b + 4)] = lo;
            }
        }
        }
        // ---- constant phase, fractional-sample correction and sign; store channels t + NT e
        {
            constexpr int RL = P::R32 ? 32 : P::LASTR, NBL = P::R32 ? 1 : 16 / RL, ML = ilog2c(RL);
            const Fe* El = tab + P::LOGF;
            const Fe* G = El + 16 + P::HI;
            float2 ea, eb;   // E of lanes A and B
            if constexpr (NPOL == 2) {
                ea = El[u];
                if constexpr (P::HI > 1) ea = cmul(ea, El[16 + (t >> 4)]);
                eb = ea;
            } else {
                c2 E = as_c2(El[u]);
                if constexpr (P::HI > 1) E = cmul2(E, as_c2(El[16 + (t >> 4)]));
                ea = make_float2(E.x.x, E.y.x);
                eb = make_float2(E.x.y, E.y.y);
            }
            const bool wa = L.wr & 1, wb = L.wr & 2;
            unsigned char* oa = L.out;
            unsigned char* ob = oa + L.out_b;
#pragma unroll
            for (int b = 0; b < NBL; b++)
#pragma unroll
                for (int r = 0; r < (CPX ? RL : RL / 2); r++) {
                    const int e = b + NBL * r;
                    const c2 y = v[b * RL + bitrev(r, ML)];
                    float2 fa, fb;   // lane A's and B's factor
                    if constexpr (NPOL == 2) {
                        fa = fb = cmul(ea, G[e]);
                    } else {
                        const c2 f = cmul2(c2{make_float2(ea.x, eb.x), make_float2(ea.y, eb.y)}, as_c2(G[e]));
                        fa = make_float2(f.x.x, f.y.x);
                        fb = make_float2(f.x.y, f.y.y);
                    }
                    const float2 ya = cmul(fa, make_float2(y.x.x, y.y.x));
                    const float2 yb = cmul(fb, make_float2(y.x.y, y.y.y));
                    if constexpr (MODE == kSpecP32) {   // both lanes side by side (stored or not together)
                        if (wa) reinterpret_cast<float4*>(oa)[t + NT * e] = make_float4(ya.x, ya.y, yb.x, yb.y);
                    } else if constexpr (MODE == kSpecF32) {
                        if (wa) reinterpret_cast<float2*>(oa)[t + NT * e] = ya;
                        if (wb) reinterpret_cast<float2*>(ob)[t + NT * e] = yb;
                    } else {
                        if (wa) reinterpret_cast<__half2*>(oa)[t + NT * e] = __floats2half2_rn(ya.x, ya.y);
                        if (wb) reinterpret_cast<__half2*>(ob)[t + NT * e] = __floats2half2_rn(yb.x, yb.y);
                    }
                }
        }
        if constexpr (P::NPASS == 2) next();
    }
    if constexpr (!P::R32) finish();
}

// Pair p of (subband sb, antenna ant) from chunk slot tb0 on: both polarisations of slot tb0 + p, or
// slots tb0 + 2 p and the next.
template <int F, int MODE, int NPOL, bool CPX>
__device__ __forceinline__ void pair_locate(const FArgs& a, int sb, int ant, int tb0, int p, int span, PairLoc& L)
{
    using P = PPlan<F, NPOL, CPX>;
    constexpr size_t EB = MODE == kSpecH16 ? sizeof(__half2) : sizeof(float2);
    const int tc = NPOL == 2 ? tb0 + p : tb0 + 2 * p;
    L.row = a.data + ((size_t)sb * a.nant + ant) * a.pitch;
    L.d = a.dtab + (size_t)ant * a.ld + a.t_base + tc;
    // P32: pairs [sb][ant][T][chan][2 polarisations], or [sb][ant][T / 2][chan][2 FFTs] (tc is even)
    const size_t slot = MODE == kSpecP32 && NPOL == 2 ? ((size_t)sb * a.nant + ant) * NPOL * a.T + 2 * (size_t)tc
                                                      : ((size_t)sb * a.nant + ant) * NPOL * a.T + tc;
    L.out = reinterpret_cast<unsigned char*>(a.spec) + slot * P::C * EB;
    L.out_b = (NPOL == 2 ? (size_t)a.T : 1) * P::C * EB;
    L.plo = a.sb_lo + sb;
    L.chalf = a.chalf;
    L.err = a.err;
    L.has = (tc < a.nfft ? 1 : 0) | (NPOL == 1 && tc + 1 < a.nfft ? 2 : 0);
    L.wr = (tc < span ? 1 : 0) | ((NPOL == 2 ? tc < span : tc + 1 < span) ? 2 : 0);
}

// Single job: nsb x nant rows of pairs.
template <int F, int MODE, int NPOL, bool CPX>
__global__ void __launch_bounds__(PPlan<F, NPOL, CPX>::NTHREADS, PPlan<F, NPOL, CPX>::MINB)
k_fpair(FArgs args)
{
    extern __shared__ __align__(16) unsigned char smem[];
    auto& sm = *reinterpret_cast<PairSmem<F, NPOL, CPX>*>(smem);
    const int span = args.tspan ? args.tspan : args.T;
    const int npr = NPOL == 2 ? span : (span + 1) / 2;
    pair_worker<F, MODE, NPOL, CPX>(sm, args.nsb * args.nant * npr, args.ctr, [&](int g, PairLoc& L) {
        const int row = g / npr;
        pair_locate<F, MODE, NPOL, CPX>(args, row / args.nant, row % args.nant, 0, g - row * npr, span, L);
    });
}

// Many jobs: tasks {job, subband, antenna, first slot} of tb slots each; every job of the launch has this F, NPOL
// and spectra layout, each its own FArgs (2-bit real input).
template <int F, int MODE, int NPOL>
__global__ void __launch_bounds__(PPlan<F, NPOL, false>::NTHREADS, PPlan<F, NPOL, false>::MINB)
k_fpair_batch(const FArgs* __restrict__ jobs, const int4* __restrict__ tasks, int ntask, int tb, int* ctr)
{
    extern __shared__ __align__(16) unsigned char smem[];
    auto& sm = *reinterpret_cast<PairSmem<F, NPOL, false>*>(smem);
    const int npr = NPOL == 2 ? tb : tb / 2;
    pair_worker<F, MODE, NPOL, false>(sm, ntask * npr, ctr, [&](int g, PairLoc& L) {
        const int4 tk = tasks[g / npr];
        const FArgs& a = jobs[tk.x];
        pair_locate<F, MODE, NPOL, false>(a, tk.y, tk.z, tk.w, g % npr, a.tspan ? a.tspan : a.T, L);
    });
}

// Persistent grid: as many CTAs as are resident, or as hold a pair per slot.
template <typename Kern>
cudaError_t pair_grid(Kern kern, int nthreads, int nslot, size_t sm, long long nitem, unsigned* configured, int* grid)
{
    cudaError_t e = set_smem_once(kern, sm, configured);
    if (e != cudaSuccess) return e;
    int dev = 0, nsm = 0, per_sm = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, nthreads, sm)) != cudaSuccess) return e;
    if (nitem < 1 || nitem > 0x7fffffffLL - (1 << 24)) return cudaErrorInvalidValue;   // pair numbers are ints
    const long long want = (nitem + nslot - 1) / nslot;
    *grid = (int)std::max(1LL, std::min(want, (long long)nsm * std::max(1, per_sm)));
    return cudaSuccess;
}

template <int F, int MODE, int NPOL, bool CPX>
cudaError_t launch_pair(const FArgs& a, cudaStream_t st)
{
    using P = PPlan<F, NPOL, CPX>;
    const size_t sm = sizeof(PairSmem<F, NPOL, CPX>);
    static unsigned configured = 0;
    const int span = a.tspan ? a.tspan : a.T;
    const long long nitem = (long long)a.nsb * a.nant * (NPOL == 2 ? span : (span + 1) / 2);
    int grid = 0;
    const cudaError_t e = pair_grid(k_fpair<F, MODE, NPOL, CPX>, P::NTHREADS, P::NSLOT, sm, nitem, &configured, &grid);
    if (e != cudaSuccess) return e;
    k_fpair<F, MODE, NPOL, CPX><<<grid, P::NTHREADS, sm, st>>>(a);
    return cudaGetLastError();
}

template <int F, int MODE, int NPOL>
cudaError_t launch_pair_batch(const FArgs* d_jobs, const int4* d_tasks, int ntask, int tb, int* ctr, cudaStream_t st)
{
    using P = PPlan<F, NPOL, false>;
    const size_t sm = sizeof(PairSmem<F, NPOL, false>);
    static unsigned configured = 0;
    const long long nitem = (long long)ntask * (NPOL == 2 ? tb : tb / 2);
    int grid = 0;
    const cudaError_t e = pair_grid(k_fpair_batch<F, MODE, NPOL>, P::NTHREADS, P::NSLOT, sm, nitem, &configured, &grid);
    if (e != cudaSuccess) return e;
    k_fpair_batch<F, MODE, NPOL><<<grid, P::NTHREADS, sm, st>>>(d_jobs, d_tasks, ntask, tb, ctr);
    return cudaGetLastError();
}

// Entry points of one FFT length, instantiated in its own translation unit.
template <int F>
cudaError_t launch_fstage_F(int mode, const FArgs& a, cudaStream_t st)
{
    if constexpr (F <= 4096) if (a.cpx) {   // complex FFT length = nchan <= 4096
        if (mode == kSpecF32)
            return a.npol == 2 ? launch_pair<F, kSpecF32, 2, true>(a, st) : launch_pair<F, kSpecF32, 1, true>(a, st);
        if (mode == kSpecP32)
            return a.npol == 2 ? launch_pair<F, kSpecP32, 2, true>(a, st) : launch_pair<F, kSpecP32, 1, true>(a, st);
        return a.npol == 2 ? launch_pair<F, kSpecH16, 2, true>(a, st) : launch_pair<F, kSpecH16, 1, true>(a, st);
    }
    if (mode == kSpecF32)
        return a.npol == 2 ? launch_pair<F, kSpecF32, 2, false>(a, st) : launch_pair<F, kSpecF32, 1, false>(a, st);
    if (mode == kSpecP32)
        return a.npol == 2 ? launch_pair<F, kSpecP32, 2, false>(a, st) : launch_pair<F, kSpecP32, 1, false>(a, st);
    return a.npol == 2 ? launch_pair<F, kSpecH16, 2, false>(a, st) : launch_pair<F, kSpecH16, 1, false>(a, st);
}

template <int F>
cudaError_t launch_fstage_batch_F(int mode, int npol, int tb, const FArgs* d_jobs, const int4* d_tasks, int ntask,
                                  int* ctr, cudaStream_t st)
{
    if (mode == kSpecF32)
        return npol == 2 ? launch_pair_batch<F, kSpecF32, 2>(d_jobs, d_tasks, ntask, tb, ctr, st)
                         : launch_pair_batch<F, kSpecF32, 1>(d_jobs, d_tasks, ntask, tb, ctr, st);
    if (mode == kSpecP32)
        return npol == 2 ? launch_pair_batch<F, kSpecP32, 2>(d_jobs, d_tasks, ntask, tb, ctr, st)
                         : launch_pair_batch<F, kSpecP32, 1>(d_jobs, d_tasks, ntask, tb, ctr, st);
    if (mode != kSpecH16) return cudaErrorInvalidValue;
    return npol == 2 ? launch_pair_batch<F, kSpecH16, 2>(d_jobs, d_tasks, ntask, tb, ctr, st)
                     : launch_pair_batch<F, kSpecH16, 1>(d_jobs, d_tasks, ntask, tb, ctr, st);
}

}  // namespace fx
