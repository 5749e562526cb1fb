// fx_fscalar.cuh -- the F stage of the FP8 form: one FFT per slot in scalar FP32, FP16 spectra out.
//
// The same steps as fx_fpair.cuh (kernel.c:397-555), with separate rotator tables, 2-bit decode per sample and
// register-resident radix-16 butterflies with one twiddle multiply per pass.  The FP8 form scales by the
// exact absmax of a chunk and rounds to 4 bits: a last-bit difference of a spectrum moves whole e4m3 steps
// (on fx_fpair.cuh's butterflies visibilities change by 3.5e-5 of their norm, more than this library lets a form's
// results move between versions), so that form keeps this arithmetic, operation by operation, though not for good one
// FFT to a slot: two in packed lanes with these operations in this order would round the same.
// Bound by instruction issue (75 instructions per sample), 1.4 to 1.7 times the F-stage time of the pairs (FP32
// spectra: 64 antennas x 8 subbands x 31250 FFTs of 2048 points 89.7 / 65.5 ms, 23 antennas x 3 subbands x 2777 of
// 1024 points 0.611 / 0.351).
#pragma once

#include "fx_fstage.cuh"

namespace fx {

template <int F, bool CPX = false>
struct SPlan : FPlan<F, CPX> {
    using P = FPlan<F, CPX>;
    static constexpr int NROT = P::S + P::STRIDE + P::FS + P::FST;   // rotator table entries
    static constexpr int BUF = F + F / 16;                    // padded exchange buffer (float2)
    static constexpr bool TWREG = (F <= 2048);                // twiddles cached in registers
    // pass twiddle tables in shared memory (F > 2048): W256^(r j) [r][j] for pass 1, W4096^(r l) [r][l]
    // and W4096^(16 r h) [r][h] for pass 2 (j = 16 h + l), and for 8192 points W8192^(64 h) [h], W8192^l
    // [l] for pass 3 (j = 64 h + l): a warp's twiddle loads are consecutive or broadcast words
    static constexpr int TWP = 3 * 256 + (F == 8192 ? 128 : 0);
};

template <int F, int PASS>
struct PassInfo {
    static constexpr int R = (PASS == SPlan<F>::NPASS - 1) ? SPlan<F>::LASTR : 16;
    static constexpr int NS = 1 << (4 * PASS);               // 16^PASS
    static constexpr int NB = 16 / R;                         // butterflies per thread
};

// e^{-2 pi i m / F} for 0 <= m < F: the first-quadrant value e^{-2 pi i m'/F} (m' = m mod F/4)
// turned by the quadrant (exact: swaps and negations)
template <int F>
__device__ __forceinline__ float2 twiddle_q(int m)
{
    const int q = m / (F / 4);
    const float2 b = twiddle_exact(m & (F / 4 - 1), F);
    switch (q & 3) {
    case 0: return b;
    case 1: return make_float2(b.y, -b.x);
    case 2: return make_float2(-b.x, -b.y);
    default: return make_float2(-b.y, b.x);
    }
}

template <int NT>
__device__ __forceinline__ void slot_sync(int slot)
{
    if constexpr (NT >= 32) {
        asm volatile("bar.sync %0, %1;" ::"r"(slot + 1), "r"(NT) : "memory");
    } else {
        __syncwarp();
    }
}

// Copy `bytes` (16-byte multiple, both addresses 16-byte aligned) from global src to shared dst.
// The issuing thread orders the slot's earlier reads of dst (made visible to it by a barrier)
// before the async-proxy write.
__device__ __forceinline__ void stg_issue(uint64_t* bar, void* dst, const void* src, uint32_t bytes)
{
    size_t gsrc;
    asm volatile("cvta.to.global.u64 %0, %1;" : "=l"(gsrc) : "l"(src));
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32a(bar)), "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32a(dst)), "l"(gsrc), "r"(bytes), "r"(smem_u32a(bar))
                 : "memory");
}

// Twiddles a thread needs for pass PASS (r = 0..R-1 of each of its NB butterflies).
template <int F, int PASS>
struct PassTw {
    float2 w[PassInfo<F, PASS>::NB * PassInfo<F, PASS>::R];
};

template <int F, int PASS>
__device__ __forceinline__ void init_pass_tw(PassTw<F, PASS>& tw, int t)
{
    using PI = PassInfo<F, PASS>;
#pragma unroll
    for (int b = 0; b < PI::NB; b++) {
        const int j = t + b * SPlan<F>::NT;
        const int jm = j & (PI::NS - 1);
#pragma unroll
        for (int r = 0; r < PI::R; r++) tw.w[b * PI::R + r] = twiddle_exact(r * jm, PI::NS * PI::R);
    }
}

// Load pass inputs from the exchange buffer and apply the DIT twiddles.  All
// offsets are multiples of 16 elements, so padi(t + c) = padi(t) + c + c/16 and
// every shared-memory access is one base register plus an immediate.
template <int F, int PASS>
__device__ __forceinline__ void pass_load(const float2* buf, const float2* tp, const PassTw<F, PASS>* tw,
                                          float2* v, int t)
{
    using PI = PassInfo<F, PASS>;
    constexpr int NT = SPlan<F>::NT;
    constexpr int STEP = F / PI::R;
    static_assert(STEP % 16 == 0 && NT % 16 == 0, "padded offsets must fold");
    const float2* p0 = buf + padi(t);
#pragma unroll
    for (int b = 0; b < PI::NB; b++) {
        const int jm = (t + b * NT) & (PI::NS - 1);
        const float2* p = p0 + b * (NT + NT / 16);
#pragma unroll
        for (int r = 0; r < PI::R; r++) {
            float2 x = p[r * (STEP + STEP / 16)];
            if (r > 0) {
                float2 w;
                if constexpr (SPlan<F>::TWREG) w = tw->w[b * PI::R + r];
                else if constexpr (PI::NS == 16 && PI::R == 16) w = tp[16 * r + jm];
                else if constexpr (PI::NS == 256 && PI::R == 16)
                    w = cmul(tp[512 + 16 * r + (jm >> 4)], tp[256 + 16 * r + (jm & 15)]);
                else {
                    static_assert(PI::NS == 4096 && PI::R == 2, "every pass of F > 2048 has its table");
                    w = cmul(tp[768 + (jm >> 6)], tp[832 + (jm & 63)]);
                }
                x = cmul(x, w);
            }
            v[b * PI::R + r] = x;
        }
    }
}

template <int F, int PASS>
__device__ __forceinline__ void pass_dft(float2* v)
{
    using PI = PassInfo<F, PASS>;
#pragma unroll
    for (int b = 0; b < PI::NB; b++) dft<PI::R>(v + b * PI::R);
}

// Stockham store: element r of butterfly j goes to (j / NS) * NS * R + j % NS + r * NS.
template <int F, int PASS>
__device__ __forceinline__ void pass_store(float2* buf, const float2* v, int t)
{
    using PI = PassInfo<F, PASS>;
    constexpr int NT = SPlan<F>::NT;
#pragma unroll
    for (int b = 0; b < PI::NB; b++) {
        const int j = t + b * NT;
        float2* p;
        constexpr int RS = (PI::NS == 1) ? 1 : PI::NS + PI::NS / 16;   // padded stride of r
        if constexpr (PI::NS == 1) p = buf + 17 * j;                    // padi(16 j)
        else p = buf + padi((j / PI::NS) * PI::NS * PI::R + (j & (PI::NS - 1)));
#pragma unroll
        for (int r = 0; r < PI::R; r++) p[r * RS] = v[b * PI::R + r];
    }
}

// Rotator table of one FFT: [fr_sub S][fr_step STRIDE][fc_sub FS][fc_step FST].
// Entries are (cos, sin)(pi * x) with x in half-turns, which needs no
// large-argument reduction: fringe x = -2 * frac(phase in turns), i.e. the
// reference's argument -2pi*frac(phase) (kernel.c:463-470) divided by pi;
// fractional-sample x = the reference's float32 argument (kernel.c:517-523) / pi.
// Divisions by F are multiplications by the exact power-of-two reciprocal.
constexpr float kInvPiF = 0.318309886183790671538f;

// Rotator argument x (half-turns) of table entry e; the entry is (cos, sin)(pi x).
template <int F, bool CPX>
__device__ __forceinline__ float rot_arg(int e, const DelayEntry& d, double lo, double lofrac, bool fraclo,
                                         const float* ctab)
{
    using P = SPlan<F, CPX>;
    constexpr double kInvF = 1.0 / F;
    if (e < P::S) {
        // kernel.c:434-466: subphase[j] = lo * (j/F * a + b'), b' = b - (int)b
        const double intdelay = trunc(d.b);
        const double bp = dsub(d.b, intdelay);
        const double xoff = dmul((double)e, kInvF);
        double ph = dmul(dadd(dmul(xoff, d.a), bp), lo);
        if (fraclo) ph = dadd(ph, dmul(lofrac, intdelay));
        return __double2float_rn(-2.0 * dsub(ph, trunc(ph)));
    } else if (e < P::S + P::STRIDE) {
        // kernel.c:145, 452, 469: stepphase[i] = lo * (i*stride/F * a)
        const double xoff = dmul((double)((e - P::S) * P::STRIDE), kInvF);
        const double ph = dmul(dmul(xoff, d.a), lo);
        return __double2float_rn(-2.0 * dsub(ph, trunc(ph)));
    } else {
        const float arg = __fmul_rn(ctab[e - P::S - P::STRIDE], __double2float_rn(d.frac));
        return __fmul_rn(arg, kInvPiF);
    }
}

template <int F, bool CPX>
__device__ __forceinline__ float2 rot_entry(int e, const DelayEntry& d, double lo, double lofrac, bool fraclo,
                                            const float* ctab)
{
    float sn, cs;
    sincospif(rot_arg<F, CPX>(e, d, lo, lofrac, fraclo, ctab), &sn, &cs);
    return make_float2(cs, sn);
}

template <int F>
using Tw2Of = PassTw<F, (SPlan<F>::NPASS > 2 ? 2 : 1)>;

// The slots' staging mbarriers: 16 bytes per slot after the channel table.
template <int F, bool CPX>
__device__ __forceinline__ uint64_t* fstage_bars(unsigned char* smem)
{
    using P = SPlan<F, CPX>;
    float2* rtabs = reinterpret_cast<float2*>(smem) + P::NSLOT * P::BUF + (P::TWREG ? 0 : P::TWP);
    return reinterpret_cast<uint64_t*>(reinterpret_cast<float*>(rtabs + 2 * P::NSLOT * P::NROT) + P::FS + P::FST);
}

template <int F, int TB, int NPOL, bool CPX>
__device__ __forceinline__ void fstage_block(const FArgs& args, int sb, int ant, int tb0, unsigned char* smem,
                                             const PassTw<F, 1>& tw1, const Tw2Of<F>& tw2, uint32_t& phase)
{
    using P = SPlan<F, CPX>;
    constexpr int NT = P::NT;
    constexpr int C = P::C;
    constexpr int INB = fstage_inb<F, NPOL, CPX>();                    // staged bytes per slot
    float2* bufs = reinterpret_cast<float2*>(smem);                   // [NSLOT][BUF]
    float2* tq = bufs + P::NSLOT * P::BUF;                              // [TWP] pass twiddle tables
    float2* rtabs = tq + (P::TWREG ? 0 : P::TWP);                      // [NSLOT][2][NROT]
    float* ctab = reinterpret_cast<float*>(rtabs + 2 * P::NSLOT * P::NROT);   // [FS + FST] channel freqs
    uint64_t* bars = reinterpret_cast<uint64_t*>(ctab + P::FS + P::FST);    // [NSLOT] (16 B each)
    uint8_t* inbs = reinterpret_cast<uint8_t*>(bars + 2 * P::NSLOT);        // [NSLOT][INB]
    const int tid = threadIdx.x;
    const int slot = tid / NT;
    const int t = tid - slot * NT;
    float2* buf = bufs + slot * P::BUF;
    // rotator tables alternate between two buffers per slot, so the next FFT's table can be
    // written while this FFT's epilogue still reads its own: no barrier between FFTs
    float2* rtab2 = rtabs + slot * 2 * P::NROT;
    uint8_t* inb = inbs + slot * INB;
    uint64_t* bar = bars + 2 * slot;

    const double lo = args.sb_lo[sb];
    const double lofrac = dsub(lo, trunc(lo));
    const bool fraclo = lofrac > 1e-11;                                  // kernel.c:39

    for (int i = tid; i < P::FS + P::FST; i += P::NTHREADS)
        ctab[i] = i < P::FS ? args.chan_sub[i] : args.chan_step[i - P::FS];
    __syncthreads();

    const uint8_t* row = args.data + ((size_t)sb * args.nant + ant) * args.pitch;
    const int nsig = args.nant * NPOL;
    constexpr int NITEM = TB * NPOL;
    const DelayEntry* dtab = args.dtab + (size_t)ant * args.ld + args.t_base;

    // Input window of an item: 16-byte aligned start, nvec 16-byte vectors (2-bit real:
    // F*NPOL/4 bytes + the read-ahead byte of kernel.c:402-409; 8-bit complex: 2*NPOL bytes
    // per sample), copied into the slot's staging buffer by one bulk copy, issued as soon
    // as the previous item's bytes are decoded so the copy overlaps that item's FFT.
    auto window = [&](const DelayEntry& d, int& base, int& nvec) {
        if constexpr (CPX) {
            const int first = d.offset * 2 * NPOL;
            base = first & ~15;
            nvec = (F * NPOL * 2 + (first - base) + 15) >> 4;
        } else {
            const int first = (NPOL == 2) ? (d.offset >> 1) : (d.offset >> 2);
            base = first & ~15;
            nvec = (F * NPOL / 4 + 1 + (first - base) + 15) >> 4;
        }
    };

    // items (polarisation-major: item = pol * TB + FFT) are dealt to the slots in contiguous runs of SEG
    constexpr int SEG = (NITEM >= P::NSLOT) ? NITEM / P::NSLOT : 1;
    const int item_end = min(slot * SEG + SEG, NITEM);

    // the first item's delay entry and input copy
    int item = slot * SEG;
    DelayEntry dn;
    bool vn = false;
    int basen = 0, nvecn = 0;
    bool expired = false;   // a staging wait gave up (recorded in *args.err)
    if (item < item_end && tb0 + item % TB < args.nfft) {
        dn = dtab[tb0 + item % TB];
        vn = dn.valid != 0;
    }
    if (vn) {
        window(dn, basen, nvecn);
        if (t == 0) stg_issue(bar, inb, row + basen, 16u * nvecn);
    }

    for (; item < item_end; item++) {
        const int pol = item / TB;
        const int tl = item - pol * TB;
        const int tc = tb0 + tl;                    // FFT slot within the chunk
        float2* rtab = rtab2 + ((item - slot * SEG) & 1) * P::NROT;
        const DelayEntry d = dn;
        const bool valid = vn;
        const int base_byte = basen;
        if (valid) {
            if (!stg_wait(bar, phase)) {
                if (t == 0 && args.err) atomicCAS(args.err, 0, 6);
                expired = true;
            }
            phase ^= 1;
        }
        // ---- the next item of this slot: delay entry now, its copy after this item's decode
        {
            const int ni = item + 1;
            vn = false;
            if (ni < item_end && tb0 + ni % TB < args.nfft) {
                dn = dtab[tb0 + ni % TB];
                vn = dn.valid != 0;
            }
            if (vn) window(dn, basen, nvecn);
        }
        // ---- rotator tables for this FFT (per slot)
        for (int e = t; e < P::NROT; e += NT)
            rtab[e] = valid ? rot_entry<F, CPX>(e, d, lo, lofrac, fraclo, ctab) : make_float2(0.f, 0.f);
        slot_sync<NT>(slot);

        // ---- pass 0: unpack + fringe rotation + radix-16 (samples n = t + r*NT)
        float2 v[16];
        {
            // an invalid item reads from the start of the staging buffer (in range;
            // its rotator is zero, so the levels do not matter)
            const int s0 = valid ? d.offset + t : t;
            const int b0 = valid ? base_byte : 0;
            const uint8_t* bp;
            int sh = 0;
            if constexpr (CPX) {
                // 8-bit complex: (re, im) int8 pairs, polarisations interleaved per sample
                bp = inb + (s0 * 2 * NPOL + 2 * pol - b0);
            } else if constexpr (NPOL == 2) {
                bp = inb + ((s0 >> 1) - b0);
                sh = 4 * (s0 & 1) + 2 * pol;
            } else {
                bp = inb + ((s0 >> 2) - b0);
                sh = 2 * (s0 & 3);
            }
            const float2* fr_sub = rtab;
            const float2* fr_step = rtab + P::S;
            float2 sub_c = make_float2(0.f, 0.f);
            const float2* stp = fr_step;
            if constexpr (NT % P::S == 0) {
                sub_c = fr_sub[t % P::S];   // j = n % S is the same for all r
                stp = fr_step + t / P::S;
            }
#pragma unroll
            for (int r = 0; r < 16; r++) {
                float2 rot;
                if constexpr (NT % P::S == 0) {
                    rot = cmul(sub_c, stp[r * (NT / P::S)]);
                } else {
                    const int n = t + r * NT;
                    rot = cmul(fr_sub[n % P::S], fr_step[n / P::S]);
                }
                if constexpr (CPX) {
                    const char2 c8 = *reinterpret_cast<const char2*>(bp + r * (NT * 2 * NPOL));
                    v[r] = cmul(make_float2((float)c8.x, (float)c8.y), rot);
                } else {
                    const uint32_t byte = bp[r * (NT * NPOL / 4)];
                    const float lv = level2bit((byte >> sh) & 3u);
                    v[r] = make_float2(lv * rot.x, lv * rot.y);
                }
            }
        }
        dft<16>(v);
        pass_store<F, 0>(buf, v, t);
        slot_sync<NT>(slot);
        // this item's bytes are decoded: the next item's copy overlaps the rest of its FFT
        if (vn && t == 0) stg_issue(bar, inb, row + basen, 16u * nvecn);

        // ---- middle passes
        if constexpr (P::NPASS > 2) {
            pass_load<F, 1>(buf, tq, &tw1, v, t);
            slot_sync<NT>(slot);
            pass_dft<F, 1>(v);
            pass_store<F, 1>(buf, v, t);
            slot_sync<NT>(slot);
        }
        if constexpr (P::NPASS > 3) {
            pass_load<F, 2>(buf, tq, nullptr, v, t);
            slot_sync<NT>(slot);
            pass_dft<F, 2>(v);
            pass_store<F, 2>(buf, v, t);
            slot_sync<NT>(slot);
        }
        // ---- last pass
        constexpr int LP = P::NPASS - 1;
        using LI = PassInfo<F, LP>;
        if constexpr (LP == 1) pass_load<F, 1>(buf, tq, &tw1, v, t);
        else if constexpr (LP == 2) pass_load<F, 2>(buf, tq, &tw2, v, t);
        else pass_load<F, 3>(buf, tq, nullptr, v, t);
        // real input: outputs r < R/2 only (channels below F/2); complex input: every output
        constexpr int NOUT = CPX ? LI::R : LI::R / 2;
#pragma unroll
        for (int b = 0; b < LI::NB; b++) {
            if constexpr (CPX) dft<LI::R>(v + b * LI::R);
            else dft_lo<LI::R>(v + b * LI::R);
        }

        // ---- fractional-sample correction + store of channels k = j + r*F/R < C
        constexpr int KSTEP = F / LI::R;
        static_assert(KSTEP % P::FS == 0, "frac rotator index must fold");
        const float2* fc_sub = rtab + P::S + P::STRIDE;
        const float2* fc_step = fc_sub + P::FS;
        const int sig = ant * NPOL + pol;
#pragma unroll
        for (int b = 0; b < LI::NB; b++) {
            const int j = t + b * NT;
            const float2 fsub = fc_sub[j % P::FS];
            const float2* fst = fc_step + j / P::FS;
#pragma unroll
            for (int r = 0; r < NOUT; r++) {
                const float2 fr = cmul(fsub, fst[r * (KSTEP / P::FS)]);
                const float2 y = cmul(fr, v[b * LI::R + r]);
                __half2* out = reinterpret_cast<__half2*>(args.spec) + (((size_t)sb * nsig + sig) * args.T + tc) * C + j;
                if (tc < args.T) out[r * KSTEP] = __floats2half2_rn(y.x, y.y);
            }
        }
        // no barrier here: the next FFT writes the other rotator table before its first barrier,
        // and buf only after it (the staging buffer's copy was issued after this FFT's decode)
    }
    // after an expired wait the copy may still land: wait for it once more (bounded) so it
    // cannot write into the staging buffer of a later task or an exited CTA
    if (expired) stg_wait(bar, phase ^ 1);

}

// Per-CTA set-up: the pass twiddle tables (large F) or the thread's register twiddles (F <= 2048).
template <int F>
__device__ __forceinline__ void fstage_prologue(unsigned char* smem, PassTw<F, 1>& tw1, Tw2Of<F>& tw2)
{
    using P = SPlan<F>;
    const int tid = threadIdx.x;
    const int t = tid % P::NT;
    if constexpr (!P::TWREG) {
        float2* tp = reinterpret_cast<float2*>(smem) + P::NSLOT * P::BUF;
        for (int e = tid; e < P::TWP; e += P::NTHREADS) {
            int m;
            if (e < 768) {
                const int k = e >> 8, r = (e >> 4) & 15, j = e & 15;
                m = k == 0 ? r * j * (F / 256) : (k == 1 ? r * j : 16 * r * j) * (F / 4096);
            } else {
                m = e < 832 ? 64 * (e - 768) : e - 832;   // 8192 points, pass 3
            }
            tp[e] = twiddle_q<F>(m);
        }
    } else {
        init_pass_tw<F, 1>(tw1, t);
        if constexpr (P::NPASS > 2) init_pass_tw<F, 2>(tw2, t);
    }
}

// One staging mbarrier per FFT slot, initialised by the slot's first thread before the
// block's first barrier (fstage_block's channel-table __syncthreads) orders it before use.
template <int F, bool CPX>
__device__ __forceinline__ void fstage_bars_init(unsigned char* smem)
{
    using P = SPlan<F, CPX>;
    if (threadIdx.x % P::NT == 0) {
        stg_bar_init(fstage_bars<F, CPX>(smem) + 2 * (threadIdx.x / P::NT));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
}

// Grid (T / TB, nant, nsb).
template <int F, int TB, int NPOL, bool CPX>
__global__ void __launch_bounds__(SPlan<F>::NTHREADS, SPlan<F>::MINB)
k_fscalar(FArgs args)
{
    extern __shared__ __align__(16) unsigned char smem[];
    PassTw<F, 1> tw1;
    Tw2Of<F> tw2;
    fstage_prologue<F>(smem, tw1, tw2);
    fstage_bars_init<F, CPX>(smem);
    uint32_t phase = 0;
    fstage_block<F, TB, NPOL, CPX>(args, blockIdx.z, blockIdx.y, blockIdx.x * TB, smem, tw1, tw2, phase);
}

template <int F, int TB, int NPOL, bool CPX>
cudaError_t launch_scalar_tb(const FArgs& a, cudaStream_t st)
{
    using P = SPlan<F, CPX>;
    const size_t sm = (size_t)P::NSLOT * P::BUF * sizeof(float2) + (P::TWREG ? 0 : (size_t)P::TWP * sizeof(float2)) +
                      (size_t)2 * P::NSLOT * P::NROT * sizeof(float2) + (size_t)(P::FS + P::FST) * sizeof(float) +
                      (size_t)P::NSLOT * 16 + (size_t)P::NSLOT * fstage_inb<F, NPOL, CPX>();
    auto kern = k_fscalar<F, TB, NPOL, CPX>;
    static unsigned configured = 0;  // per instantiation and device
    cudaError_t e = set_smem_once(kern, sm, &configured);
    if (e != cudaSuccess) return e;
    dim3 grid(((a.tspan ? a.tspan : a.T) + TB - 1) / TB, a.nant, a.nsb);
    kern<<<grid, P::NTHREADS, sm, st>>>(a);
    return cudaGetLastError();
}

template <int F, int NPOL, bool CPX>
cudaError_t launch_scalar(const FArgs& a, cudaStream_t st)
{
    // A slot takes the FFTs of its block one after the other: in a short call blocks of 4 use more of the SMs.  16 / 4
    // FFTs a block, us: 8 antennas x 64 FFTs of 8192 points 82 / 33, of 2048 28 / 17; 1024 points take the set-up of a
    // block badly, so only what fits at once: 4 antennas x 256 FFTs 24 / 20, 12 x 256 30 / 34; full SMs 31 / 38.
    if constexpr (F >= 1024) {
        int dev = 0, nsm = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
        const long long blocks = (long long)((a.nfft + 15) / 16) * a.nant * a.nsb;   // with FFTs
        const long long cap = (long long)nsm * SPlan<F, CPX>::MINB;
        if (F == 1024 ? 4 * blocks < cap : 3 * blocks < 2 * cap) return launch_scalar_tb<F, 4, NPOL, CPX>(a, st);
    }
    return launch_scalar_tb<F, 16, NPOL, CPX>(a, st);
}

template <int F>
cudaError_t launch_fscalar_F(const FArgs& a, cudaStream_t st)
{
    if constexpr (F <= 4096)
        if (a.cpx) return a.npol == 2 ? launch_scalar<F, 2, true>(a, st) : launch_scalar<F, 1, true>(a, st);
    return a.npol == 2 ? launch_scalar<F, 2, false>(a, st) : launch_scalar<F, 1, false>(a, st);
}

}  // namespace fx
