// fx_xsplit.cu -- plain X stage on the tensor cores at FP32 grade: every FP32 spectrum value as an FP16 pair of 22
// bits, three of the four products, and sums taken out of the tensor core every 32 FFTs.
//
// Per channel V[i][j] = sum_t X_i conj(X_j) (kernel.c:829-854, conjugation of kernel.c:557-568 folded in).  With
// x = h + l (h = FP16 rounding of x, l of the remainder; 22 bits), rows H = (Re, Im) and H' = (Im, -Re) of the
// high parts and L = (Re, Im) of the low ones, time as the contraction index,
//     D = [H; H'] (H + 2 L)^T     upper 64 rows: real part, lower 64: imaginary part,
//     V = (D + conj(D)^T) / 2 = H H* + H L* + L H*
// (the l l* term is below FP32 rounding), so the low parts enter one side only.
//
// The tensor core adds into its FP32 accumulator by truncation, which adds up: over 1024 FFTs that takes 5e-6
// off every visibility, over 64 FFTs 5e-7, over 32 (two additions of low parts, two of high ones, twice) 2.5e-7.
// So D holds 32 FFTs only; then the epilogue warps add it, rounded to nearest, to running sums in their registers,
// while the MMAs fill the other D, and the mean of what the truncations took, 2^-22, is put back on the way
// out: the mean over Gaussian samples and whole D.  The last D of a call may hold fewer FFTs and lose less (its share
// of the sums is too large by up to 1.5e-7), and sums of few bits lose nothing; calls of less than one D go to
// k_xplain.  After 2048 FFTs at most the sums go to the accumulators: additions to a small sum round less than to a
// large one.  Error of the whole correlation against 64 bits, k_xplain / here (without the 2^-22 / D of
// 16 FFTs with 2^-23 put back, which is 5 % slower):
//     4 antennas x 2 pol, 128 channels, 100 FFTs                               1.4 / 1.0e-7 (2.7 / 0.9e-7)
//     23 antennas, 512 channels, 2 subbands, 1037 FFTs                         3.5 / 1.0e-7 (2.8 / 1.3e-7)
//     16 antennas x 2 pol, 2048 channels, 2 subbands, 8 chunks of 1954 FFTs    1.5 / 1.0e-7 (2.7 / 1.0e-7)
//     24 antennas x 2 pol, 1024 channels, 3000 FFTs of 8-bit complex samples   1.7 / 1.1e-7 (2.8 / 1.3e-7)
//     64 antennas, 1024 channels, 4 subbands, 31250 FFTs                       5.8 / 0.9e-7 (2.6 / 1.0e-7)
//
// Time of the X stage, k_xplain / here: the second 0.411 / 0.316 ms, the third 25.0 / 14.2, the fourth 1.66 /
// 0.79, the fifth 88 / 34 ms.
//
// What bounds it is the chain of one stage: copy in (HBM: 8 bytes per spectrum value, read once), cast, 16 MMAs
// (65 cycles each), flush; shared memory carries all of it: the MMAs' operands, the cast's loads and
// stores, the copies.  12 or 16 cast warps, cast loads straight from global memory, stages of 8 FFTs, sums kept in
// TMEM and MMAs taken in turns from the four tiles all measured the same or slower.
//
// The F stage stores its two lanes side by side for this kernel ([..][chan][2]: two polarisations of an FFT, or
// two FFTs): rows of 64 bytes for 4 channels.  The copy engine moves boxes of 32-byte rows at 3.7 TB/s,
// of 64-byte rows at 6.5.
//
// Persistent, warp-specialised CTA per SM; work item = (subband, CB channels) over the chunk's FFTs: 4
// channels for 33 to 64 signals, one per operand tile, or 8 channels up to 32 signals, two per tile (rows
// H c0, H c1, H' c0, H' c1; the cross blocks of D are not used):
//   warp 0       TMA producer: box {CB channels, 16 FFTs, all signals} of the FP32 spectra into a ring of stages
//                (as many as 96 KB holds); it draws the items
//   warp 1       MMA issuer
//   warps 4-11   cast: a stage of 16 FFTs -> half h of the 4 tiles' rows (while the MMAs read the other).  A
//                thread takes a channel and 4 FFTs of one signal (two polarisations: of both) with 16-byte
//                reads, and stores three 16-byte chunks each, K-major SWIZZLE_128B.  The K order within a chunk
//                is the thread's own (any order does, the same for both operands); signal s of channel c stands
//                in row s ^ (8 / CB) c, so the channels of a quarter warp store to different 16-byte slots.
//   warps 12-19  epilogue: D -> running sums; those through shared memory to acc[sb][pair][chan], one
//                vector addition per pair and channel (two channels at NS = 32).  Additions to acc straight from
//                the registers, a value each, took 85 us per item of 64 signals, of an item's 170.
// Every wait is bounded by time; on expiry the CTA records an error code, drains what it issued (again
// bounded), frees TMEM and returns.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <cuda_fp16.h>

#include <cstring>

#include "fx_common.cuh"
#include "fx_kernels.h"
#include "fx_tc.cuh"

namespace fx {

namespace xsp {

constexpr int KS = 2;                        // K16 steps of a stage
constexpr int BT = 8 * KS;                   // FFTs per stage, a part of the tiles' rows
constexpr int NQ = 4 / KS;                   // parts: D holds the products of all of them, 32 FFTs
constexpr int SEG = 2048;                    // FFTs after which the running sums are sent off at the latest
constexpr int RING_BYTES = 96 * 1024;
constexpr int VROW = 65;                     // floats per row of an item's sums on their way out (odd: columns on all banks)
constexpr int MAXST = 16;
// item numbers handed to the other warps: the producer is at most MAXST stages, the parts of the tiles and
// two D ahead of the last of them, and an item has two stages or more
constexpr int NITEM = 16;
constexpr int NV = 4;                        // tiles
constexpr int HT = 128 * 128, LT = 64 * 128; // tile bytes: 128 (64) rows x NQ stages of (Re, Im) halves
constexpr int NCW = 8, NEW = 8;              // cast and epilogue warps
constexpr int NTHREADS = 32 * (4 + NCW + NEW);   // warp groups: producer and MMA (two warps idle), cast, epilogue
// registers per thread of the three groups; their sum fits what the block is launched with (96 a thread)
constexpr int R_ISSUE = 40, R_CAST = 64, R_EPI = 152;
static_assert(128 * R_ISSUE + 32 * NCW * R_CAST + 32 * NEW * R_EPI <= NTHREADS * 96, "register split");
constexpr int EC = 16;                       // columns the epilogue reads at a time
constexpr int TMEM_COLS = 512;               // two D: 4 x 64 columns each

enum Input { kReal, kComplex, kComplexWide };   // 2-bit real samples; 8-bit complex, up to 1024 channels and beyond

// An item of a batch's launch: what it takes from its job, and where its sums go (first subband and channel added)
struct Item {
    float2* acc;
    int nsig, nchan, nk;
};

struct Smem {
    alignas(1024) uint8_t hi[NV * HT];
    alignas(1024) uint8_t lo[NV * LT];
    alignas(1024) uint8_t ring[RING_BYTES];
    alignas(16) float v[128 * VROW];
    alignas(8) uint64_t full[MAXST];
    uint64_t empty[MAXST];
    uint64_t full16[NQ];                     // per part of the tiles
    uint64_t empty16[NQ];
    uint64_t d_full[2];                      // per D
    uint64_t d_empty[2];
    uint64_t item_full[NITEM];
    uint64_t drain;
    int item[NITEM];                         // the CTA's items in order (nitems and more: no further one)
    Item job[NITEM];                         // batch
    uint32_t tmem_base;
    int abort;
    int drain_fail;
};

__device__ __forceinline__ void tma_load_4d(const CUtensorMap* map, uint64_t* bar, void* dst, int x, int y, int z,
                                            int w)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], "
        "[%2];" ::"r"(tc::smem_u32(dst)),
        "l"(map), "r"(tc::smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(w)
        : "memory");
}

// bar.red.or over `n` threads on named barrier `id`: true if any thread passed p
__device__ __forceinline__ bool bar_or(int id, int n, bool p)
{
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred pi, po;\n\t"
        "setp.ne.u32 pi, %1, 0;\n\t"
        "bar.red.or.pred po, %2, %3, pi;\n\t"
        "selp.u32 %0, 1, 0, po;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)p), "r"(id), "r"(n)
        : "memory");
    return r != 0;
}

__device__ __forceinline__ uint32_t h2(__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); }

}  // namespace xsp

// The jobs of a batch's launch: items {job's arguments, subband, first channel, job}.  The stages of all jobs are laid
// out for nsig signals.
struct XBatch {
    const XArgs* jobs;
    const CUtensorMap* maps;     // of every job's spectra
    const int4* items;
    int nitems, nsig;
    int* ctr;
    int* const* err;             // every job's error word
    int njobs;
};

// err: 1 a stage-full wait expired (cast or MMA); 2 a stage-free wait expired (producer or cast); 3 accumulator
//      wait expired; 4 epilogue wait expired; 5 drain expired
// One job (map, a, err) or, BATCH, those of b.
template <int NS, int NPOL, xsp::Input IN, bool BATCH>
__device__ __forceinline__ void xsplit_cta(const CUtensorMap* tmap, const XArgs& a, int* err, const XBatch& b)
{
    using namespace tc;
    using namespace xsp;
    constexpr int CB = 256 / NS;                      // channels of an item
    constexpr int CPT = CB / NV;                      // channels per tile
    constexpr int SWP = 8 / CB;                       // row permutation: signal s of channel c in row s ^ SWP c
    constexpr uint32_t kIdesc = tc::idesc_f16(128, 64);
    // FP16's range.  2-bit spectra reach 3.34 x 8192 = 2.7e4; their weakest bins lie in FP32's own rounding of the FFT
    // long before 2^-25, half of FP16's smallest step.  8-bit complex spectra reach 181.1 nchan and are taken at
    // 256 / nchan, while a single unit sample in an FFT gives |X| = 1: up to 1024 channels its low part is still
    // rounded no coarser than 2^-23 of it.  Beyond (WIDE) the low parts stand 2^LS higher, out of the subnormals, and
    // go into D before the high parts, whose first product scales them back.  One unit sample per FFT, 64 FFTs, error
    // of the worst baseline at 256 / 1024 / 4096 channels: 1.1e-6 each at a fixed 2^-5, now 2.4 / 3.0 / 2.8e-7
    // (k_xplain 2.6 / 2.8 / 3.1e-7).  WIDE frees the tiles later: 24 antennas x 2 pol, 4096 channels, 800 FFTs
    // 0.406 -> 0.456 ms.
    constexpr bool CPX = IN != kReal, WIDE = IN == kComplexWide;
    constexpr int LS = WIDE ? 10 : 0;
    static_assert(!(BATCH && CPX), "a batch's jobs have 2-bit samples");
    const float scale = CPX ? 256.f / (float)a.nchan : 1.f;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    Smem& sm = *reinterpret_cast<Smem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    volatile int* abort_flag = &sm.abort;

    const int ncg = BATCH ? 1 : a.nchan / CB;     // channel groups per subband
    const int nitems = BATCH ? b.nitems : a.nsb * ncg;
    int* ctr = BATCH ? b.ctr : a.ctr;
    const uint32_t stage_stride = (uint32_t)(BATCH ? b.nsig : a.nsig) * BT * CB * 8;
    const int nst = min(MAXST, (int)(RING_BYTES / stage_stride));
    // signals, channels and stages per item (a multiple of NQ)
    Item one{nullptr, a.nsig, a.nchan, (a.ntk ? a.ntk : a.T) / BT};
    auto from_args = [&](const XArgs& x, int sb, int c0) {
        return Item{reinterpret_cast<float2*>(x.acc) + (size_t)sb * (x.nsig * (x.nsig + 1) / 2) * x.nchan + c0, x.nsig, x.nchan,
                    (x.ntk ? x.ntk : x.T) / BT};
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < nst; s++) {
            mbar_init(&sm.full[s], 1);
            mbar_init(&sm.empty[s], NCW);
        }
        for (int h = 0; h < NQ; h++) {
            mbar_init(&sm.full16[h], NCW);
            mbar_init(&sm.empty16[h], 1);     // tcgen05.commit of the part's MMAs
        }
        for (int c = 0; c < 2; c++) {
            mbar_init(&sm.d_full[c], 1);
            mbar_init(&sm.d_empty[c], NEW);
        }
        for (int n = 0; n < NITEM; n++) mbar_init(&sm.item_full[n], 1);
        mbar_init(&sm.drain, 1);
        sm.abort = 0;
        sm.drain_fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc(&sm.tmem_base, TMEM_COLS);
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sm.tmem_base;

    // n-th item of the CTA (every lane of the warp; nitems: none, or a wait gave up)
    auto item_of = [&](int n) -> int {
        return mbar_wait_warp(&sm.item_full[n % NITEM], (n / NITEM) & 1, abort_flag)
                   ? *reinterpret_cast<volatile int*>(&sm.item[n % NITEM])
                   : nitems;
    };
    auto job_of = [&](int n) { return BATCH ? sm.job[n % NITEM] : one; };   // after item_of(n) gave an item
    auto record = [&](int code) {
        if constexpr (BATCH) {
            for (int j = 0; j < b.njobs; j++) atomicCAS(b.err[j], 0, code);
        } else {
            atomicCAS(err, 0, code);
        }
    };
    auto fail = [&](int code) {
        if (!*abort_flag) record(code);
        *abort_flag = 1;
    };

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R_ISSUE));
        if (warp == 0) {
            // ------------------------------------------------------------ producer
            if (lane == 0) {
                int stage = 0;
                uint32_t phase = 0;
                long long issued = 0;
                // the first item by the block's number, the others from the counter: some SMs get a quarter less
                // of the memory's rate than others
                int item = blockIdx.x;
                [[maybe_unused]] const CUtensorMap* mapped = nullptr;
                for (int n = 0;; n++) {
                    if (*abort_flag) item = nitems;
                    Item job = one;
                    int sb, c0;
                    const CUtensorMap* map = tmap;
                    if constexpr (BATCH) {
                        if (item < nitems) {
                            const int4 it = b.items[item];
                            sb = it.y;
                            c0 = it.z;
                            job = from_args(b.jobs[it.x], sb, c0);
                            map = b.maps + it.w;
                            sm.job[n % NITEM] = job;
                            if (map != mapped)   // the copy of the map in global memory, before its first use
                                asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(map) : "memory");
                            mapped = map;
                        }
                    } else {
                        sb = item / ncg;
                        c0 = (item - sb * ncg) * CB;
                    }
                    sm.item[n % NITEM] = item;
                    mbar_arrive(&sm.item_full[n % NITEM]);
                    if (item >= nitems) break;
                    const int next = nitems > (int)gridDim.x ? (int)gridDim.x + atomicAdd(ctr, 1) : nitems;
                    const uint32_t stage_bytes = (uint32_t)job.nsig * BT * CB * 8;
                    for (int kb = 0; kb < job.nk; kb++) {
                        if (!mbar_wait(&sm.empty[stage], phase ^ 1, abort_flag)) {
                            fail(2);
                            break;
                        }
                        mbar_expect_tx(&sm.full[stage], stage_bytes);
                        tma_load_4d(map, &sm.full[stage], sm.ring + (size_t)stage * stage_stride, 2 * c0,
                                    kb * (NPOL == 2 ? BT : BT / 2), 0, sb);
                        issued++;
                        if (++stage == nst) {
                            stage = 0;
                            phase ^= 1;
                        }
                    }
                    item = next;
                }
                if (nitems > (int)gridDim.x) {   // the last CTA to have drawn leaves the counter zero
                    __threadfence();
                    if (atomicAdd(ctr + 1, 1) == (int)gridDim.x - 1) {
                        ctr[0] = 0;
                        ctr[1] = 0;
                    }
                }
                // drain: the last nst fills are the only ones that may still be in flight
                for (int s = 0; s < nst && issued > 0; s++) {
                    const long long idx = issued - 1 - s;
                    if (idx < 0) break;
                    if (!mbar_drain(&sm.full[(int)(idx % nst)], (uint32_t)((idx / nst) & 1))) {
                        record(5);
                        sm.drain_fail = 1;
                        break;
                    }
                }
            }
        } else if (warp == 1) {
            // ------------------------------------------------------------ MMA issuer
            const uint32_t dsm = (uint32_t)umma_desc(smem_u32(&sm));
            uint32_t ph = 0;      // phase of the parts of the tiles (one turn for all of them)
            int db = 0;           // the D of these 32 FFTs, and its phase
            uint32_t dph = 0;
            bool ok = true;
            for (int n = 0; ok; n++) {
                if (item_of(n) >= nitems) break;
                const int nk = job_of(n).nk;
                for (int kb = 0; kb < nk && ok; kb += NQ) {
                    if (!mbar_wait_warp(&sm.d_empty[db], dph ^ 1, abort_flag)) {
                        if (lane == 0) fail(3);
                        ok = false;
                    }
#pragma unroll
                    for (int h = 0; h < NQ; h++) {
                        if (ok && !mbar_wait_warp(&sm.full16[h], ph, abort_flag)) {
                            if (lane == 0) fail(1);
                            ok = false;
                        }
                        tc_fence_after();
                        if (ok && elect_one()) {
                            const uint32_t d0 = tmem + db * 256;
                            uint32_t ds = dsm;
                            asm volatile("" : "+r"(ds));   // the descriptors are added up here, not kept
                            auto hi = [&](int c, int h, int k) {   // K16 step k of part h: 32 bytes of the rows
                                return udesc(ds + (uint32_t)((offsetof(Smem, hi) + c * HT) >> 4) + 2 * (KS * h + k));
                            };
                            auto lo = [&](int c, int h, int k) {
                                return udesc(ds + (uint32_t)((offsetof(Smem, lo) + c * LT) >> 4) + 2 * (KS * h + k));
                            };
                            // a part's low products, then its high ones (WIDE: the low ones of all parts first)
#pragma unroll
                            for (int c = 0; c < NV; c++) {
#pragma unroll
                                for (int k = 0; k < KS; k++) {
                                    if (h == 0 && k == 0) umma_ss_acc<false>(d0 + c * 64, hi(c, h, k), lo(c, h, k), kIdesc);
                                    else umma_ss_acc<true>(d0 + c * 64, hi(c, h, k), lo(c, h, k), kIdesc);
                                }
                                if constexpr (!WIDE)
#pragma unroll
                                    for (int k = 0; k < KS; k++)
                                        umma_ss_acc<true>(d0 + c * 64, hi(c, h, k), hi(c, h, k), kIdesc);
                            }
                            if constexpr (!WIDE) {
                                umma_commit(&sm.empty16[h]);
                            } else if (h == NQ - 1) {
#pragma unroll
                                for (int g = 0; g < NQ; g++) {
#pragma unroll
                                    for (int c = 0; c < NV; c++)
#pragma unroll
                                        for (int k = 0; k < KS; k++) {
                                            if (g == 0 && k == 0) umma_ss_scaled<LS>(d0 + c * 64, hi(c, g, k), hi(c, g, k), kIdesc);
                                            else umma_ss_acc<true>(d0 + c * 64, hi(c, g, k), hi(c, g, k), kIdesc);
                                        }
                                    umma_commit(&sm.empty16[g]);
                                }
                            }
                            if (h == NQ - 1) umma_commit(&sm.d_full[db]);
                        }
                        __syncwarp();
                    }
                    dph ^= db;
                    db ^= 1;
                    ph ^= 1;
                }
            }
            // drain: every issued MMA retires before TMEM is freed (committed by the issuing lane)
            if (elect_one()) {
                umma_commit(&sm.drain);
                if (!mbar_drain(&sm.drain, 0)) {
                    record(5);
                    sm.drain_fail = 1;
                }
            }
            __syncwarp();
        }
    } else if (warp < 4 + NCW) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R_CAST));
        // ------------------------------------------------------------ cast
        const int c = lane & (CB - 1);
        constexpr int NG = 2 * KS;                        // 16-byte chunks of a row and stage, one per thread
        const int tg = (lane / CB) & (NG - 1);
        constexpr int UPW = 32 / (NG * CB);               // units (a signal, or an antenna's two) of a warp at a time
        const int u0 = (warp - 4) * UPW + lane / (NG * CB);
        // two channels of a tile at NS = 32: rows H c0, H c1, H' c0, H' c1, so that its first 64 rows are B
        uint8_t* hi = sm.hi + (c / CPT) * HT + (c % CPT) * 32 * 128;
        uint8_t* lo = sm.lo + (c / CPT) * LT + (c % CPT) * 32 * 128;
        // one signal's four values into row s ^ SWP c, chunk NG h + tg
        auto put = [&](const float2 (&x)[4], int s, int h) {
            uint32_t hw[4], gw[4], lw[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float2 v = CPX ? make_float2(x[i].x * scale, x[i].y * scale) : x[i];
                const __half2 hh = __floats2half2_rn(v.x, v.y);
                const float2 f = __half22float2(hh);
                const float2 l = __fadd2_rn(v, make_float2(-f.x, -f.y));
                const __half2 ll = __floats2half2_rn(l.x * (float)(1 << LS), l.y * (float)(1 << LS));
                hw[i] = h2(hh);
                gw[i] = __byte_perm(hw[i], 0u, 0x1032) ^ 0x80000000u;   // (Im, -Re)
                lw[i] = h2(__hadd2(ll, ll));
            }
            const int r = s ^ (SWP * c);
            const int off = r * 128 + (((NG * h + tg) ^ (r & 7)) << 4);
            *reinterpret_cast<uint4*>(hi + off) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
            *reinterpret_cast<uint4*>(hi + 64 * 128 + off) = make_uint4(gw[0], gw[1], gw[2], gw[3]);
            *reinterpret_cast<uint4*>(lo + off) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
        };
        int st = 0;
        uint32_t ph = 0;
        uint32_t ph16 = 0;   // phase of the parts
        bool stop = false;
        for (int n = 0; !stop; n++) {
            if (item_of(n) >= nitems) break;
            const Item job = job_of(n);
            const int nunit = job.nsig / NPOL, nk = job.nk;
            for (int kb = 0; kb < nk; kb++) {
                const int h = kb & (NQ - 1);
                if (!mbar_wait_warp(&sm.full[st], ph, abort_flag)) {
                    if (lane == 0) fail(1);
                    stop = true;
                    break;
                }
                if (!mbar_wait_warp(&sm.empty16[h], ph16 ^ 1, abort_flag)) {
                    if (lane == 0) fail(2);
                    stop = true;
                    break;
                }
                const float4* src = reinterpret_cast<const float4*>(sm.ring + (size_t)st * stage_stride) + tg * CB + c;
#pragma unroll 2
                for (int u = u0; u < nunit; u += NCW * UPW) {
                    if constexpr (NPOL == 2) {   // [ant][BT][chan] of both polarisations: FFTs tg + NG i
                        float4 y[4];
#pragma unroll
                        for (int i = 0; i < 4; i++) y[i] = src[(u * BT + NG * i) * CB];
                        const float2 p0[4] = {{y[0].x, y[0].y}, {y[1].x, y[1].y}, {y[2].x, y[2].y}, {y[3].x, y[3].y}};
                        const float2 p1[4] = {{y[0].z, y[0].w}, {y[1].z, y[1].w}, {y[2].z, y[2].w}, {y[3].z, y[3].w}};
                        put(p0, 2 * u, h);
                        put(p1, 2 * u + 1, h);
                    } else {                     // [sig][BT / 2][chan] of both FFTs of a pair: pairs tg, tg + NG
                        const float4 y0 = src[u * (BT / 2) * CB], y1 = src[(u * (BT / 2) + NG) * CB];
                        const float2 x[4] = {{y0.x, y0.y}, {y0.z, y0.w}, {y1.x, y1.y}, {y1.z, y1.w}};
                        put(x, u, h);
                    }
                }
                fence_async_smem();   // the tiles are read by the tensor cores (async proxy)
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&sm.empty[st]);
                    mbar_arrive(&sm.full16[h]);
                }
                if (++st == nst) {
                    st = 0;
                    ph ^= 1;
                }
                if (h == NQ - 1) ph16 ^= 1;
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R_EPI));
        // ------------------------------------------------------------ epilogue
        const int q = warp & 3;                  // TMEM lane quadrant of this warp
        const int e = (warp - 4 - NCW) >> 2;     // tiles e and e + 2
        // columns of this warp's rows: all 64 signals, or the 32 of its own channel of the tile
        constexpr int NCOL = NS;
        const uint32_t lane0 = ((uint32_t)(q * 32) << 16) + (NS == 32 ? 32 * (q & 1) : 0);
        const float inv = 0.5f * (1.f + 0x1p-22f) / (scale * scale);   // what truncation took put back
        int db = 0;
        uint32_t dph = 0;
        bool stop = false;
        for (int nit = 0; !stop; nit++) {
            const int item = item_of(nit);
            // all of these warps leave together (a wait may have given up in one of them)
            if (bar_or(1, 32 * NEW, item >= nitems)) break;
            const Item job = BATCH ? job_of(nit) : from_args(a, item / ncg, item % ncg * CB);
            const int nsig = job.nsig;
            const int nseg = (job.nk * BT + SEG - 1) / SEG;
            const int nd = job.nk / NQ;
            const int dseg = (nd + nseg - 1) / nseg;      // D per segment of an item
            for (int d = 0; d < nd && !stop;) {
                float2 sum[2][NCOL / 2];
#pragma unroll
                for (int t = 0; t < 2; t++)
#pragma unroll
                    for (int k = 0; k < NCOL / 2; k++) sum[t][k] = make_float2(0.f, 0.f);
                for (const int dend = min(d + dseg, nd); d < dend; d++) {
                    if (!mbar_wait_warp(&sm.d_full[db], dph, abort_flag)) {
                        if (lane == 0) fail(4);
                        stop = true;
                        break;
                    }
                    tc_fence_after();
#pragma unroll
                    for (int t = 0; t < 2; t++)
#pragma unroll
                        for (int n = 0; n < NCOL; n += EC) {
                            uint32_t v[EC];
                            tmem_ld16(tmem + lane0 + db * 256 + (e + 2 * t) * 64 + n, v);
                            tmem_wait_ld();
#pragma unroll
                            for (int k = 0; k < EC; k += 2)
                                sum[t][(n + k) / 2] = __fadd2_rn(
                                    sum[t][(n + k) / 2], make_float2(__uint_as_float(v[k]), __uint_as_float(v[k + 1])));
                        }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sm.d_empty[db]);
                    dph ^= db;
                    db ^= 1;
                }
                // ---- sums to the accumulators, a tile at a time (two tiles at NS = 32, one beside the other)
                // through shared memory: V[i][j] needs D[i][j] and D[j][i], real and imaginary rows
#pragma unroll
                for (int t = 0; t < 2; t++) {
#pragma unroll
                    for (int ee = 0; ee < (NS == 32 ? 1 : 2); ee++) {
                        if (NS == 32 || e == ee) {
                            float* out = sm.v + (q * 32 + lane) * VROW + (NS == 32 ? 32 * e : 0);
#pragma unroll
                            for (int n = 0; n < NCOL; n += 2) {
                                out[n] = sum[t][n / 2].x;
                                out[n + 1] = sum[t][n / 2].y;
                            }
                        }
                        stop = bar_or(1, 32 * NEW, stop);
                        if (!stop) {
                            const int w = 4 * e + q;   // 0 .. 7
                            float2* acc = job.acc;
                            if constexpr (NS == 32) {
                                // channels 4 t + g, g = 0 .. 3: tile 2 t + (g >> 1)'s half g & 1; a thread takes channels
                                // 4 t + 2 x and the next
                                const int x = w & 1;
                                for (int i = w >> 1; i < nsig; i += 4) {
                                    const int j = lane;
                                    if (j >= i && j < nsig) {
                                        float r[4];
#pragma unroll
                                        for (int y = 0; y < 2; y++) {
                                            const int k = SWP * (4 * t + 2 * x + y);
                                            const float* re = sm.v + 32 * y * VROW + 32 * x;
                                            const float* ig = re + 64 * VROW;
                                            r[2 * y] = inv * (re[(i ^ k) * VROW + (j ^ k)] + re[(j ^ k) * VROW + (i ^ k)]);
                                            r[2 * y + 1] = inv * (ig[(i ^ k) * VROW + (j ^ k)] - ig[(j ^ k) * VROW + (i ^ k)]);
                                        }
                                        const int p = i * nsig - i * (i - 1) / 2 + (j - i);
                                        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(
                                                         acc + (size_t)p * job.nchan + 4 * t + 2 * x),
                                                     "f"(r[0]), "f"(r[1]), "f"(r[2]), "f"(r[3])
                                                     : "memory");
                                    }
                                }
                            } else {
                                const int ch = ee + 2 * t, k = SWP * ch;
                                for (int i = w; i < nsig; i += 8)
                                    for (int j = (i & ~31) + lane; j < nsig; j += 32)
                                        if (j >= i) {
                                            const float* re = sm.v;
                                            const float* ig = sm.v + 64 * VROW;
                                            const float vr = inv * (re[(i ^ k) * VROW + (j ^ k)] + re[(j ^ k) * VROW + (i ^ k)]);
                                            const float vm = inv * (ig[(i ^ k) * VROW + (j ^ k)] - ig[(j ^ k) * VROW + (i ^ k)]);
                                            const int p = i * nsig - i * (i - 1) / 2 + (j - i);
                                            asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(
                                                             acc + (size_t)p * job.nchan + ch),
                                                         "f"(vr), "f"(vm)
                                                         : "memory");
                                        }
                            }
                        }
                        stop = bar_or(1, 32 * NEW, stop);
                    }
                }
            }
        }
    }

    __syncthreads();
    // after an expired drain, MMAs may still write TMEM: it stays allocated (code 5 was recorded;
    // the context's later tensor-core launches cannot be trusted and the process should reset)
    if (warp == 0 && !sm.drain_fail) {
        tc_fence_after();
        tmem_dealloc(tmem, TMEM_COLS);
    }
}

template <int NS, int NPOL, xsp::Input IN>
__global__ void __launch_bounds__(xsp::NTHREADS, 1)
k_xsplit(const __grid_constant__ CUtensorMap tmap, XArgs a, int* err)
{
    xsplit_cta<NS, NPOL, IN, false>(&tmap, a, err, XBatch{});
}

template <int NS, int NPOL>
__global__ void __launch_bounds__(xsp::NTHREADS, 1)
k_xsplit_batch(XBatch b)
{
    xsplit_cta<NS, NPOL, xsp::kReal, true>(nullptr, XArgs{}, nullptr, b);
}

// Spectra [sb][ant][T][chan][2 polarisations] or [sb][sig][T / 2][chan][2 FFTs] of 8-byte complex values
static cudaError_t xsplit_map(const XArgs& a, int npol, CUtensorMap* map)
{
    using namespace xsp;
    auto enc = tc::tensor_map_encoder();
    if (!enc) return cudaErrorNotSupported;
    const cuuint32_t cb = a.nsig <= 32 ? 8 : 4;
    const cuuint64_t nt = npol == 2 ? a.T : a.T / 2, nr = a.nsig / npol, row = (cuuint64_t)a.nchan * 16;
    const cuuint64_t dims[4] = {(cuuint64_t)2 * a.nchan, nt, nr, (cuuint64_t)a.nsb};
    const cuuint64_t strides[3] = {row, nt * row, nr * nt * row};
    const cuuint32_t box[4] = {2 * cb, (cuuint32_t)(npol == 2 ? BT : BT / 2), (cuuint32_t)nr, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_INT64, 4, const_cast<void*>(a.spec), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

template <int NS, int NPOL, xsp::Input IN>
static cudaError_t launch_xsplit_t(const XArgs& a, int* d_err, int nsm, cudaStream_t st)
{
    using namespace xsp;
    constexpr int CB = 256 / NS;
    CUtensorMap map;
    cudaError_t e = xsplit_map(a, NPOL, &map);
    if (e != cudaSuccess) return e;
    const size_t sm = sizeof(Smem) + 1024;
    static unsigned configured = 0;
    e = set_smem_once(k_xsplit<NS, NPOL, IN>, sm, &configured);
    if (e != cudaSuccess) return e;
    const long long nitems = (long long)a.nsb * (a.nchan / CB);
    const int grid = nitems < nsm ? (int)nitems : nsm;
    k_xsplit<NS, NPOL, IN><<<grid, NTHREADS, sm, st>>>(map, a, d_err);
    return cudaGetLastError();
}

template <int NS, int NPOL>
static cudaError_t launch_xsplit_n(const XArgs& a, int cpx, int* d_err, int nsm, cudaStream_t st)
{
    using namespace xsp;
    return !cpx            ? launch_xsplit_t<NS, NPOL, kReal>(a, d_err, nsm, st)
           : a.nchan <= 1024 ? launch_xsplit_t<NS, NPOL, kComplex>(a, d_err, nsm, st)
                             : launch_xsplit_t<NS, NPOL, kComplexWide>(a, d_err, nsm, st);
}

// A geometry-only rule (a batch's jobs take the same path as alone).  The kernel's time is that of an item,
// 10 us + 0.042 (2 signals) to 0.07 us (64) per FFT, times the items over the SMs; k_xplain's grows with the
// multiply-adds but takes 23 us or more.  Measured k_xplain / here, us (items):
//   17 to 64 signals, items for most SMs: here, also with a last round of items that is nearly empty
//       4096 FFTs, 17 signals (128) 389 / 213, (160) 490 / 414; 32 (128) 443 / 261, (160) 556 / 509, (320) 1083 / 763;
//       33 (160) 506 / 439; 64 (160) 959 / 553, (512) 5683 / 2143; below, not: 32 (64) 226 / 256; 33 (64) 207 / 224
//   9 to 16 signals: the faster one where every round of items is 6/7 full (an item is not cut)
//       4096 FFTs, 9 signals (128) 210 / 198, (288) 445 / 387; 16 (128) 234 / 203; 512 FFTs, 12 (288) 72 / 61
//     where it is not, the slower one by up to 1.45 (a batch's jobs share rounds), and still chosen: its sums are the
//     more accurate (9 signals, 160 items, 4096 FFTs 1.1e-7, k_xplain 2.2e-7)
//       4096 FFTs, 9 signals (160) 264 / 385, (224) 364 / 390, (320) 498 / 566, (448) 693 / 751; 16 (192) 338 / 394,
//       (320) 558 / 579; 512 FFTs, 12 (160) 50 / 58, (192) 57 / 59
//     with half of the SMs idle, not: 9 (64) 117 / 195; 1024 FFTs, 9 (64) 41 / 59
//   up to 8 signals k_xplain has little to do: 4096 FFTs (512) 290 / 699
//   fewer FFTs than one D holds: what the truncations take is less than what is put back (1 FFT: error of the sums
//       2.0e-7, 0.3e-7 on the FP32 units; 16: 1.4, 0.9; 24: 1.0, 1.1; 32: 0.9, 1.2)
//   short calls of one item per SM: 64 FFTs, 2 signals (16) 23 / 13; 8 (128) 33 / 14; 64 (64) 45 / 23;
//       not with more items: 2 (512) 24 / 25
bool xsplit_pays(int nsig, int nchan, int nsb, int numffts, int nsm)
{
    if (nsig < 1 || nsig > 64 || nchan < 8 || nchan % 8 != 0) return false;
    if (numffts < kXsplitMinFfts) return false;
    const long long nitems = (long long)nsb * (nchan / (nsig <= 32 ? 8 : 4));
    if (numffts <= 128 && nitems <= nsm) return true;
    return nsig > 8 && nitems * 7 >= (long long)nsm * 6;
}

static bool xsplit_fits(const XArgs& a, int npol)
{
    using namespace xsp;
    const int nslot = a.ntk ? a.ntk : a.T;
    return a.nsig >= 1 && a.nsig <= 64 && a.nsig % npol == 0 && a.nchan % 8 == 0 && a.nchan >= 8 && a.T % BT == 0 && nslot >= 1 &&
           nslot % (NQ * BT) == 0 && nslot <= a.T && a.nsb >= 1 && a.spec && a.acc;
}

cudaError_t launch_xsplit(const XArgs& a, int npol, int cpx, int* d_err, int nsm, cudaStream_t st)
{
    using namespace xsp;
    if (!xsplit_fits(a, npol)) return cudaErrorInvalidValue;
    static_assert(sizeof(Smem) + 1024 <= 227 * 1024, "one CTA's shared memory");
    if (npol == 2)
        return a.nsig <= 32 ? launch_xsplit_n<32, 2>(a, cpx, d_err, nsm, st) : launch_xsplit_n<64, 2>(a, cpx, d_err, nsm, st);
    return a.nsig <= 32 ? launch_xsplit_n<32, 1>(a, cpx, d_err, nsm, st) : launch_xsplit_n<64, 1>(a, cpx, d_err, nsm, st);
}

// ---- a batch's jobs in one launch: the items of many short jobs fill the SMs together and share one start.  Whole
// batch, a launch per job / one launch per group (one k_xplain launch): 32 jobs of 4 antennas x 128 channels x 100
// FFTs 479 / 176 us (206); 64 of 16 antennas x 512 channels x 128 FFTs 1424 / 786 (1132); 12 of 9 antennas x 256
// channels x 5 subbands x 2000 FFTs, whose items fill a last round of SMs badly alone, 3828 / 2752 (3296).
int xsplit_items(const XArgs& a) { return a.nsb * (a.nchan / (a.nsig <= 32 ? 8 : 4)); }

int4 xsplit_item(const XArgs& a, int args, int job, int n)
{
    const int cb = a.nsig <= 32 ? 8 : 4, ncg = a.nchan / cb;
    return make_int4(args, n / ncg, n % ncg * cb, job);
}

cudaError_t xsplit_map_bytes(const XArgs& a, int npol, void* map128)
{
    static_assert(sizeof(CUtensorMap) == 128, "stride of the maps in memory");
    if (!xsplit_fits(a, npol)) return cudaErrorInvalidValue;
    CUtensorMap map;
    const cudaError_t e = xsplit_map(a, npol, &map);
    if (e == cudaSuccess) std::memcpy(map128, &map, sizeof map);
    return e;
}

template <int NS, int NPOL>
static cudaError_t launch_xsplit_batch_t(const XBatch& b, int nsm, cudaStream_t st)
{
    using namespace xsp;
    const size_t sm = sizeof(Smem) + 1024;
    static unsigned configured = 0;
    const cudaError_t e = set_smem_once(k_xsplit_batch<NS, NPOL>, sm, &configured);
    if (e != cudaSuccess) return e;
    k_xsplit_batch<NS, NPOL><<<b.nitems < nsm ? b.nitems : nsm, NTHREADS, sm, st>>>(b);
    return cudaGetLastError();
}

cudaError_t launch_xsplit_batch(int nsig_max, int npol, const XArgs* d_jobs, const void* d_maps, const int4* d_items,
                                int nitems, int* ctr, int* const* d_errs, int njobs, int nsm, cudaStream_t st)
{
    if (nsig_max < 1 || nsig_max > 64 || nitems < 1 || (npol != 1 && npol != 2)) return cudaErrorInvalidValue;
    const XBatch b{d_jobs, static_cast<const CUtensorMap*>(d_maps), d_items, nitems, nsig_max, ctr, d_errs, njobs};
    if (npol == 2)
        return nsig_max <= 32 ? launch_xsplit_batch_t<32, 2>(b, nsm, st) : launch_xsplit_batch_t<64, 2>(b, nsm, st);
    return nsig_max <= 32 ? launch_xsplit_batch_t<32, 1>(b, nsm, st) : launch_xsplit_batch_t<64, 1>(b, nsm, st);
}

}  // namespace fx
