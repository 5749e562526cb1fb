// fx_xtch.cu -- tensor-core X stage on channel-contiguous FP16 spectra (tcgen05, FP32 accumulation), up to
// 64 signals.
//
// The same Gram as fx_xtc.cu (per channel G = A A^T over the real-ified, time-major rows
// A[2s] = Re X_s, A[2s+1] = Im X_s; kernel.c:846 with the conjugation of kernel.c:557-568), but
// the operand is read from the FFT F stage's own layout [sb][sig][T][chan] of (Re, Im) half pairs.
// The K-major layout the tensor cores need is a corner turn (time-contiguous rows); here it is done
// on the way into the MMA operand, so it costs no pass over HBM.  Values and MMA order are those
// of fx_xtc.cu on turned spectra, so the visibilities are bit-identical to it.
//
// Bound by HBM and the stage pipeline's latency: 2 bytes per sample against 65 flop/B.  32 signals x 4
// subbands x 2048 channels x 31250 FFTs take 7.5 ms (4.4 TB/s); reading FP32 spectra and rounding
// them here took 12.9 ms for twice the bytes.
//
// Persistent, warp-specialised CTA per SM; work item = (subband, CB channels): 8 channels (one whole
// 32-byte sector of each spectrum row, N = 64 accumulator columns each) up to 32 signals, 4 channels
// (N = 128) up to 64, which fills the 512 TMEM columns and 64 KB of operand tiles either way, or 4 channels
// (N = 64) for up to 32 signals of few channels; with 4 the other half of a sector is the next item's,
// which another SM reads at the same time (L2):
//   warp 0     TMA producer: box {CB channels, 32 FFTs, nsig signals} (unswizzled: (Re, Im) of the CB
//              channels of FFT t of signal s at 4 CB (32 s + t)) into a ring of stages (as many as
//              128 KB holds, up to 8)
//   warp 1     MMA issuer: per stage and channel 2 x tcgen05.mma.kind::f16 M128 K16 on the channel's
//              tile (A and B descriptors the same tile; with 64-row tiles rows 64 .. 127 of A are the
//              next tile's, whose accumulator lanes nothing reads)
//   warps 2-9  turn: stage j -> K half j % 2 (FFTs 32 (j % 2) .. + 31) of the CB channels' tiles, 2 nsig
//              rows x 64 FFTs, K-major SWIZZLE_128B, rows >= 2 nsig zero; the two halves of a tile are
//              disjoint, so the turn fills one while the MMAs read the other
//   warps 10-13 epilogue: tcgen05.ld of the CB channels' accumulators, Re/Im combination, FP32
//              accumulate into acc[sb][c][pair(i,j)], i <= j; an item is T / 32 stages long, so its
//              epilogue (one accumulator set, not double-buffered) is a small part of it.
// Every wait is bounded by time; on expiry the CTA records an error code, drains what it
// issued (again bounded), frees TMEM and returns.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <cuda_fp16.h>

#include "fx_common.cuh"
#include "fx_kernels.h"
#include "fx_tc.cuh"

namespace fx {

namespace tcxh {

constexpr int BT = 32;                       // FFTs per stage (a K half of the tiles)
constexpr int MAXSIG = 64;
constexpr int RING_BYTES = 128 * 1024;       // stages of 4 CB BT nsig bytes
constexpr int MAXST = 8;
constexpr int TILES_BYTES = 64 * 1024;       // CB tiles of N rows x 64 FP16
constexpr int NTW = 8;                       // turn warps
constexpr int NTHREADS = 32 * (2 + NTW + 4);   // producer, MMA, turn, 4 epilogue warps
constexpr int TMEM_COLS = 512;               // CB channels x N FP32 columns

struct Smem {
    alignas(1024) uint8_t f16[TILES_BYTES];
    alignas(1024) uint8_t ring[RING_BYTES];  // (also what the last tile's rows 64 .. 127 read)
    alignas(8) uint64_t full[MAXST];
    uint64_t empty[MAXST];
    uint64_t full16[2];                      // per K half
    uint64_t empty16[2];
    uint64_t acc_full;
    uint64_t acc_empty;
    uint64_t drain;
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

}  // namespace tcxh

// err: 0 ok; 1 a stage-full wait expired (turn or MMA); 2 a stage-free wait expired (producer or
//      turn); 3 accumulator wait expired; 4 epilogue wait expired; 5 drain expired
template <int CB, int N>
__global__ void __launch_bounds__(tcxh::NTHREADS, 1)
k_xtch(const __grid_constant__ CUtensorMap tmap, XArgs a, int* err)
{
    using namespace tc;
    using namespace tcxh;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    Smem& sm = *reinterpret_cast<Smem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    volatile int* abort_flag = &sm.abort;

    // N: accumulator columns (and tile rows) of a channel
    static_assert(CB * N <= TMEM_COLS && CB * N * 128 <= TILES_BYTES, "tiles and accumulators");
    constexpr int TILE_BYTES = N * 128;
    constexpr uint32_t kIdesc = tc::idesc_f16(128, N);
    const int nsig = a.nsig;
    const int npair = nsig * (nsig + 1) / 2;
    const int ncq = a.nchan / CB;                 // channel groups per subband
    const int nitems = a.nsb * ncq;
    const int nk = (a.ntk ? a.ntk : a.T) / BT;    // stages per item (even)
    const uint32_t stage_bytes = (uint32_t)nsig * BT * CB * 4;
    const int nst = min(MAXST, (int)(RING_BYTES / stage_bytes));   // stages in flight

    if (threadIdx.x == 0) {
        for (int s = 0; s < nst; s++) {
            mbar_init(&sm.full[s], 1);
            mbar_init(&sm.empty[s], NTW);   // one arrival per turn warp
        }
        for (int h = 0; h < 2; h++) {
            mbar_init(&sm.full16[h], NTW);
            mbar_init(&sm.empty16[h], 1);     // tcgen05.commit of the half's MMAs
        }
        mbar_init(&sm.acc_full, 1);
        mbar_init(&sm.acc_empty, 128);
        mbar_init(&sm.drain, 1);
        sm.abort = 0;
        sm.drain_fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // rows 2 nsig .. N - 1 of every tile stay zero: the turn writes rows below 2 nsig only
    {
        const int nz = (N - 2 * nsig) * 8;   // 16-byte chunks per tile
        for (int i = threadIdx.x; i < CB * nz; i += NTHREADS) {
            const int tile = i / nz;
            const int rem = i - tile * nz;
            *reinterpret_cast<uint4*>(sm.f16 + (size_t)tile * TILE_BYTES + (2 * nsig + rem / 8) * 128 + (rem % 8) * 16) =
                make_uint4(0u, 0u, 0u, 0u);
        }
        fence_async_smem();
    }
    if (warp == 0) tmem_alloc(&sm.tmem_base, TMEM_COLS);
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sm.tmem_base;

    if (warp == 0) {
        // ------------------------------------------------------------ producer
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            long long issued = 0;
            for (int item = blockIdx.x; item < nitems && !*abort_flag; item += gridDim.x) {
                const int sb = item / ncq;
                const int c0 = (item - sb * ncq) * CB;
                for (int kb = 0; kb < nk; kb++) {
                    if (!mbar_wait(&sm.empty[stage], phase ^ 1, abort_flag)) {
                        if (!*abort_flag) atomicCAS(err, 0, 2);
                        *abort_flag = 1;
                        break;
                    }
                    mbar_expect_tx(&sm.full[stage], stage_bytes);
                    tma_load_4d(&tmap, &sm.full[stage], sm.ring + (size_t)stage * stage_bytes, c0, kb * BT, 0, sb);
                    issued++;
                    if (++stage == nst) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
            // drain: the last nst fills are the only ones that may still be in flight
            for (int s = 0; s < nst && issued > 0; s++) {
                const long long idx = issued - 1 - s;
                if (idx < 0) break;
                const int st = (int)(idx % nst);
                const uint32_t ph = (uint32_t)((idx / nst) & 1);
                const unsigned long long t0 = globaltimer();
                while (!mbar_try(&sm.full[st], ph)) {
                    if (globaltimer() - t0 > WAIT_NS) {
                        atomicCAS(err, 0, 5);
                        sm.drain_fail = 1;
                        break;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        const uint32_t dsm = (uint32_t)umma_desc(smem_u32(&sm));
        auto dlo = [&](const void* p) -> uint32_t {
            return dsm + (uint32_t)(((const char*)p - (const char*)&sm) >> 4);
        };
        uint32_t ph16 = 0;   // bit h: phase of K half h
        uint32_t acc_phase = 0;
        for (int item = blockIdx.x; item < nitems && !__any_sync(0xffffffffu, *abort_flag); item += gridDim.x) {
            if (!mbar_wait_warp(&sm.acc_empty, acc_phase ^ 1, abort_flag)) {
                if (lane == 0) {
                    if (!*abort_flag) atomicCAS(err, 0, 3);
                    *abort_flag = 1;
                }
                break;
            }
            tc_fence_after();
            bool ok = true;
            for (int kb = 0; kb < nk; kb++) {
                const int h = kb & 1;
                if (!mbar_wait_warp(&sm.full16[h], (ph16 >> h) & 1, abort_flag)) {
                    if (lane == 0) {
                        if (!*abort_flag) atomicCAS(err, 0, 1);
                        *abort_flag = 1;
                    }
                    ok = false;
                    break;
                }
                tc_fence_after();
                if (elect_one()) {
                    // the Gram of each channel's tile over K half h: K16 steps 2h, 2h + 1 (32 bytes of
                    // K each, +2 in the descriptors' start field)
#pragma unroll
                    for (int c = 0; c < CB; c++) {
                        const uint32_t dt = dlo((sm.f16 + c * TILE_BYTES)) + 4 * h;
                        const uint32_t d = tmem + c * N;
                        umma<false>(d, udesc(dt), udesc(dt), kIdesc, kb > 0 ? 1u : 0u);
                        umma<false>(d, udesc(dt + 2), udesc(dt + 2), kIdesc, 1u);
                    }
                    umma_commit(&sm.empty16[h]);
                }
                __syncwarp();
                ph16 ^= 1u << h;
            }
            if (!ok) break;
            if (elect_one()) umma_commit(&sm.acc_full);
            __syncwarp();
            acc_phase ^= 1;
        }
        // drain: every issued MMA retires before TMEM is freed (committed by the issuing lane)
        if (elect_one()) {
            umma_commit(&sm.drain);
            const unsigned long long t0 = globaltimer();
            while (!mbar_try(&sm.drain, 0)) {
                if (globaltimer() - t0 > WAIT_NS) {
                    atomicCAS(err, 0, 5);
                    sm.drain_fail = 1;
                    break;
                }
            }
        }
        __syncwarp();
    } else if (warp < 2 + NTW) {
        // ------------------------------------------------------------ turn (warps 2 .. 1 + NTW)
        // Lane (w, g) takes FFTs 2w, 2w + 1 of 4 channels: two 16-byte reads give the 4 channels' Re and Im
        // words of K chunk 4h + w / 4 (byte_perm), eight 4-byte stores put them into the tiles.  With 4
        // channels g picks the signal, s or s + 2; with 8 it is the channel quad, of signal s + 2 (g ^ it)
        // in step it.  The rows of s and s + 2 differ in bit 2 of the swizzle, so the two half warps
        // store to different halves of the 32 banks; the reads take the odd FFT first where that
        // puts a quarter warp on 8 different 16-byte slots.  Each warp takes 4 signals at a time.
        const int w = CB == 4 ? lane & 15 : lane >> 1;
        const int g = CB == 4 ? lane >> 4 : lane & 1;
        const int j = CB == 4 ? (w >> 2) & 1 : (w >> 1) & 1;
        const uint32_t sre = j ? 0x1054u : 0x5410u, sim = j ? 0x3276u : 0x7632u;
        int st = 0;
        uint32_t ph = 0;
        uint32_t ph16 = 0;   // bit h: phase of K half h
        bool stop = false;
        for (int item = blockIdx.x; item < nitems && !stop; item += gridDim.x) {
            for (int kb = 0; kb < nk; kb++) {
                const int h = kb & 1;
                if (!mbar_wait_warp(&sm.full[st], ph, abort_flag)) {
                    if (lane == 0) {
                        if (!*abort_flag) atomicCAS(err, 0, 1);
                        *abort_flag = 1;
                    }
                    stop = true;
                    break;
                }
                if (!mbar_wait_warp(&sm.empty16[h], ((ph16 >> h) & 1) ^ 1, abort_flag)) {
                    if (lane == 0) {
                        if (!*abort_flag) atomicCAS(err, 0, 2);
                        *abort_flag = 1;
                    }
                    stop = true;
                    break;
                }
                const uint8_t* src = sm.ring + (size_t)st * stage_bytes + (CB == 4 ? 0 : 16 * g);
                const int k = 4 * h + (w >> 2);                // chunk of the 128-byte tile row
                constexpr int STEPS = CB == 4 ? 2 : 4;         // (signals, quads) of 4 signals per lane
                for (int s0 = 4 * (warp - 2); s0 < nsig; s0 += 4 * NTW) {
                    uint4 v[STEPS][2];
#pragma unroll
                    for (int u = 0; u < STEPS; u++) {
                        const int s = s0 + (CB == 4 ? u + 2 * g : (u >> 1) + 2 * (g ^ (u & 1)));
                        const uint4* p = reinterpret_cast<const uint4*>(src + (s * BT + 2 * w) * (4 * CB));
                        if (s < nsig) {
                            v[u][0] = p[j * (CB / 4)];
                            v[u][1] = p[(1 - j) * (CB / 4)];
                        }
                    }
#pragma unroll
                    for (int u = 0; u < STEPS; u++) {
                        const int s = s0 + (CB == 4 ? u + 2 * g : (u >> 1) + 2 * (g ^ (u & 1)));
                        if (s < nsig) {
                            const uint32_t x[4] = {v[u][0].x, v[u][0].y, v[u][0].z, v[u][0].w};
                            const uint32_t y[4] = {v[u][1].x, v[u][1].y, v[u][1].z, v[u][1].w};
                            const int r0 = 2 * s, r1 = 2 * s + 1;
                            uint8_t* re = sm.f16 + (CB == 4 ? 0 : 4 * g * TILE_BYTES) + (w & 3) * 4 + r0 * 128 + ((k ^ (r0 & 7)) << 4);
                            uint8_t* im = sm.f16 + (CB == 4 ? 0 : 4 * g * TILE_BYTES) + (w & 3) * 4 + r1 * 128 + ((k ^ (r1 & 7)) << 4);
#pragma unroll
                            for (int c = 0; c < 4; c++) {
                                *reinterpret_cast<uint32_t*>(re + c * TILE_BYTES) = __byte_perm(x[c], y[c], sre);
                                *reinterpret_cast<uint32_t*>(im + c * TILE_BYTES) = __byte_perm(x[c], y[c], sim);
                            }
                        }
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
                ph16 ^= 1u << h;
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue (last 4 warps)
        const int q = warp & 3;                  // TMEM lane quadrant of this warp
        const int r = q * 32 + lane;             // accumulator row
        const bool odd = (r & 1) != 0;
        const int i = r >> 1;                    // signal of this row
        const int pbase = i * nsig - (i * (i - 1)) / 2 - i;   // pair(i, j) = pbase + j
        uint32_t acc_phase = 0;
        float2* acc = reinterpret_cast<float2*>(a.acc);
        for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
            const int sb = item / ncq;
            const int c0 = (item - sb * ncq) * CB;
            if (!mbar_wait(&sm.acc_full, acc_phase, abort_flag)) {
                if (!*abort_flag) atomicCAS(err, 0, 4);
                *abort_flag = 1;
                break;
            }
            tc_fence_after();
            for (int c = 0; c < CB; c++) {
                float* out = reinterpret_cast<float*>(acc + ((size_t)sb * a.nchan + c0 + c) * npair);
                const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + c * N;
#pragma unroll 1
                for (int cq = 0; cq < N / 32; cq++) {      // 32 columns = 16 signal pairs j per chunk
                    uint32_t v[32];
                    tmem_ld32(taddr + cq * 32, v);
                    tmem_wait_ld();
                    if (c == CB - 1 && cq == N / 32 - 1) {
                        tc_fence_before();
                        mbar_arrive(&sm.acc_empty);
                    }
#pragma unroll
                    for (int jj = 0; jj < 16; jj++) {
                        const int j = cq * 16 + jj;
                        const float g0 = __uint_as_float(v[2 * jj]);      // G[r][2j]
                        const float g1 = __uint_as_float(v[2 * jj + 1]);  // G[r][2j+1]
                        // even row 2i: (G[2i][2j], G[2i][2j+1]) = (a, b); odd row: (c, d).  Re = a + d,
                        // Im = c - b: each row takes the other's column 2j+1
                        const float other = __shfl_xor_sync(0xffffffffu, g1, 1);
                        const float val = odd ? (g0 - other) : (g0 + other);
                        if (j >= i && j < nsig) atomicAdd(out + 2 * (pbase + j) + (odd ? 1 : 0), val);
                    }
                }
            }
            acc_phase ^= 1;
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

template <int CB, int N>
static cudaError_t launch_xtch_t(const XArgs& a, int* d_err, int nsm, cudaStream_t st)
{
    using namespace tcxh;
    auto enc = tc::tensor_map_encoder();
    if (!enc) return cudaErrorNotSupported;
    // spectra [sb][sig][T][chan] (4-byte complex elements): box {CB channels, 32 FFTs, nsig, 1}, unswizzled
    // (dense 16- or 32-byte rows: with a swizzle, rows narrower than the swizzle span are each padded
    // to a whole 128-byte line)
    CUtensorMap map;
    const cuuint64_t dims[4] = {(cuuint64_t)a.nchan, (cuuint64_t)a.T, (cuuint64_t)a.nsig, (cuuint64_t)a.nsb};
    const cuuint64_t strides[3] = {(cuuint64_t)a.nchan * 4, (cuuint64_t)a.T * a.nchan * 4,
                                   (cuuint64_t)a.nsig * a.T * a.nchan * 4};
    const cuuint32_t box[4] = {(cuuint32_t)CB, (cuuint32_t)BT, (cuuint32_t)a.nsig, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = enc(&map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, const_cast<void*>(a.spec), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
    const size_t sm = sizeof(Smem) + 1024;
    static unsigned configured = 0;
    cudaError_t e = set_smem_once(k_xtch<CB, N>, sm, &configured);
    if (e != cudaSuccess) return e;
    const long long nitems = (long long)a.nsb * (a.nchan / CB);
    const int grid = nitems < nsm ? (int)nitems : nsm;
    k_xtch<CB, N><<<grid, NTHREADS, sm, st>>>(map, a, d_err);
    return cudaGetLastError();
}

cudaError_t launch_xtch(const XArgs& a, int* d_err, int nsm, cudaStream_t st)
{
    using namespace tcxh;
    const int nslot = a.ntk ? a.ntk : a.T;
    if (a.nsig < 1 || a.nsig > MAXSIG || a.nchan % 8 != 0 || a.nchan < 8 || a.T % BT != 0 || nslot % (2 * BT) != 0 ||
        nslot > a.T || a.nsb < 1 || !a.spec || !a.acc)
        return cudaErrorInvalidValue;
    static_assert(sizeof(Smem) + 1024 <= 227 * 1024, "one CTA's shared memory");
    if (a.nsig > 32) return launch_xtch_t<4, 128>(a, d_err, nsm, st);
    // Up to 32 signals, items of 4 channels (still 64 accumulator columns each) where one round of them is enough: an
    // item of 8 takes 1.5 to 1.7 times as long, which pays only where it saves rounds.  128 to 512 channels, 4096
    // FFTs, 8 / 4 channels: 4 signals 123 / 72 us, 16 113 / 78, 32 131 / 87; two rounds of 4, 1024 channels, 4 signals
    // 123 / 163 (with 128 columns).
    if ((long long)a.nsb * (a.nchan / 4) <= nsm) return launch_xtch_t<4, 64>(a, d_err, nsm, st);
    return launch_xtch_t<8, 64>(a, d_err, nsm, st);
}

}  // namespace fx
