// fx_fstage.cu -- dispatch of the fused F stage by FFT length (kernels in fx_fpair.cuh, one translation
// unit per length) and the debug unpack export.
#include "fx_fstage.cuh"

namespace fx {

cudaError_t launch_fstage_256(int mode, const FArgs& a, cudaStream_t st);
cudaError_t launch_fstage_batch_256(int mode, int npol, int tb, const FArgs* d_jobs, const int4* d_tasks, int ntask,
                                  int* ctr, cudaStream_t st);
cudaError_t launch_fstage_512(int mode, const FArgs& a, cudaStream_t st);
cudaError_t launch_fstage_batch_512(int mode, int npol, int tb, const FArgs* d_jobs, const int4* d_tasks, int ntask,
                                  int* ctr, cudaStream_t st);
cudaError_t launch_fstage_1024(int mode, const FArgs& a, cudaStream_t st);
cudaError_t launch_fstage_batch_1024(int mode, int npol, int tb, const FArgs* d_jobs, const int4* d_tasks, int ntask,
                                  int* ctr, cudaStream_t st);
cudaError_t launch_fstage_2048(int mode, const FArgs& a, cudaStream_t st);
cudaError_t launch_fstage_batch_2048(int mode, int npol, int tb, const FArgs* d_jobs, const int4* d_tasks, int ntask,
                                  int* ctr, cudaStream_t st);
cudaError_t launch_fstage_4096(int mode, const FArgs& a, cudaStream_t st);
cudaError_t launch_fstage_batch_4096(int mode, int npol, int tb, const FArgs* d_jobs, const int4* d_tasks, int ntask,
                                  int* ctr, cudaStream_t st);
cudaError_t launch_fstage_8192(int mode, const FArgs& a, cudaStream_t st);
cudaError_t launch_fstage_batch_8192(int mode, int npol, int tb, const FArgs* d_jobs, const int4* d_tasks, int ntask,
                                  int* ctr, cudaStream_t st);

cudaError_t launch_fstage(int nchan, int mode, const FArgs& a, cudaStream_t st)
{
    // the FP16 tensor-core DFT only where the context asked for it (fxc_config.fstage);
    // the configuration check admits it only for geometries it covers
    if (a.fkind == FXC_F_TC16) {
        if (!ftc_supported(nchan, mode, a)) return cudaErrorInvalidValue;
        return launch_ftc(a, st);
    }
    if (a.fkind == FXC_F_TC32) {
        if (!ftc32_supported(nchan, mode, a)) return cudaErrorInvalidValue;
        return launch_ftc32(mode, a, st);
    }
    if (mode == kSpecF16) return cudaErrorInvalidValue;   // the FFT kernels store channel-contiguous spectra
    switch (a.cpx ? nchan : 2 * nchan) {   // FFT length: complex samples fill every bin
    case 256: return launch_fstage_256(mode, a, st);
    case 512: return launch_fstage_512(mode, a, st);
    case 1024: return launch_fstage_1024(mode, a, st);
    case 2048: return launch_fstage_2048(mode, a, st);
    case 4096: return launch_fstage_4096(mode, a, st);
    case 8192: return launch_fstage_8192(mode, a, st);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_fstage_batch(int nchan, int npol, int mode, int tb, const FArgs* d_jobs, const int4* d_tasks,
                                int ntask, int* ctr, cudaStream_t st)
{
    switch (2 * nchan) {
    case 256: return launch_fstage_batch_256(mode, npol, tb, d_jobs, d_tasks, ntask, ctr, st);
    case 512: return launch_fstage_batch_512(mode, npol, tb, d_jobs, d_tasks, ntask, ctr, st);
    case 1024: return launch_fstage_batch_1024(mode, npol, tb, d_jobs, d_tasks, ntask, ctr, st);
    case 2048: return launch_fstage_batch_2048(mode, npol, tb, d_jobs, d_tasks, ntask, ctr, st);
    case 4096: return launch_fstage_batch_4096(mode, npol, tb, d_jobs, d_tasks, ntask, ctr, st);
    case 8192: return launch_fstage_batch_8192(mode, npol, tb, d_jobs, d_tasks, ntask, ctr, st);
    default: return cudaErrorInvalidValue;
    }
}

// Debug export of the unpacked (pre-rotation) samples, decoded byte by byte: out[sb][ant][pol][t][n] for n < F, zero where the
// antenna is invalid for FFT t.
template <int F>
__global__ void k_unpack_debug(FArgs args, float* out)
{
    __shared__ __align__(16) uint8_t inb[F / 2 + 16];
    const int tc = blockIdx.x, ant = blockIdx.y, sb = blockIdx.z;
    const int npol = args.npol;
    const DelayEntry d = args.dtab[(size_t)ant * args.ld + args.t_base + tc];
    const uint8_t* row = args.data + ((size_t)sb * args.nant + ant) * args.pitch;
    int base_byte = 0;
    if (d.valid) base_byte = stage_fft_bytes(row, d.offset, npol, F, inb, threadIdx.x, blockDim.x);
    __syncthreads();
    for (int pol = 0; pol < npol; pol++) {
        float* o = out + ((((size_t)sb * args.nant + ant) * npol + pol) * args.nfft + tc) * F;
        for (int n = threadIdx.x; n < F; n += blockDim.x) {
            float lv = 0.f;
            if (d.valid) lv = decode_sample(inb, base_byte, d.offset + n, npol, pol);
            o[n] = lv;
        }
    }
}

cudaError_t launch_unpack_debug(int nchan, const FArgs& a, float* out, cudaStream_t st)
{
    dim3 grid(a.nfft, a.nant, a.nsb);
    switch (2 * nchan) {
    case 256: k_unpack_debug<256><<<grid, 128, 0, st>>>(a, out); break;
    case 512: k_unpack_debug<512><<<grid, 128, 0, st>>>(a, out); break;
    case 1024: k_unpack_debug<1024><<<grid, 128, 0, st>>>(a, out); break;
    case 2048: k_unpack_debug<2048><<<grid, 128, 0, st>>>(a, out); break;
    case 4096: k_unpack_debug<4096><<<grid, 128, 0, st>>>(a, out); break;
    case 8192: k_unpack_debug<8192><<<grid, 128, 0, st>>>(a, out); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

// Failure-path check: the F stage's bounded staging wait on an mbarrier that nothing
// completes (no copy is ever issued, so nothing is left in flight) runs out after 1 s and
// records code 6 in the error word, as an expired input copy would.
__global__ void k_expire_wait(int* err)
{
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        stg_bar_init(&bar);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (!stg_wait(&bar, 0)) atomicCAS(err, 0, 6);
    }
}

cudaError_t launch_expire_wait(int* err, cudaStream_t st)
{
    k_expire_wait<<<1, 32, 0, st>>>(err);
    return cudaGetLastError();
}

}  // namespace fx
