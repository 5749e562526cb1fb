// fx_kernels.h -- host-side launchers of the sm_100a kernels (internal).
#pragma once

#include <cuda_runtime.h>

#include "fx_internal.h"

namespace fx {

cudaError_t launch_delay_table(const double* delays, const double* fileoffsets, const int* fftindex, int first,
                               int nant, int nfft, int ld, int F, int maxoffset, double sampletime, DelayEntry* tab,
                               uint32_t* vbits, cudaStream_t st);
// as launch_delay_table, for input windows: antenna a's rows start at sample win[a] and hold
// win[nant + a] samples (device doubles holding integers; spb samples per byte); FFTs not inside
// their window are left out and set kWindowMiss in *err
cudaError_t launch_delay_table_window(const double* delays, const double* fileoffsets, const int* fftindex,
                                      int first, int nant, int nfft, int ld, int F, int maxoffset, double sampletime,
                                      const double* win, int spb, int* err, DelayEntry* tab, uint32_t* vbits,
                                      cudaStream_t st);
cudaError_t launch_counts(const uint32_t* vbits, int nant, int nwords, int* counts, cudaStream_t st);
cudaError_t launch_finalize(const float2* acc, int acc_layout, int nsig, int npol, int nant, int nchan, int nsb,
                            const int* counts, int normalize, float2* vis, cudaStream_t st);
cudaError_t launch_amp_phase(float2* vis, long long n, cudaStream_t st);
cudaError_t launch_fstage(int nchan, int mode, const FArgs& a, cudaStream_t st);
// tensor-core F stage (F16 layout, 2048-point FFTs of one polarisation of 2-bit real input)
bool ftc_supported(int nchan, int mode, const FArgs& a);
cudaError_t launch_ftc(const FArgs& a, cudaStream_t st);
// FP32-grade tensor-core F stage (error-compensated FP16 pairs), same geometry, F16 or F32 layout
bool ftc32_supported(int nchan, int mode, const FArgs& a);
cudaError_t launch_ftc32(int mode, const FArgs& a, cudaStream_t st);
// FP16 spectra [sb][sig][src_T][chan] -> K-major [sb][chan][rows][dst_T] from slot t_off on (fx_kmajor.cu)
cudaError_t launch_kmajor(const void* src, int src_T, int span, int nsb, int nsig, int nchan, int rows, void* dst,
                          int dst_T, int t_off, unsigned* amax, cudaStream_t st);
// the same for many jobs in one launch, each [sb][sig][src_T][chan] -> [sb][chan][rows][dst_T], slots [0, span)
// (multiples of 64); first: blocks of the jobs before it
struct KJob {
    const void* src;
    void* dst;
    int src_T, dst_T, span, nsb, nsig, nchan, rows, first;
};
int kmajor_blocks(const KJob& j);
cudaError_t launch_kmajor_batch(const KJob* d_jobs, int njobs, int nblocks, cudaStream_t st);
cudaError_t launch_fstage_batch(int nchan, int npol, int mode, int tb, const FArgs* d_jobs, const int4* d_tasks,
                                int ntask, int* ctr, cudaStream_t st);
cudaError_t launch_xplain_reduce(const XArgs& a, cudaStream_t st);
void xplain_segments(int nsig, int nchan, int nsb, int T, int nsm, int* tseg, int* tlen);
void xplain_segment_model(long long ctas, long long slots, int T, int* tseg, int* tlen);
int xplain_segments_used(const XArgs& a);
cudaError_t launch_xplain(const XArgs& a, cudaStream_t st);
// whether the plain form of this geometry takes launch_xsplit (else launch_xplain); calls of fewer than
// kXsplitMinFfts FFTs take launch_xplain either way
constexpr int kXsplitMinFfts = 32;
bool xsplit_pays(int nsig, int nchan, int nsb, int numffts, int nsm);
// the plain form's sums on the tensor cores, each FP32 value as an FP16 pair of 22 bits (up to 64 signals); cpx:
// 8-bit complex input (spectra beyond FP16's range); spectra in the layout kSpecP32
cudaError_t launch_xsplit(const XArgs& a, int npol, int cpx, int* d_err, int nsm, cudaStream_t st);
// the same for the jobs of a batch (2-bit samples) in one launch.  Work item n of xsplit_items(a) of job `job`, whose
// arguments are d_jobs[args]; 128 bytes per job of what the kernel reads its spectra by (at d_maps + 128 job, which is
// 64-byte aligned); nsig_max: signals of the largest job, all of them up to 32 or all above; d_errs: every job's
// error word
int xsplit_items(const XArgs& a);
int4 xsplit_item(const XArgs& a, int args, int job, int n);
cudaError_t xsplit_map_bytes(const XArgs& a, int npol, void* map128);
cudaError_t launch_xsplit_batch(int nsig_max, int npol, const XArgs* d_jobs, const void* d_maps, const int4* d_items,
                                int nitems, int* ctr, int* const* d_errs, int njobs, int nsm, cudaStream_t st);
cudaError_t launch_xplain_batch(int nsig, int alt, const XArgs* d_jobs, const int4* d_tasks, int ntask,
                                cudaStream_t st);
int xplain_channel_group(int nsig, int alt);
cudaError_t launch_xtc(const XArgs& a, int* d_err, int nsm, cudaStream_t st);
// the same Gram on the FFT F stage's channel-contiguous FP16 spectra, turned in shared memory (up to 64 signals)
cudaError_t launch_xtch(const XArgs& a, int* d_err, int nsm, cudaStream_t st);
// FP8 form: e4m3 copy of the F16 spectra scaled by 448/absmax per (item = sb*nchan + chan, signal),
// then the e4m3 Gram with the inverse scales applied per product
cudaError_t launch_cast_fp8(const void* spec16, const unsigned* amax, int rows, int nsig, int T, int ts, int nitems,
                            uint8_t* spec8, float* inv_scale, cudaStream_t st);
cudaError_t launch_xtc8(const XArgs& a, int* d_err, int nsm, cudaStream_t st);
size_t xtc_smem_bytes();
cudaError_t launch_unpack_debug(int nchan, const FArgs& a, float* out, cudaStream_t st);
// a bounded device wait that runs out (error word code 6), for tests of the failure path
cudaError_t launch_expire_wait(int* err, cudaStream_t st);
// the same for the tensor-core kernels' mbarrier wait (error word code 7)
cudaError_t launch_expire_wait_tc(int* err, cudaStream_t st);

}  // namespace fx
