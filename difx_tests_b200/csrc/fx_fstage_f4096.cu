// fx_fstage_f4096.cu -- F-stage kernels for FFT length 4096 (see fx_fpair.cuh, fx_fscalar.cuh).
#include "fx_fpair.cuh"
#include "fx_fscalar.cuh"

namespace fx {

cudaError_t launch_fstage_4096(int mode, const FArgs& a, cudaStream_t st)
{
    return a.exact8 ? launch_fscalar_F<4096>(a, st) : launch_fstage_F<4096>(mode, a, st);
}

cudaError_t launch_fstage_batch_4096(int mode, int npol, int tb, const FArgs* d_jobs, const int4* d_tasks, int ntask,
                                  int* ctr, cudaStream_t st)
{
    return launch_fstage_batch_F<4096>(mode, npol, tb, d_jobs, d_tasks, ntask, ctr, st);
}

}  // namespace fx
