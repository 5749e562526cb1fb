// fx_fstage_f512.cu -- F-stage kernels for FFT length 512 (see fx_fpair.cuh, fx_fscalar.cuh).
#include "fx_fpair.cuh"
#include "fx_fscalar.cuh"

namespace fx {

cudaError_t launch_fstage_512(int mode, const FArgs& a, cudaStream_t st)
{
    return a.exact8 ? launch_fscalar_F<512>(a, st) : launch_fstage_F<512>(mode, a, st);
}

cudaError_t launch_fstage_batch_512(int mode, int npol, int tb, const FArgs* d_jobs, const int4* d_tasks, int ntask,
                                  int* ctr, cudaStream_t st)
{
    return launch_fstage_batch_F<512>(mode, npol, tb, d_jobs, d_tasks, ntask, ctr, st);
}

}  // namespace fx
