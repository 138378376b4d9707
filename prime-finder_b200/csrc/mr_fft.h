// Host side of the floating-point Montgomery engine (fft_device.cuh): its
// tables and launches, by length class.  Implemented in mr_fft.cu.
#pragma once
#include <cuda_runtime.h>

#include "fft_device.cuh"
#include "mr_job.cuh"

namespace pfb {
namespace mr {
namespace fp {

struct Engine {
    Cplx *mem = nullptr;     // roots of all classes
    Tab tab[kClasses];
    int per_sm[kClasses];    // resident CTAs per SM
};

int engine_create(Engine &e);
void engine_free(Engine &e);

// Points of device scratch the persistent kernel of a class needs per CTA.
size_t scratch_points(int cls);

// Arguments and launch shape of one launch of the persistent kernel.
struct Launch {
    void *func;
    dim3 grid, block;
    size_t smem;
};
Launch persist_launch(const Engine &e, int cls, int n, int sms);

cudaError_t prep(const Engine &e, int cls, JobDev *jobs, const int *d_list, int n, cudaStream_t st);

}  // namespace fp
}  // namespace mr
}  // namespace pfb
