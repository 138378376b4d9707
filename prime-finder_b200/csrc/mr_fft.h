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
    int per_sm[2][kClasses];  // resident CTAs per SM: strong tests, Lucas tests
};

int engine_create(Engine &e);
void engine_free(Engine &e);

// Arguments and launch shape of one launch of the persistent kernel.
struct Launch {
    void *func;
    dim3 grid, block;
    size_t smem;
};
Launch persist_launch(const Engine &e, bool lucas, int cls, int n, int sms);

cudaError_t ctx(const Engine &e, int cls, const JobDev *jobs, const int *d_list, int n, const uint64_t *a,
                const uint64_t *b, uint64_t *out, int n16, int op, const CtxExtra *ex,
                cudaStream_t st);

cudaError_t prep(const Engine &e, int cls, JobDev *jobs, const int *d_list, int n, cudaStream_t st);

}  // namespace fp
}  // namespace mr
}  // namespace pfb
