// The Miller-Rabin engine's handle, and the launches of its integer kernels
// (mr_int.cu) for the host code (mr.cu).
#pragma once
#include <cuda_runtime.h>

#include "mr_device.cuh"
#include "mr_fft.h"
#include "mr_job.cuh"

struct pfb_mr {
    int device = 0;
    int num_sms = 0;
    cudaStream_t stream = nullptr;
    uint32_t *d_tw = nullptr;
    uint32_t *d_wide = nullptr;
    pfb::mr::Twiddles tw{};
    pfb::mr::WideTabs wt{};  // (each source with integer kernels has its own constant copy)
    pfb::mr::fp::Engine fe;
    // persistent-kernel parameters per transform length (pfb_mr_autotune):
    // steps of one candidate per quantum, steps per launch
    int quantum[pfb::mr::LOG_LMAX + 1];
    int chunk[pfb::mr::LOG_LMAX + 1];
};

namespace pfb {
namespace mr {

// Constant tables and shared-memory limits, once per engine.
int int_setup(const CrtConsts &cc, const WideTabs &wt);

void *int_persist_func();  // persist_kernel

cudaError_t int_prep(JobDev *jobs, const int *list, int n, int maxlog, const Twiddles &tw, cudaStream_t st);

cudaError_t int_ctx(const JobDev *jobs, const CtxExtra *ex, int n, int maxlog, const uint64_t *a, const uint64_t *b,
                    uint64_t *out, int n16, int out_stride, int op, const Twiddles &tw, cudaStream_t st);

cudaError_t int_ctx_check(const uint64_t *r, const uint64_t *one, const uint64_t *nm1, uint8_t *passed, int n,
                          int n16, cudaStream_t st);

}  // namespace mr
}  // namespace pfb
