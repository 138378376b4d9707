// The integer Montgomery engine's kernels (mr_kernels.cuh, mr_ctx_kernels.cuh)
// and their launches, apart from the host code: they take minutes to compile.
#include <algorithm>

#include "common.cuh"
#include "mr_ctx_kernels.cuh"
#include "mr_engine.h"
#include "mr_kernels.cuh"

namespace pfb {
namespace mr {

int int_setup(const CrtConsts &cc, const WideTabs &wt) {
    PFB_CUDA(cudaMemcpyToSymbol(c_crt, &cc, sizeof(cc)));
    PFB_CUDA(cudaMemcpyToSymbol(c_wide, &wt, sizeof(wt)));
    const int mx = (int)std::max(smem_bytes(LOG_LCTA), smem_bytes(LOG_LSEQ));
    PFB_CUDA(cudaFuncSetAttribute(persist_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, mx));
    PFB_CUDA(cudaFuncSetAttribute(prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, mx));
    PFB_CUDA(cudaFuncSetAttribute(ctx_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, mx));
    return PFB_OK;
}

void *int_persist_func() { return (void *)persist_kernel; }

cudaError_t int_prep(JobDev *jobs, const int *list, int n, int maxlog, const Twiddles &tw, cudaStream_t st) {
    prep_kernel<<<n, THREADS, smem_bytes(maxlog), st>>>(jobs, list, tw);
    return cudaGetLastError();
}

cudaError_t int_ctx(const JobDev *jobs, const CtxExtra *ex, int n, int maxlog, const uint64_t *a, const uint64_t *b,
                    uint64_t *out, int n16, int out_stride, int op, const Twiddles &tw, cudaStream_t st) {
    ctx_kernel<<<n, THREADS, smem_bytes(maxlog), st>>>(jobs, ex, a, b, out, n16, out_stride, op, tw);
    return cudaGetLastError();
}

cudaError_t int_ctx_check(const uint64_t *r, const uint64_t *one, const uint64_t *nm1, uint8_t *passed, int n,
                          int n16, cudaStream_t st) {
    ctx_check_kernel<<<n, 256, 0, st>>>(r, one, nm1, passed, n16);
    return cudaGetLastError();
}

}  // namespace mr
}  // namespace pfb
