// The floating-point Montgomery engine: instances of its kernels per length
// class, tables and launches.
#include <algorithm>
#include <vector>

#include "common.cuh"
#include "fft_kernels.cuh"
#include "fft_tables_host.h"
#include "mr_fft.h"

namespace pfb {
namespace mr {
namespace fp {

namespace {

template <class F>
int setup_class(Engine &e, std::vector<Cplx> &all) {
    size_t off[2][3] = {};
    const std::vector<Cplx> v = class_roots<F>(off);
    // offsets for now: turned into addresses once the table has one
    for (int mod = 0; mod < 2; mod++)
        for (int p = 0; p < 3; p++) e.tab[F::ID].t[mod][p] = (const Cplx *)((all.size() + off[mod][p]) * sizeof(Cplx));
    all.insert(all.end(), v.begin(), v.end());
    PFB_CUDA(cudaFuncSetAttribute(fft_persist_kernel<F>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)F::smem()));
    PFB_CUDA(cudaFuncSetAttribute(fft_prep_kernel<F>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)F::smem()));
    PFB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&e.per_sm[F::ID], fft_persist_kernel<F>, F::T, F::smem()));
    return PFB_OK;
}

}  // namespace

int engine_create(Engine &e) {
    std::vector<Cplx> all;
#define PFB_CLS(F)                               \
    {                                            \
        const int rc = setup_class<F>(e, all);   \
        if (rc) return rc;                       \
    }
    PFB_FP_CLASSES(PFB_CLS)
#undef PFB_CLS
    PFB_CUDA(cudaMalloc(&e.mem, all.size() * sizeof(Cplx)));
    PFB_CUDA(cudaMemcpy(e.mem, all.data(), all.size() * sizeof(Cplx), cudaMemcpyHostToDevice));
    for (auto &t : e.tab)
        for (auto &m : t.t)
            for (auto &p : m) p = (const Cplx *)((const char *)e.mem + (size_t)p);
    const First f = first_roots();
    PFB_CUDA(cudaMemcpyToSymbol(c_first, &f, sizeof(f)));
    return PFB_OK;
}

void engine_free(Engine &e) {
    cudaFree(e.mem);
    e.mem = nullptr;
}

size_t scratch_points(int cls) {
    switch (cls) {
#define PFB_CLS(F) \
    case F::ID: return F::SQS ? 0 : (size_t)F::C;
        PFB_FP_CLASSES(PFB_CLS)
#undef PFB_CLS
    }
    return 0;
}

Launch persist_launch(const Engine &e, int cls, int n, int sms) {
    Launch l{};
    const int grid = std::max(1, std::min(n, sms * std::max(1, e.per_sm[cls])));
    switch (cls) {
#define PFB_CLS(F) \
    case F::ID: l = Launch{(void *)fft_persist_kernel<F>, dim3(grid), dim3(F::T), F::smem()}; break;
        PFB_FP_CLASSES(PFB_CLS)
#undef PFB_CLS
    }
    return l;
}

cudaError_t prep(const Engine &e, int cls, JobDev *jobs, const int *d_list, int n, cudaStream_t st) {
    switch (cls) {
#define PFB_CLS(F)                                                                    \
    case F::ID: fft_prep_kernel<F><<<n, F::T, F::smem(), st>>>(jobs, d_list, e.tab[F::ID]); break;
        PFB_FP_CLASSES(PFB_CLS)
#undef PFB_CLS
    }
    return cudaGetLastError();
}

}  // namespace fp
}  // namespace mr
}  // namespace pfb
