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

// Contexts have the integer engine's lengths: powers of two from 2^7 on.
template <class F>
constexpr bool in_ctx() {
    return F::C >= 128 && (F::C & (F::C - 1)) == 0;
}

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
    PFB_CUDA(cudaFuncSetAttribute(fft_persist_kernel<F, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)F::smem()));
    PFB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&e.per_sm[0][F::ID], fft_persist_kernel<F>, F::T,
                                                           F::smem()));
    PFB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&e.per_sm[1][F::ID], fft_persist_kernel<F, true>, F::T,
                                                           F::smem()));
    if constexpr (in_ctx<F>())
        PFB_CUDA(cudaFuncSetAttribute(fft_ctx_kernel<F>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)F::smem()));
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

Launch persist_launch(const Engine &e, bool lucas, int cls, int n, int sms) {
    Launch l{};
    const int grid = std::max(1, std::min(n, sms * std::max(1, e.per_sm[lucas][cls])));
    switch (cls) {
#define PFB_CLS(F)                                                                                    \
    case F::ID:                                                                                       \
        l = Launch{lucas ? (void *)fft_persist_kernel<F, true> : (void *)fft_persist_kernel<F, false>, \
                   dim3(grid), dim3(F::T), F::smem()};                                                \
        break;
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

namespace {

template <class F>
void launch_ctx(const Tab &tab, const JobDev *jobs, const int *list, int n, const uint64_t *a, const uint64_t *b,
                uint64_t *out, int n16, int op, const CtxExtra *ex, cudaStream_t st) {
    if constexpr (in_ctx<F>())
        fft_ctx_kernel<F><<<n, F::T, F::smem(), st>>>(jobs, list, a, b, out, n16, op, tab, ex);
}

}  // namespace

cudaError_t ctx(const Engine &e, int cls, const JobDev *jobs, const int *d_list, int n, const uint64_t *a,
                const uint64_t *b, uint64_t *out, int n16, int op, const CtxExtra *ex,
                cudaStream_t st) {
    switch (cls) {
#define PFB_CLS(F)                                                                                                \
    case F::ID: launch_ctx<F>(e.tab[F::ID], jobs, d_list, n, a, b, out, n16, op, ex, st); break;
        PFB_FP_CLASSES(PFB_CLS)
#undef PFB_CLS
    }
    return cudaGetLastError();
}

}  // namespace fp
}  // namespace mr
}  // namespace pfb
