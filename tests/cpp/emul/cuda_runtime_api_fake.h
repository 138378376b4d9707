// Host stand-in for the CUDA runtime API, for running the engine's host code
// (mr.cu) on the CPU in the tests: device memory is host memory under a limit
// on bytes and on calls, copies are memcpy, everything is done when the call
// returns, and a kernel launch calls fake::launch.
#pragma once
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include <functional>
#include <map>
#include <mutex>
#include <vector>

enum : int { cudaErrorMemoryAllocation = 2, cudaDevAttrMultiProcessorCount = 16, cudaStreamNonBlocking = 1,
             cudaEventDisableTiming = 2 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1, cudaMemcpyDeviceToHost = 2, cudaMemcpyDeviceToDevice = 3 };

struct dim3 {
    unsigned x, y, z;
    dim3(unsigned x_ = 1, unsigned y_ = 1, unsigned z_ = 1) : x(x_), y(y_), z(z_) {}
};

typedef int *cudaStream_t;
typedef int *cudaEvent_t;
#define cudaStreamLegacy ((cudaStream_t)0x1)

struct cudaMemsetParams {
    void *dst;
    size_t pitch;
    unsigned value, elementSize;
    size_t width, height;
};
struct cudaKernelNodeParams {
    void *func;
    dim3 gridDim, blockDim;
    unsigned sharedMemBytes;
    void **kernelParams;
    void **extra;
};

namespace fake {

// Device memory.
inline std::mutex mu;
inline std::map<void *, size_t> blocks;
inline size_t used = 0, peak = 0, limit = ~(size_t)0;
inline long allow = -1;  // allocations left (-1: no limit)
inline bool no_streams = false;  // no further stream can be created

// What a launch of `func` with these arguments does, ready to be called once
// the argument array is gone; set by the test.
inline std::function<std::function<void()>(void *func, void **args)> launch;

struct Graph {
    std::vector<std::function<void()>> nodes;
};

}  // namespace fake

typedef fake::Graph *cudaGraph_t;
typedef fake::Graph *cudaGraphExec_t;
typedef int *cudaGraphNode_t;

template <class T>
inline cudaError_t cudaMalloc(T **p, size_t n) {
    std::lock_guard<std::mutex> lk(fake::mu);
    if (fake::allow == 0 || fake::used + n > fake::limit) {
        return cudaErrorMemoryAllocation;
    }
    if (fake::allow > 0) fake::allow--;
    void *m = aligned_alloc(256, (n + 256) & ~(size_t)255);
    memset(m, 0xAB, n);  // (not zero)
    fake::blocks[m] = n;
    fake::used += n;
    if (fake::used > fake::peak) fake::peak = fake::used;
    *p = (T *)m;
    return cudaSuccess;
}
inline cudaError_t cudaFree(void *p) {
    if (!p) return cudaSuccess;
    std::lock_guard<std::mutex> lk(fake::mu);
    fake::used -= fake::blocks.at(p);
    fake::blocks.erase(p);
    free(p);
    return cudaSuccess;
}
inline cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
    memcpy(d, s, n);
    return cudaSuccess;
}
inline cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    memcpy(d, s, n);
    return cudaSuccess;
}
inline cudaError_t cudaMemset(void *d, int v, size_t n) {
    memset(d, v, n);
    return cudaSuccess;
}
inline cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) {
    memset(d, v, n);
    return cudaSuccess;
}
inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
inline cudaError_t cudaDeviceGetAttribute(int *v, int, int) {
    *v = 4;  // SMs
    return cudaSuccess;
}
inline cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, int) {
    if (fake::no_streams) return cudaErrorMemoryAllocation;
    *s = new int(0);
    return cudaSuccess;
}
inline cudaError_t cudaStreamDestroy(cudaStream_t s) {
    delete s;
    return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, int) { return cudaSuccess; }
inline cudaError_t cudaEventCreate(cudaEvent_t *e) {
    *e = new int(0);
    return cudaSuccess;
}
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, int) { return cudaEventCreate(e); }
inline cudaError_t cudaEventDestroy(cudaEvent_t e) {
    delete e;
    return cudaSuccess;
}
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.f;
    return cudaSuccess;
}
inline cudaError_t cudaLaunchKernel(void *func, dim3, dim3, void **args, size_t, cudaStream_t) {
    fake::launch(func, args)();
    return cudaSuccess;
}
inline cudaError_t cudaGraphCreate(cudaGraph_t *g, int) {
    *g = new fake::Graph();
    return cudaSuccess;
}
inline cudaError_t cudaGraphDestroy(cudaGraph_t g) {
    delete g;
    return cudaSuccess;
}
inline cudaError_t cudaGraphAddMemsetNode(cudaGraphNode_t *, cudaGraph_t g, const cudaGraphNode_t *, size_t,
                                          const cudaMemsetParams *p) {
    const cudaMemsetParams m = *p;
    g->nodes.push_back([m] { memset(m.dst, (int)m.value, m.width * m.elementSize); });
    return cudaSuccess;
}
inline cudaError_t cudaGraphAddKernelNode(cudaGraphNode_t *, cudaGraph_t g, const cudaGraphNode_t *, size_t,
                                          const cudaKernelNodeParams *p) {
    g->nodes.push_back(fake::launch(p->func, p->kernelParams));
    return cudaSuccess;
}
inline cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t g, int) {
    *e = new fake::Graph(*g);
    return cudaSuccess;
}
inline cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) {
    delete e;
    return cudaSuccess;
}
inline cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
    for (auto &n : e->nodes) n();
    return cudaSuccess;
}
