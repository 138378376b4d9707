// Batched Miller-Rabin engine: kernels and host driver.
//
// One CTA per candidate runs its whole chain of Montgomery squarings on chip:
// on double-precision FFTs (fft_device.cuh) up to 344 058 bits, on the integer
// transforms (mr_device.cuh) above.  The host side does the per-modulus set-up the reference
// does with GMP (barrett.cu:58-107, montgomery.cu:30-45,
// miller_rabin_runner.cu:315-325): N' = -N^-1 mod R, R mod N, N - 1 = 2^s d.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <thread>
#include <vector>

#include "bigint_host.h"
#include "common.cuh"
#include "lucas_host.h"
#include "mr_engine.h"
#include "mr_prep_host.h"
#include "mr_tables_host.h"
#include "pfb_mr.h"

using namespace pfb::mr;

static int build_tables(pfb_mr *e) {
    const int half = 1 << (LOG_LMAX - 1);
    const std::vector<uint32_t> h = twiddle_table();
    PFB_CUDA(cudaMalloc(&e->d_tw, h.size() * sizeof(uint32_t)));
    PFB_CUDA(cudaMemcpy(e->d_tw, h.data(), h.size() * sizeof(uint32_t), cudaMemcpyHostToDevice));
    for (int pr = 0; pr < 2; pr++) {
        uint32_t *base = e->d_tw + (size_t)(4 * pr) * half;
        e->tw.w[pr] = base;
        e->tw.wsh[pr] = base + half;
        e->tw.wi[pr] = base + 2 * half;
        e->tw.wish[pr] = base + 3 * half;
    }
    const CrtConsts cc = crt_consts();
    WideTabs wt{};
    const std::vector<uint32_t> wide = wide_tables(h, wt);
    PFB_CUDA(cudaMalloc(&e->d_wide, wide.size() * sizeof(uint32_t)));
    PFB_CUDA(cudaMemcpy(e->d_wide, wide.data(), wide.size() * sizeof(uint32_t), cudaMemcpyHostToDevice));
    wt.base = (const uint4 *)e->d_wide;
    e->wt = wt;
    return int_setup(cc, wt);
}

extern "C" int pfb_mr_device(const pfb_mr_t *e) { return e ? e->device : -1; }

extern "C" int pfb_mr_create(pfb_mr_t **out, int device) {
    if (!out) {
        pfb::set_error("pfb_mr_create: null out");
        return PFB_E_ARG;
    }
    *out = nullptr;
    pfb_mr *e = new pfb_mr();
    e->device = device;
    for (int lg = 0; lg <= LOG_LMAX; lg++) {
        e->quantum[lg] = 64;
        e->chunk[lg] = 2048;
    }
    int rc = PFB_OK;
    cudaError_t ce = cudaSetDevice(device);
    if (ce != cudaSuccess) rc = pfb::cuda_fail(ce, "cudaSetDevice", __FILE__, __LINE__);
    if (!rc) {
        ce = cudaDeviceGetAttribute(&e->num_sms, cudaDevAttrMultiProcessorCount, device);
        if (ce != cudaSuccess) rc = pfb::cuda_fail(ce, "attr", __FILE__, __LINE__);
    }
    if (!rc) {
        ce = cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking);
        if (ce != cudaSuccess) rc = pfb::cuda_fail(ce, "stream", __FILE__, __LINE__);
    }
    if (!rc) rc = build_tables(e);
    if (!rc) rc = fp::engine_create(e->fe);
    if (rc) {
        if (e->stream) cudaStreamDestroy(e->stream);
        cudaFree(e->d_tw);
        cudaFree(e->d_wide);
        fp::engine_free(e->fe);
        delete e;
        return rc;
    }
    *out = e;
    return PFB_OK;
}

extern "C" void pfb_mr_destroy(pfb_mr_t *e) {
    if (!e) return;
    cudaSetDevice(e->device);
    if (e->stream) {
        cudaStreamSynchronize(e->stream);
        cudaStreamDestroy(e->stream);
    }
    cudaFree(e->d_tw);
    cudaFree(e->d_wide);
    fp::engine_free(e->fe);
    delete e;
}

namespace {

// Per-candidate device layout inside the arena (32-bit words).
struct Layout {
    size_t x, res, nn, nh, npl, nl, exp, yb, lv0, lv1, lqk, lt, lone, gy, raw, sq, total;
};

Layout layout_for(int logl, size_t exp_words, bool lucas = false, bool raw = false) {
    const size_t L = (size_t)1 << logl, H = L / 2;
    Layout l{};
    size_t o = 0;
    auto take = [&](size_t words) {
        const size_t at = o;
        o += (words + 63) & ~(size_t)63;  // 256-byte alignment
        return at;
    };
    l.x = take(H);
    l.res = take(H);
    l.nn = take(2 * H);
    l.nh = take(2 * H);
    l.npl = take(H);
    l.nl = take(H);
    l.exp = take(exp_words);
    if (logl > LOG_LCTA) l.yb = take(H + H / 32);  // padded like the shared-memory residue
    if (lucas) {
        l.lv0 = take(H);
        l.lv1 = take(H);
        l.lqk = take(H);
        l.lt = take(H);
        l.lone = take(H);
        l.gy = take(2 * L);
    }
    if (raw) l.raw = take(2 * L);  // L 64-bit coefficients
    l.total = o;
    return l;
}

// Layout of a candidate of the floating-point engine: n = 2 C digits, spectra
// of C points (4 words each); x^2's spectrum takes the place of N'', which only
// the set-up reads.  ctx_logl: a modulus of a context instead, with the buffers
// of the integer engine's raw products at that transform length: the second
// factor's limbs take the place of N'' too, and a modular product has its
// second factor's spectra (2 C points) where gy and raw lie, one behind the
// other.
Layout layout_fp(int cls, size_t exp_words, bool lucas, int ctx_logl = 0) {
    const size_t C = (size_t)fp::class_points(cls), n = 2 * C;
    Layout l{};
    size_t o = 0;
    auto take = [&](size_t words) {
        const size_t at = o;
        o += (words + 63) & ~(size_t)63;
        return at;
    };
    l.nn = take(4 * C);
    l.nh = take(4 * C);
    l.npl = l.sq = l.lt = take(fp::spectrum_outside(cls) ? 4 * C : n);
    l.nl = take(n);
    if (ctx_logl) {
        const size_t L = (size_t)1 << ctx_logl;
        l.gy = take(2 * L);
        l.raw = take(2 * L);
    } else {
        l.x = take(n);
        l.res = take(n);
        l.exp = take(exp_words);
    }
    if (lucas) {
        l.lv0 = take(n);
        l.lv1 = take(n);
        l.lqk = take(n);
        l.lt = take(n);
        l.lone = take(n);
        l.gy = take(8 * C);
    }
    l.total = o;
    return l;
}

Layout layout_for(const HostPrep &hp, bool lucas) {
    return hp.fpc ? layout_fp(hp.fpc - 1, hp.exp.size(), lucas) : layout_for(hp.logl, hp.exp.size(), lucas);
}

// Bits of a digit of a candidate's x0, npl, nl and residue.
int digit_bits(const HostPrep &hp) { return hp.fpc ? hp.fbits : LIMB_BITS; }

// The unfinished candidates by engine: the integer engine's count, and per
// length class of the floating-point engine a run of `order` (job indices).
struct ClassRuns {
    int n_int = 0;
    int first[fp::kClasses] = {}, count[fp::kClasses] = {};
    std::vector<int> order;
    template <class Live, class Fpc>
    void build(int n, Live live, Fpc fpc) {
        n_int = 0;
        order.clear();
        for (int i = 0; i < n; i++) n_int += live(i) && !fpc(i);
        for (int c = 0; c < fp::kClasses; c++) {
            first[c] = (int)order.size();
            for (int i = 0; i < n; i++)
                if (live(i) && fpc(i) == c + 1) order.push_back(i);
            count[c] = (int)order.size() - first[c];
        }
    }
};

// Quanta of one launch of a class: jobs that each have a CTA of their own run
// their whole chunk in one quantum.
void fp_quanta(const pfb_mr *e, bool lucas, int cls, int n, long long chunk, int tuned, int *quantum, unsigned *total) {
    const int ctas = (int)fp::persist_launch(e->fe, lucas, cls, n, e->num_sms).grid.x;
    *quantum = (int)(n <= ctas ? chunk : std::min<long long>(chunk, tuned));
    *total = (unsigned)std::min<long long>((long long)n * ((chunk + *quantum - 1) / *quantum), 0x7fffffffll);
}

// Slot layout of the server: the exponent region sized for the longest
// modulus of the length class, so that slots of one class are interchangeable.
// The length class is the transform length's logarithm, or for the
// floating-point engine kFpKey + its class.
constexpr int kFpKey = 64;
int slot_key(const HostPrep &hp) { return hp.fpc ? kFpKey + hp.fpc - 1 : hp.logl; }
Layout slot_layout(int key) {
    if (key >= kFpKey) {
        const int cls = key - kFpKey;
        return layout_fp(cls, ((size_t)fp::limb_bits(cls) * 2 * fp::class_points(cls) + 31) / 32 + 1, false);
    }
    const size_t H = (size_t)1 << (key - 1);
    return layout_for(key, (LIMB_BITS * H + 31) / 32 + 1);
}

size_t slot_bytes(int key) { return slot_layout(key).total * sizeof(uint32_t); }

// fft: candidates that the floating-point engine can hold are set up for it.
void prep_all(const pfb_mr_number_t *nums, int n, uint32_t base, int mode, const pfb_mr_number_t *exps,
              std::vector<HostPrep> &hp, bool fft) {
    hp.resize(n);
    const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
    const int nt = (int)std::min<unsigned>(hw, (unsigned)std::max(1, n));
    if (nt <= 1 || n < 4) {
        for (int i = 0; i < n; i++) host_prep(nums[i], base, mode, exps ? exps + i : nullptr, hp[i], fft);
        return;
    }
    std::vector<std::thread> th;
    for (int t = 0; t < nt; t++)
        th.emplace_back([&, t]() {
            for (int i = t; i < n; i += nt)
                host_prep(nums[i], base, mode, exps ? exps + i : nullptr, hp[i], fft);
        });
    for (auto &x : th) x.join();
}

}  // namespace

// A set of candidates resident in device memory, advanced step by step.
struct pfb_mr_batch {
    pfb_mr *e = nullptr;
    int n = 0, mode = 1, maxlog = LOG_LMIN, n_ok = 0;
    long long max_steps = 0, steps_done = 0;
    uint8_t *d_arena = nullptr;
    JobDev *d_jobs = nullptr;
    int *d_locks = nullptr;           // [n] per-candidate locks of the persistent kernel
    unsigned int *d_counter = nullptr;  // quanta handed out in the current launch: integer engine, then per class
    ClassRuns runs;
    int *d_order = nullptr;             // runs.order
    LucasDev *d_lucas = nullptr;        // [n] (strong Lucas batches only)
    std::vector<HostPrep> hp;
    std::vector<JobDev> jobs;
    std::vector<LucasDev> lucas;
    struct Graph {
        long long chunk;
        int quantum;
        cudaGraphExec_t exec;
    };
    std::vector<Graph> graphs;  // one launch of the persistent kernel per (chunk, quantum)
};

namespace {

void batch_free(pfb_mr_batch *b) {
    for (auto &g : b->graphs) cudaGraphExecDestroy(g.exec);
    cudaFree(b->d_arena);
    delete b;
}

// One step chunk of a batch -- the quanta counter reset and the persistent
// kernel -- as a CUDA graph, built on first use per (chunk, quantum) and
// replayed by every later advance of the batch.
int chunk_graph(pfb_mr_batch *b, long long chunk, int quantum, cudaGraphExec_t *out) {
    for (const auto &g : b->graphs)
        if (g.chunk == chunk && g.quantum == quantum) {
            *out = g.exec;
            return PFB_OK;
        }
    JobDev *jobs = b->d_jobs;
    int n = b->n, q = quantum;
    int *locks = b->d_locks;
    unsigned int *counter = b->d_counter;
    const long long qpj = (chunk + quantum - 1) / quantum;
    unsigned int total = (unsigned int)std::min<long long>((long long)b->runs.n_int * qpj, 0x7fffffffll);
    Twiddles tw = b->e->tw;
    void *args[] = {&jobs, &n, &locks, &counter, &total, &q, &tw};
    cudaGraph_t graph = nullptr;
    PFB_CUDA(cudaGraphCreate(&graph, 0));
    cudaMemsetParams mp{};
    mp.dst = counter;
    mp.value = 0;
    mp.elementSize = sizeof(unsigned int);
    mp.width = 1 + fp::kClasses;
    mp.height = 1;
    cudaGraphNode_t n_mem = nullptr, n_ker = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaError_t ce = cudaGraphAddMemsetNode(&n_mem, graph, nullptr, 0, &mp);
    if (ce == cudaSuccess && b->runs.n_int) {
        cudaKernelNodeParams kp{};
        kp.func = int_persist_func();
        kp.gridDim = dim3((unsigned)std::min(b->runs.n_int, std::max(1, b->e->num_sms)));
        kp.blockDim = dim3(THREADS);
        kp.sharedMemBytes = (unsigned)smem_bytes(b->maxlog);
        kp.kernelParams = args;
        ce = cudaGraphAddKernelNode(&n_ker, graph, &n_mem, 1, &kp);
    }
    // the length classes' kernels side by side, the longest numbers first
    for (int c = fp::kClasses - 1; c >= 0 && ce == cudaSuccess; c--) {
        int nc = b->runs.count[c], qc = 0;
        if (!nc) continue;
        unsigned tc = 0;
        fp_quanta(b->e, b->mode == 2, c, nc, chunk, quantum, &qc, &tc);
        const fp::Launch l = fp::persist_launch(b->e->fe, b->mode == 2, c, nc, b->e->num_sms);
        const int *order = b->d_order + b->runs.first[c];
        unsigned int *cnt = counter + 1 + c;
        fp::Tab tab = b->e->fe.tab[c];
        void *fa[] = {&jobs, &order, &nc, &locks, &cnt, &tc, &qc, &tab};
        cudaKernelNodeParams kp{};
        kp.func = l.func;
        kp.gridDim = l.grid;
        kp.blockDim = l.block;
        kp.sharedMemBytes = (unsigned)l.smem;
        kp.kernelParams = fa;
        ce = cudaGraphAddKernelNode(&n_ker, graph, &n_mem, 1, &kp);
    }
    if (ce == cudaSuccess) ce = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ce != cudaSuccess) return pfb::cuda_fail(ce, "chunk graph", __FILE__, __LINE__);
    b->graphs.push_back(pfb_mr_batch::Graph{chunk, quantum, exec});
    *out = exec;
    return PFB_OK;
}

int batch_build_on(pfb_mr *e, const pfb_mr_number_t *nums, int n, uint32_t base, int mode,
                   const pfb_mr_number_t *exps, bool fft, pfb_mr_batch **out) {
    *out = nullptr;
    if (!e || !nums || n <= 0 || base < 2 || base > 0xFFFFu) {
        pfb::set_error("pfb_mr: bad argument (n=%d base=%u)", n, base);
        return PFB_E_ARG;
    }
    PFB_CUDA(cudaSetDevice(e->device));
    pfb_mr_batch *b = new pfb_mr_batch();
    b->e = e;
    b->n = n;
    b->mode = mode;
    prep_all(nums, n, base, mode, exps, b->hp, fft);
    std::vector<Layout> lay(n);
    size_t total = 0;
    for (int i = 0; i < n; i++) {
        if (!b->hp[i].ok || b->hp[i].decided >= 0) continue;
        lay[i] = layout_for(b->hp[i], mode == 2);
        total += lay[i].total;
        b->maxlog = std::max(b->maxlog, b->hp[i].logl);  // (by size: also for the floating-point engine)
        b->max_steps = std::max(b->max_steps, (long long)b->hp[i].cursor + 2 + b->hp[i].s);
        b->n_ok++;
    }
    const size_t job_bytes = ((size_t)n * sizeof(JobDev) + 255) & ~(size_t)255;
    const size_t lock_bytes = ((size_t)n * sizeof(int) + 256 + 255) & ~(size_t)255;
    const size_t lucas_bytes = mode == 2 ? (((size_t)n * sizeof(LucasDev) + 255) & ~(size_t)255) : 0;
    b->runs.build(n, [&](int i) { return b->hp[i].ok && b->hp[i].decided < 0; }, [&](int i) { return b->hp[i].fpc; });
    const size_t order_bytes = (b->runs.order.size() * sizeof(int) + 255) & ~(size_t)255;
    const size_t need = job_bytes + lock_bytes + lucas_bytes + order_bytes + total * sizeof(uint32_t);
    if (cudaMalloc(&b->d_arena, need) != cudaSuccess) {
        cudaGetLastError();
        pfb::set_error("pfb_mr: cannot allocate %zu bytes of device memory", need);
        delete b;
        return PFB_E_NOMEM;
    }
    b->d_jobs = (JobDev *)b->d_arena;
    b->d_locks = (int *)(b->d_arena + job_bytes);
    b->d_counter = (unsigned int *)(b->d_arena + job_bytes + lock_bytes - 256);
    if (mode == 2) {
        b->d_lucas = (LucasDev *)(b->d_arena + job_bytes + lock_bytes);
        b->lucas.assign(n, LucasDev{});
    }
    b->d_order = (int *)(b->d_arena + job_bytes + lock_bytes + lucas_bytes);
    uint32_t *d_words = (uint32_t *)(b->d_arena + job_bytes + lock_bytes + lucas_bytes + order_bytes);
    if (cudaMemsetAsync(b->d_locks, 0, lock_bytes, e->stream) != cudaSuccess) {
        batch_free(b);
        return pfb::cuda_fail(cudaGetLastError(), "lock reset", __FILE__, __LINE__);
    }
    b->jobs.assign(n, JobDev{});
    size_t off = 0;
    int rc = PFB_OK;
    for (int i = 0; i < n && !rc; i++) {
        JobDev &j = b->jobs[i];
        memset(&j, 0, sizeof(j));
        const HostPrep &h = b->hp[i];
        if (!h.ok || h.decided >= 0) {
            j.phase = 3;
            j.verdict = h.ok ? h.decided : -1;
            continue;
        }
        uint32_t *w = d_words + off;
        const Layout &l = lay[i];
        j.x = w + l.x;
        j.res = w + l.res;
        j.nn = w + l.nn;
        j.nh = w + l.nh;
        j.npl = w + l.npl;
        j.nl = w + l.nl;
        j.exp = w + l.exp;
        if (!h.fpc && h.logl > LOG_LCTA) j.ybuf = w + l.yb;
        j.logl = h.logl;
        j.fpc = h.fpc;
        j.fbits = h.fbits;
        if (h.fpc && fp::spectrum_outside(h.fpc - 1)) j.sq = w + l.sq;
        j.cursor = h.cursor;
        j.extra = mode >= 1 ? h.s - 1 : 0;
        j.phase = 0;
        j.base = base;
        j.mode = mode;
        const size_t H = h.x0.size();
        cudaError_t ce = cudaMemcpyAsync(j.x, h.x0.data(), H * 4, cudaMemcpyHostToDevice, e->stream);
        if (mode == 2) {
            LucasDev &lc = b->lucas[i];
            lc.lv0 = w + l.lv0;
            lc.lv1 = w + l.lv1;
            lc.lqk = w + l.lqk;
            lc.lt = w + l.lt;
            lc.lone = w + l.lone;
            lc.gy = w + l.gy;
            lc.q = h.q;
            lc.lb = h.lb;
            j.lucas = b->d_lucas + i;
            // V_0 = 2, V_1 = P = 1, Q^0 = 1, and 1 itself, in Montgomery form (the
            // floating-point engine's set-up kernel makes them from x0)
            if (!h.fpc) {
                if (ce == cudaSuccess)
                    ce = cudaMemcpyAsync(lc.lv0, h.v0.data(), H * 4, cudaMemcpyHostToDevice, e->stream);
                if (ce == cudaSuccess)
                    ce = cudaMemcpyAsync(lc.lv1, h.x0.data(), H * 4, cudaMemcpyHostToDevice, e->stream);
                if (ce == cudaSuccess)
                    ce = cudaMemcpyAsync(lc.lqk, h.x0.data(), H * 4, cudaMemcpyHostToDevice, e->stream);
                if (ce == cudaSuccess)
                    ce = cudaMemcpyAsync(lc.lone, h.x0.data(), H * 4, cudaMemcpyHostToDevice, e->stream);
            }
        }
        if (ce == cudaSuccess) ce = cudaMemcpyAsync((void *)j.npl, h.npl.data(), H * 4, cudaMemcpyHostToDevice, e->stream);
        if (ce == cudaSuccess) ce = cudaMemcpyAsync((void *)j.nl, h.nl.data(), H * 4, cudaMemcpyHostToDevice, e->stream);
        if (ce == cudaSuccess)
            ce = cudaMemcpyAsync((void *)j.exp, h.exp.data(), h.exp.size() * 4, cudaMemcpyHostToDevice, e->stream);
        if (ce != cudaSuccess) rc = pfb::cuda_fail(ce, "batch upload", __FILE__, __LINE__);
        off += l.total;
    }
    cudaError_t ce = cudaSuccess;
    if (!rc) ce = cudaMemcpyAsync(b->d_jobs, b->jobs.data(), n * sizeof(JobDev), cudaMemcpyHostToDevice, e->stream);
    if (!rc && ce == cudaSuccess && mode == 2)
        ce = cudaMemcpyAsync(b->d_lucas, b->lucas.data(), n * sizeof(LucasDev), cudaMemcpyHostToDevice, e->stream);
    if (!rc && ce != cudaSuccess) rc = pfb::cuda_fail(ce, "job upload", __FILE__, __LINE__);
    if (!rc && !b->runs.order.empty()) {
        ce = cudaMemcpyAsync(b->d_order, b->runs.order.data(), b->runs.order.size() * sizeof(int),
                             cudaMemcpyHostToDevice, e->stream);
        for (int c = 0; c < fp::kClasses && ce == cudaSuccess; c++)
            if (b->runs.count[c])
                ce = fp::prep(e->fe, c, b->d_jobs, b->d_order + b->runs.first[c], b->runs.count[c], e->stream);
        if (ce != cudaSuccess) rc = pfb::cuda_fail(ce, "fft_prep_kernel", __FILE__, __LINE__);
    }
    if (!rc && b->runs.n_int) {
        ce = int_prep(b->d_jobs, nullptr, n, b->maxlog, e->tw, e->stream);
        if (ce != cudaSuccess) rc = pfb::cuda_fail(ce, "prep_kernel", __FILE__, __LINE__);
    }
    // host staging must outlive the copies; later work may use other streams
    if (!rc) {
        ce = cudaStreamSynchronize(e->stream);
        if (ce != cudaSuccess) rc = pfb::cuda_fail(ce, "batch sync", __FILE__, __LINE__);
    }
    if (rc) {
        batch_free(b);
        return rc;
    }
    *out = b;
    return PFB_OK;
}

// A batch on the floating-point engine, whose spectra take up to half as much
// memory again as the integer engine's; where the device cannot hold that,
// the whole batch on the integer engine.
int batch_build(pfb_mr *e, const pfb_mr_number_t *nums, int n, uint32_t base, int mode,
                const pfb_mr_number_t *exps, pfb_mr_batch **out) {
    const int rc = batch_build_on(e, nums, n, base, mode, exps, true, out);
    return rc == PFB_E_NOMEM ? batch_build_on(e, nums, n, base, mode, exps, false, out) : rc;
}

// Enqueues about `steps` steps of every unfinished candidate: launches of the
// persistent kernel, each handing out n * ceil(chunk / quantum) quanta.
int batch_advance(pfb_mr_batch *b, long long steps, cudaStream_t st) {
    if (!b->n_ok || steps <= 0) return PFB_OK;
    const long long cmax = b->e->chunk[b->maxlog];
    const int q0 = b->e->quantum[b->maxlog];
    while (steps > 0) {
        const long long chunk = std::min<long long>(steps, cmax);
        const int quantum = (int)std::min<long long>(chunk, q0);
        cudaGraphExec_t g = nullptr;
        const int rc = chunk_graph(b, chunk, quantum, &g);
        if (rc) return rc;
        PFB_CUDA(cudaGraphLaunch(g, st));
        steps -= chunk;
        b->steps_done += chunk;
    }
    return PFB_OK;
}

// Whether a launch depends on the quantum: not where every candidate has a CTA
// of its own (fp_quanta).
bool uses_quantum(const pfb_mr_batch *b) {
    bool used = b->runs.n_int > 0;
    for (int c = 0; c < fp::kClasses; c++) {
        const int n = b->runs.count[c];
        used = used || (n && n > (int)fp::persist_launch(b->e->fe, b->mode == 2, c, n, b->e->num_sms).grid.x);
    }
    return used;
}

int batch_pending(pfb_mr_batch *b, int *pending, long long *steps_total) {
    PFB_CUDA(cudaStreamSynchronize(b->e->stream));
    PFB_CUDA(cudaDeviceSynchronize());
    PFB_CUDA(cudaMemcpy(b->jobs.data(), b->d_jobs, b->n * sizeof(JobDev), cudaMemcpyDeviceToHost));
    int c = 0;
    long long st = 0;
    for (int i = 0; i < b->n; i++) {
        c += b->jobs[i].phase != 3;
        st += b->jobs[i].steps;
    }
    if (pending) *pending = c;
    if (steps_total) *steps_total = st;
    return PFB_OK;
}

int batch_results(pfb_mr_batch *b, int8_t *verdict, uint16_t *residue, int residue_stride) {
    pfb_mr *e = b->e;
    PFB_CUDA(cudaMemcpyAsync(b->jobs.data(), b->d_jobs, b->n * sizeof(JobDev), cudaMemcpyDeviceToHost, e->stream));
    PFB_CUDA(cudaStreamSynchronize(e->stream));
    std::vector<uint32_t> r22;
    int rc = PFB_OK;
    for (int i = 0; i < b->n; i++) {
        const JobDev &j = b->jobs[i];
        if (!b->hp[i].ok || b->hp[i].decided >= 0) {
            if (verdict) verdict[i] = (int8_t)(b->hp[i].ok ? b->hp[i].decided : -1);
            if (residue) memset(residue + (size_t)i * residue_stride, 0, sizeof(uint16_t) * residue_stride);
            continue;
        }
        if (j.phase != 3) {
            if (verdict) verdict[i] = -2;
            rc = PFB_E_STATE;
            continue;
        }
        if (verdict) verdict[i] = (int8_t)(b->mode >= 1 ? j.verdict : 0);
        if (residue && b->mode != 2) {
            const size_t H = b->hp[i].x0.size();
            r22.resize(H);
            PFB_CUDA(cudaMemcpy(r22.data(), j.res, H * 4, cudaMemcpyDeviceToHost));
            pfb::big::Words r = pfb::big::from_limbs(r22.data(), digit_bits(b->hp[i]), H);
            pfb::big::to_u16(r, residue + (size_t)i * residue_stride, (size_t)residue_stride);
        }
    }
    if (rc) pfb::set_error("pfb_mr: some candidates have not finished");
    return rc;
}

int run_jobs(pfb_mr *e, const pfb_mr_number_t *nums, int n, uint32_t base, int mode,
             const pfb_mr_number_t *exps, int8_t *verdict, uint16_t *residue, int residue_stride) {
    if (residue && residue_stride <= 0) {
        pfb::set_error("pfb_mr: residue_stride must be > 0");
        return PFB_E_ARG;
    }
    pfb_mr_batch *b = nullptr;
    int rc = batch_build(e, nums, n, base, mode, exps, &b);
    if (rc) return rc;
    rc = batch_advance(b, b->max_steps, e->stream);
    // The round-robin hands a locked candidate's quantum to another one, so a
    // few candidates may still need steps: continue until none is pending.
    // Every round advances each unfinished candidate, so a round count of
    // max_steps / 4096 + 64 is never reached unless the device stopped
    // making progress.
    const long long max_rounds = b->max_steps / 4096 + 64;
    for (long long round = 0; !rc; round++) {
        int pending = 0;
        rc = batch_pending(b, &pending, nullptr);
        if (rc || pending == 0) break;
        if (round >= max_rounds) {
            pfb::set_error("pfb_mr: %d candidates unfinished after %lld extra rounds", pending, round);
            rc = PFB_E_STATE;
            break;
        }
        rc = batch_advance(b, 4096, e->stream);
    }
    if (!rc) rc = batch_results(b, verdict, residue, residue_stride);
    cudaStreamSynchronize(e->stream);
    batch_free(b);
    return rc;
}

}  // namespace

extern "C" int pfb_mr_test(pfb_mr_t *e, const pfb_mr_number_t *nums, int n, uint32_t base, int8_t *verdict,
                           uint16_t *residue, int residue_stride) {
    return run_jobs(e, nums, n, base, 1, nullptr, verdict, residue, residue_stride);
}

extern "C" int pfb_mr_lucas(pfb_mr_t *e, const pfb_mr_number_t *nums, int n, int8_t *verdict) {
    if (!verdict) {
        pfb::set_error("pfb_mr_lucas: verdict is required");
        return PFB_E_ARG;
    }
    return run_jobs(e, nums, n, 2u, 2, nullptr, verdict, nullptr, 0);
}

extern "C" int pfb_mr_powm(pfb_mr_t *e, const pfb_mr_number_t *nums, int n, uint32_t base,
                           const pfb_mr_number_t *exps, uint16_t *residue, int residue_stride) {
    if (!exps || !residue) {
        pfb::set_error("pfb_mr_powm: exps and residue are required");
        return PFB_E_ARG;
    }
    return run_jobs(e, nums, n, base, 0, exps, nullptr, residue, residue_stride);
}

extern "C" int pfb_mr_batch_create(pfb_mr_t *e, const pfb_mr_number_t *nums, int n, uint32_t base,
                                   pfb_mr_batch_t **out) {
    if (!out) {
        pfb::set_error("pfb_mr_batch_create: null out");
        return PFB_E_ARG;
    }
    return batch_build(e, nums, n, base, 1, nullptr, out);
}

extern "C" int pfb_mr_batch_advance(pfb_mr_batch_t *b, int steps, void *stream) {
    if (!b || steps < 0) {
        pfb::set_error("pfb_mr_batch_advance: bad argument");
        return PFB_E_ARG;
    }
    PFB_CUDA(cudaSetDevice(b->e->device));
    return batch_advance(b, steps, stream ? (cudaStream_t)stream : b->e->stream);
}

extern "C" int pfb_mr_batch_pending(pfb_mr_batch_t *b, int *pending) {
    if (!b || !pending) {
        pfb::set_error("pfb_mr_batch_pending: bad argument");
        return PFB_E_ARG;
    }
    PFB_CUDA(cudaSetDevice(b->e->device));
    return batch_pending(b, pending, nullptr);
}

extern "C" long long pfb_mr_batch_steps_done(pfb_mr_batch_t *b) {
    if (!b) return -1;
    if (cudaSetDevice(b->e->device) != cudaSuccess) return -1;
    long long st = 0;
    if (batch_pending(b, nullptr, &st)) return -1;
    return st;
}

extern "C" long long pfb_mr_batch_steps_left(pfb_mr_batch_t *b) {
    if (!b) return -1;
    return std::max(0ll, b->max_steps - b->steps_done);
}

extern "C" int pfb_mr_batch_results(pfb_mr_batch_t *b, int8_t *verdict, uint16_t *residue, int residue_stride) {
    if (!b || (residue && residue_stride <= 0)) {
        pfb::set_error("pfb_mr_batch_results: bad argument");
        return PFB_E_ARG;
    }
    PFB_CUDA(cudaSetDevice(b->e->device));
    PFB_CUDA(cudaDeviceSynchronize());
    return batch_results(b, verdict, residue, residue_stride);
}

extern "C" void pfb_mr_batch_destroy(pfb_mr_batch_t *b) {
    if (!b) return;
    cudaSetDevice(b->e->device);
    cudaDeviceSynchronize();
    batch_free(b);
}

extern "C" int pfb_mr_autotune(pfb_mr_t *e, int logl_lo, int logl_hi, pfb_mr_tune_t *results, int cap,
                               int *n_results) {
    if (!e || logl_lo < LOG_LMIN || logl_hi > LOG_LSEQ || logl_lo > logl_hi || (cap > 0 && !results)) {
        pfb::set_error("pfb_mr_autotune: bad argument (transform lengths 2^%d .. 2^%d)", LOG_LMIN, LOG_LSEQ);
        return PFB_E_ARG;
    }
    if (n_results) *n_results = 0;
    PFB_CUDA(cudaSetDevice(e->device));
    // quanta above 64 steps leave SMs idle at the end of each launch once a
    // batch holds several candidates per SM, so the search stays below
    static const int kQuanta[] = {64, 32, 16};  // (of equal rates the first, the default, is kept)
    static const int kChunks[] = {2048, 1024};
    constexpr int NQ = 3, NC = 2, NP = NQ * NC;
    const long long kSteps = 2048;  // timed steps per tried pair and batch shape
    const int sms = std::max(1, e->num_sms);
    int rows = 0;
    uint64_t x = 0x9E3779B97F4A7C15ull;  // xorshift64: synthetic moduli
    cudaEvent_t ev[2];
    PFB_CUDA(cudaEventCreate(&ev[0]));
    PFB_CUDA(cudaEventCreate(&ev[1]));
    int rc = PFB_OK;
    for (int lg = logl_lo; lg <= logl_hi && !rc; lg++) {
        // the longest base-2 modulus of this length, R = 2^(22 L/2) >= 2^(bits + 6),
        // that the floating-point engine takes (all but the last 5 % of 2^15)
        const size_t fp_bits = (size_t)fp::limb_bits(fp::kClasses - 1) * 2 * fp::class_points(fp::kClasses - 1) - 6;
        const size_t bits = std::min((size_t)LIMB_BITS * ((size_t)1 << (lg - 1)) - 8, fp_bits);
        const int n16 = (int)((bits + 15) / 16);
        const int q_old = e->quantum[lg], c_old = e->chunk[lg];
        double rate[2][NP] = {};
        // two batch shapes: one and two candidates per SM (the tail of a launch
        // weighs more with one)
        for (int shape = 0; shape < 2 && !rc; shape++) {
            const int n = (shape + 1) * sms;
            std::vector<uint16_t> limbs((size_t)n * n16);
            std::vector<pfb_mr_number_t> nums(n);
            for (int i = 0; i < n; i++) {
                uint16_t *l = limbs.data() + (size_t)i * n16;
                for (int w = 0; w < n16; w++) {
                    x ^= x << 13;
                    x ^= x >> 7;
                    x ^= x << 17;
                    l[w] = (uint16_t)x;
                }
                const int top = (int)((bits - 1) % 16);
                l[n16 - 1] = (uint16_t)((l[n16 - 1] & ((1u << top) - 1u)) | (1u << top));
                l[0] |= 1u;
                nums[i] = pfb_mr_number_t{l, n16};
            }
            pfb_mr_batch *b = nullptr;
            rc = batch_build(e, nums.data(), n, 2u, 1, nullptr, &b);
            if (rc) break;
            rc = batch_advance(b, 64, e->stream);  // warm-up
            const bool quantum_used = uses_quantum(b);
            for (int k = 0; k < NP && !rc; k++) {
                if (k >= NC && !quantum_used) {  // the launches of the first quantum again
                    rate[shape][k] = rate[shape][k % NC];
                    continue;
                }
                e->quantum[lg] = kQuanta[k / NC];
                e->chunk[lg] = kChunks[k % NC];
                long long before = 0, after = 0;
                rc = batch_pending(b, nullptr, &before);
                if (!rc && cudaEventRecord(ev[0], e->stream) != cudaSuccess) rc = PFB_E_CUDA;
                if (!rc) rc = batch_advance(b, kSteps, e->stream);
                if (!rc && cudaEventRecord(ev[1], e->stream) != cudaSuccess) rc = PFB_E_CUDA;
                if (!rc) rc = batch_pending(b, nullptr, &after);
                float ms = 0.f;
                if (!rc && cudaEventElapsedTime(&ms, ev[0], ev[1]) != cudaSuccess) rc = PFB_E_CUDA;
                if (!rc) rate[shape][k] = ms > 0.f ? (double)(after - before) / (1e-3 * (double)ms) : 0.0;
            }
            batch_free(b);
        }
        e->quantum[lg] = q_old;
        e->chunk[lg] = c_old;
        if (rc) break;
        // score: the sum over shapes of the rate relative to the shape's best
        double best_rate[2] = {0.0, 0.0}, best = -1.0;
        for (int shape = 0; shape < 2; shape++)
            for (int k = 0; k < NP; k++) best_rate[shape] = std::max(best_rate[shape], rate[shape][k]);
        for (int k = 0; k < NP; k++) {
            double score = 0.0;
            for (int shape = 0; shape < 2; shape++)
                score += best_rate[shape] > 0.0 ? rate[shape][k] / best_rate[shape] : 0.0;
            if (results && rows < cap)
                results[rows] = pfb_mr_tune_t{lg, kQuanta[k / NC], kChunks[k % NC], rate[0][k], rate[1][k]};
            rows++;
            if (score > best) {
                best = score;
                e->quantum[lg] = kQuanta[k / NC];
                e->chunk[lg] = kChunks[k % NC];
            }
        }
    }
    cudaEventDestroy(ev[0]);
    cudaEventDestroy(ev[1]);
    if (n_results) *n_results = std::min(rows, cap);
    return rc;
}

extern "C" int pfb_mr_get_tuning(pfb_mr_t *e, int logl, int *quantum, int *chunk) {
    if (!e || logl < 0 || logl > LOG_LMAX) {
        pfb::set_error("pfb_mr_get_tuning: bad argument");
        return PFB_E_ARG;
    }
    if (quantum) *quantum = e->quantum[logl];
    if (chunk) *chunk = e->chunk[logl];
    return PFB_OK;
}

extern "C" long long pfb_mr_test_cost(const uint16_t *limbs, int n_limbs) {
    if (!limbs || n_limbs <= 0) return -1;
    pfb::big::Words N = pfb::big::from_u16(limbs, (size_t)n_limbs);
    const size_t nb = pfb::big::bit_length(N);
    if (nb < 2) return -1;
    return (long long)nb;  // ~ bits(d) squarings + one conversion
}

// ===========================================================================
// Serving: continuous batching on one GPU.
//
// Requests (candidates of any length) are prepared on host worker threads
// (N', R mod N, exponent) and admitted into free slots of a device-resident
// job table between launches of the persistent kernel, as slots and the HBM
// budget allow; every launch advances all resident candidates, whatever
// their lengths, round-robin by quanta; finished candidates are retired with
// their timestamps and their slot memory returns to a size-class pool.  All
// host waits are bounded (condition variables with timeouts); nothing on the
// device waits.

#include <chrono>
#include <condition_variable>
#include <deque>
#include <map>
#include <mutex>

namespace {

using Clock = std::chrono::steady_clock;

struct SrvRequest {
    uint64_t tag = 0;
    std::vector<uint16_t> limbs;
    uint16_t *residue_out = nullptr;
    int residue_cap = 0;
    double t_submit = 0.0, t_admit = 0.0;
    HostPrep hp;
};

struct SrvSlot {
    bool busy = false;
    int logl = 0;
    uint8_t *mem = nullptr;
    SrvRequest req;
};

}  // namespace

struct pfb_mr_server {
    pfb_mr *e = nullptr;
    pfb_mr_server_config_t cfg{};
    Clock::time_point t0;
    // device job table
    JobDev *d_jobs = nullptr;
    int *d_locks = nullptr;
    unsigned int *d_counter = nullptr;
    int *d_list = nullptr;
    uint8_t *d_table_mem = nullptr;
    std::vector<JobDev> jobs;
    ClassRuns runs;               // resident candidates by engine and class
    int *d_order = nullptr;       // runs.order
    bool runs_stale = true;
    cudaStream_t side[fp::kClasses] = {};  // classes run side by side
    cudaEvent_t fork = nullptr, join[fp::kClasses] = {};
    std::vector<SrvSlot> slots;
    std::map<int, std::vector<uint8_t *>> pool;  // free slot memory by transform length
    size_t bytes_in_use = 0, bytes_owned = 0;
    cudaStream_t stream = nullptr;
    // queues
    std::mutex mu;
    std::condition_variable cv_work, cv_done;
    std::deque<SrvRequest> submitted, prepared;
    std::deque<pfb_mr_result_t> done;
    bool stop = false;
    int preparing = 0;
    // statistics
    long long n_submitted = 0, n_admitted = 0, n_completed = 0, launches = 0;
    long long steps_total = 0;
    int resident = 0;
    std::vector<std::thread> workers;
    std::thread driver;
    int error = PFB_OK;
    // host-side fault injection (pfb_mr_server_inject_alloc_failures)
    int inject_alloc_failures = 0;
    int injected_alloc_failures = 0;
};

namespace {

double now_s(const pfb_mr_server *s) {
    return std::chrono::duration<double>(Clock::now() - s->t0).count();
}


// Slot memory; a failure injected from the host (a test hook) is reported as
// cudaErrorMemoryAllocation without calling cudaMalloc.
cudaError_t srv_alloc(pfb_mr_server *s, uint8_t **mem, size_t need) {
    {
        std::lock_guard<std::mutex> lk(s->mu);
        if (s->inject_alloc_failures > 0) {
            s->inject_alloc_failures--;
            s->injected_alloc_failures++;
            return cudaErrorMemoryAllocation;
        }
    }
    return cudaMalloc(mem, need);
}

void srv_prep_worker(pfb_mr_server *s) {
    for (;;) {
        SrvRequest r;
        {
            std::unique_lock<std::mutex> lk(s->mu);
            while (!s->stop && s->submitted.empty()) s->cv_work.wait_for(lk, std::chrono::milliseconds(100));
            if (s->stop) return;
            r = std::move(s->submitted.front());
            s->submitted.pop_front();
            s->preparing++;
        }
        pfb_mr_number_t num{r.limbs.data(), (int)r.limbs.size()};
        host_prep(num, s->cfg.base, 1, nullptr, r.hp, true);
        // a budget below one slot of the floating-point engine: the integer
        // engine's slots are smaller
        if (r.hp.ok && r.hp.fpc && s->cfg.hbm_budget_bytes && slot_bytes(slot_key(r.hp)) > s->cfg.hbm_budget_bytes)
            host_prep(num, s->cfg.base, 1, nullptr, r.hp, false);
        {
            std::lock_guard<std::mutex> lk(s->mu);
            s->preparing--;
            if (!r.hp.ok) {
                pfb_mr_result_t res{};
                res.tag = r.tag;
                res.verdict = -1;
                res.submit_s = r.t_submit;
                res.admit_s = res.done_s = now_s(s);
                s->done.push_back(res);
                s->n_completed++;
                s->cv_done.notify_all();
            } else {
                s->prepared.push_back(std::move(r));
            }
        }
        s->cv_work.notify_all();
    }
}

// Admits prepared requests into free slots; returns the slots admitted.
int srv_admit(pfb_mr_server *s, std::vector<int> &admitted) {
    admitted.clear();
    for (;;) {
        SrvRequest r;
        {
            std::lock_guard<std::mutex> lk(s->mu);
            if (s->prepared.empty()) break;
            int free_slot = -1;
            for (int i = 0; i < (int)s->slots.size(); i++)
                if (!s->slots[i].busy) {
                    free_slot = i;
                    break;
                }
            if (free_slot < 0) break;
            const int lg = slot_key(s->prepared.front().hp);
            const size_t need = slot_bytes(lg);
            const bool pooled = !s->pool[lg].empty();
            if (s->cfg.hbm_budget_bytes && !pooled && s->bytes_owned + need > s->cfg.hbm_budget_bytes) {
                // give back pooled blocks of other lengths first
                for (auto &kv : s->pool) {
                    while (!kv.second.empty() && s->bytes_owned + need > s->cfg.hbm_budget_bytes) {
                        const size_t blk = slot_bytes(kv.first);
                        cudaFree(kv.second.back());
                        kv.second.pop_back();
                        s->bytes_owned -= std::min(s->bytes_owned, blk);
                    }
                }
            }
            if (s->cfg.hbm_budget_bytes && !pooled && s->bytes_owned + need > s->cfg.hbm_budget_bytes) {
                if (s->resident == 0 && admitted.empty()) {
                    // a single request above the whole budget can never run
                    SrvRequest bad = std::move(s->prepared.front());
                    s->prepared.pop_front();
                    pfb_mr_result_t res{};
                    res.tag = bad.tag;
                    res.verdict = -1;
                    res.submit_s = bad.t_submit;
                    res.admit_s = res.done_s = now_s(s);
                    s->done.push_back(res);
                    s->n_completed++;
                    s->cv_done.notify_all();
                    continue;
                }
                break;  // wait for memory to come back
            }
            r = std::move(s->prepared.front());
            s->prepared.pop_front();
            SrvSlot &sl = s->slots[free_slot];
            sl.busy = true;
            sl.logl = lg;
            if (pooled) {
                sl.mem = s->pool[lg].back();
                s->pool[lg].pop_back();
            } else {
                sl.mem = nullptr;
            }
            s->bytes_in_use += need;
            admitted.push_back(free_slot);
            r.t_admit = now_s(s);
            sl.req = std::move(r);
        }
        SrvSlot &sl = s->slots[admitted.back()];
        if (!sl.mem) {
            const size_t need = slot_bytes(sl.logl);
            cudaError_t ce = srv_alloc(s, &sl.mem, need);
            if (ce != cudaSuccess) {
                // the device ran out below the budget (memory held elsewhere):
                // give back the pooled blocks and try once more
                cudaGetLastError();
                std::lock_guard<std::mutex> lk(s->mu);
                for (auto &kv : s->pool) {
                    const size_t blk = slot_bytes(kv.first);
                    for (uint8_t *m : kv.second) {
                        cudaFree(m);
                        s->bytes_owned -= std::min(s->bytes_owned, blk);
                    }
                    kv.second.clear();
                }
                sl.mem = nullptr;
            }
            if (ce != cudaSuccess) ce = srv_alloc(s, &sl.mem, need);
            if (ce != cudaSuccess) {
                // undo the admission: the request waits for resident candidates
                // to retire, or fails if none is resident
                cudaGetLastError();
                sl.mem = nullptr;
                admitted.pop_back();
                std::lock_guard<std::mutex> lk(s->mu);
                sl.busy = false;
                s->bytes_in_use -= need;
                if (s->resident == 0 && admitted.empty()) {
                    pfb_mr_result_t res{};
                    res.tag = sl.req.tag;
                    res.verdict = -1;
                    res.submit_s = sl.req.t_submit;
                    res.admit_s = res.done_s = now_s(s);
                    s->done.push_back(res);
                    s->n_completed++;
                    s->cv_done.notify_all();
                } else {
                    s->prepared.push_front(std::move(sl.req));
                }
                sl.req = SrvRequest();
                break;
            }
            std::lock_guard<std::mutex> lk(s->mu);
            s->bytes_owned += need;
        }
        // fill the job and upload its inputs
        const HostPrep &h = sl.req.hp;
        const Layout l = slot_layout(sl.logl);
        uint32_t *w = (uint32_t *)sl.mem;
        JobDev &j = s->jobs[admitted.back()];
        memset(&j, 0, sizeof(j));
        j.x = w + l.x;
        j.res = w + l.res;
        j.nn = w + l.nn;
        j.nh = w + l.nh;
        j.npl = w + l.npl;
        j.nl = w + l.nl;
        j.exp = w + l.exp;
        if (!h.fpc && h.logl > LOG_LCTA) j.ybuf = w + l.yb;
        j.logl = h.logl;
        j.fpc = h.fpc;
        j.fbits = h.fbits;
        if (h.fpc && fp::spectrum_outside(h.fpc - 1)) j.sq = w + l.sq;
        j.cursor = h.cursor;
        j.extra = h.s - 1;
        j.phase = 0;
        j.base = s->cfg.base;
        j.mode = 1;
        const size_t H = h.x0.size();
        PFB_CUDA(cudaMemcpyAsync(j.x, h.x0.data(), H * 4, cudaMemcpyHostToDevice, s->stream));
        PFB_CUDA(cudaMemcpyAsync((void *)j.npl, h.npl.data(), H * 4, cudaMemcpyHostToDevice, s->stream));
        PFB_CUDA(cudaMemcpyAsync((void *)j.nl, h.nl.data(), H * 4, cudaMemcpyHostToDevice, s->stream));
        PFB_CUDA(cudaMemcpyAsync((void *)j.exp, h.exp.data(), h.exp.size() * 4, cudaMemcpyHostToDevice, s->stream));
        PFB_CUDA(cudaMemcpyAsync(s->d_jobs + admitted.back(), &j, sizeof(JobDev), cudaMemcpyHostToDevice, s->stream));
        PFB_CUDA(cudaStreamSynchronize(s->stream));  // host staging is freed below / reused
    }
    if (!admitted.empty()) {
        // d_list: the integer engine's candidates, then each class'
        ClassRuns adm;
        adm.build((int)admitted.size(), [](int) { return true; },
                  [&](int i) { return s->slots[admitted[i]].req.hp.fpc; });
        std::vector<int> list;
        int maxlog = LOG_LMIN;
        for (int i : admitted)
            if (!s->slots[i].req.hp.fpc) {
                list.push_back(i);
                maxlog = std::max(maxlog, s->slots[i].logl);
            }
        for (int i : adm.order) list.push_back(admitted[i]);
        PFB_CUDA(cudaMemcpyAsync(s->d_list, list.data(), list.size() * sizeof(int), cudaMemcpyHostToDevice,
                                 s->stream));
        if (adm.n_int) {
            PFB_CUDA(int_prep(s->d_jobs, s->d_list, adm.n_int, maxlog, s->e->tw, s->stream));
        }
        for (int c = 0; c < fp::kClasses; c++)
            if (adm.count[c])
                PFB_CUDA(fp::prep(s->e->fe, c, s->d_jobs, s->d_list + adm.n_int + adm.first[c], adm.count[c],
                                  s->stream));
        PFB_CUDA(cudaStreamSynchronize(s->stream));
        s->runs_stale = true;
        for (int i : admitted) {  // the set-up inputs are on the device now
            HostPrep &h = s->slots[i].req.hp;
            std::vector<uint32_t>().swap(h.npl);
            std::vector<uint32_t>().swap(h.exp);
        }
        std::lock_guard<std::mutex> lk(s->mu);
        s->resident += (int)admitted.size();
        s->n_admitted += (long long)admitted.size();
    }
    return PFB_OK;
}

// Retires finished candidates (host mirror of the job table already read).
void srv_retire(pfb_mr_server *s) {
    std::vector<uint32_t> r22;
    for (int i = 0; i < (int)s->slots.size(); i++) {
        SrvSlot &sl = s->slots[i];
        if (!sl.busy || s->jobs[i].phase != 3) continue;
        pfb_mr_result_t res{};
        res.tag = sl.req.tag;
        res.verdict = (int8_t)s->jobs[i].verdict;
        res.submit_s = sl.req.t_submit;
        res.admit_s = sl.req.t_admit;
        if (sl.req.residue_out && sl.req.residue_cap > 0) {
            const size_t H = sl.req.hp.x0.size();
            r22.resize(H);
            if (cudaMemcpy(r22.data(), s->jobs[i].res, H * 4, cudaMemcpyDeviceToHost) == cudaSuccess) {
                pfb::big::Words r = pfb::big::from_limbs(r22.data(), digit_bits(sl.req.hp), H);
                pfb::big::to_u16(r, sl.req.residue_out, (size_t)sl.req.residue_cap);
            }
        }
        res.done_s = now_s(s);
        const size_t bytes = slot_bytes(sl.logl);
        std::lock_guard<std::mutex> lk(s->mu);
        s->pool[sl.logl].push_back(sl.mem);
        sl.mem = nullptr;
        sl.busy = false;
        s->runs_stale = true;
        s->bytes_in_use -= bytes;
        s->resident--;
        s->n_completed++;
        s->steps_total += s->jobs[i].steps;
        s->done.push_back(res);
        s->cv_done.notify_all();
    }
}

// Whether a class has a stream and an event of its own, made on first use;
// where they cannot be made, it runs on the server's stream after the others.
bool srv_side(pfb_mr_server *s, int c) {
    if (s->side[c]) return true;
    if (!s->join[c] && cudaEventCreateWithFlags(&s->join[c], cudaEventDisableTiming) != cudaSuccess) s->join[c] = nullptr;
    if (s->join[c] && cudaStreamCreateWithFlags(&s->side[c], cudaStreamNonBlocking) != cudaSuccess) s->side[c] = nullptr;
    if (!s->side[c]) cudaGetLastError();
    return s->side[c] != nullptr;
}

// Enqueues one launch of the persistent kernel per engine and length class
// with residents, side by side, and joins them on the server's stream.
int srv_launch(pfb_mr_server *s) {
    pfb_mr *e = s->e;
    const int cap = (int)s->slots.size();
    if (s->runs_stale) {
        s->runs.build(cap, [&](int i) { return s->slots[i].busy; }, [&](int i) { return s->jobs[i].fpc; });
        if (!s->runs.order.empty())
            PFB_CUDA(cudaMemcpyAsync(s->d_order, s->runs.order.data(), s->runs.order.size() * sizeof(int),
                                     cudaMemcpyHostToDevice, s->stream));
        s->runs_stale = false;
    }
    PFB_CUDA(cudaMemsetAsync(s->d_counter, 0, (1 + fp::kClasses) * sizeof(unsigned int), s->stream));
    const int quantum = std::min(64, s->cfg.chunk_steps);
    bool forked = false;
    if (s->runs.n_int) {
        const long long qpj = (s->cfg.chunk_steps + quantum - 1) / quantum;
        int maxlog = LOG_LMIN;
        for (auto &sl : s->slots)
            if (sl.busy && sl.logl < kFpKey) maxlog = std::max(maxlog, sl.logl);
        if (!s->runs.order.empty()) {
            PFB_CUDA(cudaEventRecord(s->fork, s->stream));
            forked = true;
        }
        int n = cap, q = quantum;
        unsigned int *counter = s->d_counter, total = (unsigned int)(s->runs.n_int * qpj);
        Twiddles tw = e->tw;
        void *args[] = {&s->d_jobs, &n, &s->d_locks, &counter, &total, &q, &tw};
        PFB_CUDA(cudaLaunchKernel(int_persist_func(), dim3(std::min(s->runs.n_int, std::max(1, e->num_sms))),
                                  dim3(THREADS), args, smem_bytes(maxlog), s->stream));
    }
    int classes = 0;
    for (int c = 0; c < fp::kClasses; c++) classes += s->runs.count[c] > 0;
    if (classes > 1 && !forked) {
        PFB_CUDA(cudaEventRecord(s->fork, s->stream));
        forked = true;
    }
    for (int c = fp::kClasses - 1; c >= 0; c--) {
        int nc = s->runs.count[c], qc = 0;
        if (!nc) continue;
        cudaStream_t st = s->stream;
        if (forked && srv_side(s, c)) {
            st = s->side[c];
            PFB_CUDA(cudaStreamWaitEvent(st, s->fork, 0));
        }
        unsigned tc = 0;
        fp_quanta(e, false, c, nc, s->cfg.chunk_steps, quantum, &qc, &tc);
        const fp::Launch l = fp::persist_launch(e->fe, false, c, nc, e->num_sms);
        const int *order = s->d_order + s->runs.first[c];
        unsigned int *cnt = s->d_counter + 1 + c;
        fp::Tab tab = e->fe.tab[c];
        void *fa[] = {&s->d_jobs, &order, &nc, &s->d_locks, &cnt, &tc, &qc, &tab};
        PFB_CUDA(cudaLaunchKernel(l.func, l.grid, l.block, fa, l.smem, st));
    }
    if (forked)
        for (int c = 0; c < fp::kClasses; c++)
            if (s->runs.count[c] && s->side[c]) {
                PFB_CUDA(cudaEventRecord(s->join[c], s->side[c]));
                PFB_CUDA(cudaStreamWaitEvent(s->stream, s->join[c], 0));
            }
    return PFB_OK;
}

void srv_driver(pfb_mr_server *s) {
    if (cudaSetDevice(s->e->device) != cudaSuccess) {
        s->error = PFB_E_CUDA;
        return;
    }
    std::vector<int> admitted;
    const int cap = (int)s->slots.size();
    while (true) {
        {
            std::unique_lock<std::mutex> lk(s->mu);
            while (!s->stop && s->resident == 0 && s->prepared.empty())
                s->cv_work.wait_for(lk, std::chrono::milliseconds(50));
            if (s->stop) break;
        }
        int rc = srv_admit(s, admitted);
        if (rc) {
            s->error = rc;
            break;
        }
        int res_now;
        {
            std::lock_guard<std::mutex> lk(s->mu);
            res_now = s->resident;
        }
        if (res_now == 0) continue;
        // one launch per engine and class: every resident candidate advances
        // about chunk_steps steps
        if (srv_launch(s) != PFB_OK ||
            cudaMemcpyAsync(s->jobs.data(), s->d_jobs, cap * sizeof(JobDev), cudaMemcpyDeviceToHost, s->stream) !=
                cudaSuccess ||
            cudaStreamSynchronize(s->stream) != cudaSuccess) {
            pfb::set_error("pfb_mr_server: CUDA failure in the step loop");
            s->error = PFB_E_CUDA;
            break;
        }
        s->launches++;
        srv_retire(s);
    }
    std::lock_guard<std::mutex> lk(s->mu);
    s->stop = true;
    s->cv_done.notify_all();
    s->cv_work.notify_all();
}

}  // namespace

extern "C" int pfb_mr_server_create(pfb_mr_t *e, const pfb_mr_server_config_t *cfg, pfb_mr_server_t **out) {
    if (!e || !out) {
        pfb::set_error("pfb_mr_server_create: null argument");
        return PFB_E_ARG;
    }
    *out = nullptr;
    pfb_mr_server *s = new pfb_mr_server();
    s->e = e;
    if (cfg) s->cfg = *cfg;
    if (s->cfg.max_resident <= 0) s->cfg.max_resident = 2 * std::max(1, e->num_sms);
    if (s->cfg.chunk_steps <= 0) s->cfg.chunk_steps = 512;
    if (s->cfg.base < 2 || s->cfg.base > 0xFFFFu) s->cfg.base = 2;
    if (s->cfg.prep_threads <= 0) s->cfg.prep_threads = 4;
    s->t0 = Clock::now();
    const int cap = s->cfg.max_resident;
    PFB_CUDA(cudaSetDevice(e->device));
    const size_t job_bytes = ((size_t)cap * sizeof(JobDev) + 255) & ~(size_t)255;
    const size_t int_bytes = ((size_t)cap * sizeof(int) + 255) & ~(size_t)255;
    if (cudaMalloc(&s->d_table_mem, job_bytes + 3 * int_bytes + 256) != cudaSuccess) {
        cudaGetLastError();
        delete s;
        pfb::set_error("pfb_mr_server_create: cannot allocate the job table");
        return PFB_E_NOMEM;
    }
    s->d_jobs = (JobDev *)s->d_table_mem;
    s->d_locks = (int *)(s->d_table_mem + job_bytes);
    s->d_list = (int *)(s->d_table_mem + job_bytes + int_bytes);
    s->d_order = (int *)(s->d_table_mem + job_bytes + 2 * int_bytes);
    s->d_counter = (unsigned int *)(s->d_table_mem + job_bytes + 3 * int_bytes);
    s->jobs.assign(cap, JobDev{});
    for (auto &j : s->jobs) j.phase = 3;
    s->slots.resize(cap);
    int rc = PFB_OK;
    cudaError_t ce = cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking);
    if (ce == cudaSuccess) ce = cudaEventCreateWithFlags(&s->fork, cudaEventDisableTiming);
    if (ce == cudaSuccess) ce = cudaMemcpy(s->d_jobs, s->jobs.data(), cap * sizeof(JobDev), cudaMemcpyHostToDevice);
    if (ce == cudaSuccess) ce = cudaMemset(s->d_locks, 0, int_bytes);
    if (ce != cudaSuccess) rc = pfb::cuda_fail(ce, "server set-up", __FILE__, __LINE__);
    if (rc) {
        cudaFree(s->d_table_mem);
        if (s->fork) cudaEventDestroy(s->fork);
        if (s->stream) cudaStreamDestroy(s->stream);
        delete s;
        return rc;
    }
    for (int t = 0; t < s->cfg.prep_threads; t++) s->workers.emplace_back(srv_prep_worker, s);
    s->driver = std::thread(srv_driver, s);
    *out = s;
    return PFB_OK;
}

extern "C" int pfb_mr_server_submit(pfb_mr_server_t *s, const uint16_t *limbs, int n_limbs, uint64_t tag,
                                    uint16_t *residue_out, int residue_cap) {
    if (!s || !limbs || n_limbs <= 0 || (residue_out && residue_cap <= 0)) {
        pfb::set_error("pfb_mr_server_submit: bad argument");
        return PFB_E_ARG;
    }
    SrvRequest r;
    r.tag = tag;
    r.limbs.assign(limbs, limbs + n_limbs);
    r.residue_out = residue_out;
    r.residue_cap = residue_cap;
    {
        std::lock_guard<std::mutex> lk(s->mu);
        if (s->stop) {
            pfb::set_error("pfb_mr_server_submit: server stopped (%d)", s->error);
            return PFB_E_STATE;
        }
        r.t_submit = now_s(s);
        s->submitted.push_back(std::move(r));
        s->n_submitted++;
    }
    s->cv_work.notify_all();
    return PFB_OK;
}

extern "C" int pfb_mr_server_poll(pfb_mr_server_t *s, pfb_mr_result_t *out, int cap, int timeout_ms) {
    if (!s || !out || cap <= 0) {
        pfb::set_error("pfb_mr_server_poll: bad argument");
        return PFB_E_ARG;
    }
    std::unique_lock<std::mutex> lk(s->mu);
    if (s->done.empty() && timeout_ms > 0 && !s->stop)
        s->cv_done.wait_for(lk, std::chrono::milliseconds(timeout_ms), [&] { return !s->done.empty() || s->stop; });
    int n = 0;
    while (n < cap && !s->done.empty()) {
        out[n++] = s->done.front();
        s->done.pop_front();
    }
    if (n == 0 && s->stop && s->error) return s->error;
    return n;
}

extern "C" int pfb_mr_server_inject_alloc_failures(pfb_mr_server_t *s, int n) {
    if (!s || n < 0) {
        pfb::set_error("pfb_mr_server_inject_alloc_failures: bad argument");
        return PFB_E_ARG;
    }
    std::lock_guard<std::mutex> lk(s->mu);
    s->inject_alloc_failures += n;
    return s->injected_alloc_failures;
}

extern "C" int pfb_mr_server_stats(pfb_mr_server_t *s, pfb_mr_server_stats_t *st) {
    if (!s || !st) {
        pfb::set_error("pfb_mr_server_stats: bad argument");
        return PFB_E_ARG;
    }
    std::lock_guard<std::mutex> lk(s->mu);
    st->submitted = s->n_submitted;
    st->admitted = s->n_admitted;
    st->completed = s->n_completed;
    st->resident = s->resident;
    st->queued = (int)(s->submitted.size() + s->prepared.size()) + s->preparing;
    st->launches = s->launches;
    st->steps_retired = s->steps_total;
    st->bytes_in_use = s->bytes_in_use;
    st->bytes_owned = s->bytes_owned;
    st->error = s->error;
    return PFB_OK;
}

extern "C" void pfb_mr_server_destroy(pfb_mr_server_t *s) {
    if (!s) return;
    {
        std::lock_guard<std::mutex> lk(s->mu);
        s->stop = true;
    }
    s->cv_work.notify_all();
    s->cv_done.notify_all();
    if (s->driver.joinable()) s->driver.join();
    for (auto &t : s->workers)
        if (t.joinable()) t.join();
    cudaSetDevice(s->e->device);
    cudaStreamSynchronize(s->stream);
    for (auto &sl : s->slots)
        if (sl.mem) cudaFree(sl.mem);
    for (auto &kv : s->pool)
        for (uint8_t *m : kv.second) cudaFree(m);
    cudaEventDestroy(s->fork);
    for (int c = 0; c < fp::kClasses; c++) {
        if (s->side[c]) cudaStreamDestroy(s->side[c]);
        if (s->join[c]) cudaEventDestroy(s->join[c]);
    }
    cudaFree(s->d_table_mem);
    cudaStreamDestroy(s->stream);
    delete s;
}

// ---------------------------------------------------------------------------
// Per-operation modular context (BatchModCtx's methods).

struct pfb_mr_ctx {
    pfb_mr *e = nullptr;
    int n = 0, n16 = 0, maxlog = LOG_LMIN;
    uint8_t *d_arena = nullptr;
    JobDev *d_jobs = nullptr;
    CtxExtra *d_ex = nullptr;
    uint64_t *d_one = nullptr, *d_nm1 = nullptr, *d_tmp = nullptr, *d_n = nullptr;  // [n][n16] each
    // moduli of the floating-point engine (transform lengths up to 2^LOG_LCTA)
    // by class; the others, and all raw products, on the integer engine
    ClassRuns runs;
    int *d_order = nullptr;
    std::vector<HostPrep> hp;
};

namespace {

int ctx_fail(pfb_mr_ctx *c, int rc) {
    if (c) {
        cudaFree(c->d_arena);
        delete c;
    }
    return rc;
}

std::vector<uint64_t> widen16(const pfb::big::Words &w, size_t n16) {
    std::vector<uint16_t> t(n16);
    pfb::big::to_u16(w, t.data(), n16);
    return std::vector<uint64_t>(t.begin(), t.end());
}

int ctx_launch(pfb_mr_ctx *c, const uint64_t *a, const uint64_t *b, uint64_t *out, int out_stride, int op,
               void *stream) {
    if (!c || !a || !out || ((op == CTX_MODMUL || op == CTX_RAW_MUL) && !b)) {
        pfb::set_error("pfb_mr_ctx: bad argument");
        return PFB_E_ARG;
    }
    PFB_CUDA(cudaSetDevice(c->e->device));
    // NULL: the legacy default stream, ordered with the caller's other
    // default-stream work (the reference's methods run there)
    cudaStream_t st = stream ? (cudaStream_t)stream : cudaStreamLegacy;
    if (op != CTX_RAW_SQ && op != CTX_RAW_MUL) {
        for (int k = 0; k < fp::kClasses; k++)
            if (c->runs.count[k])
                PFB_CUDA(fp::ctx(c->e->fe, k, c->d_jobs, c->d_order + c->runs.first[k], c->runs.count[k], a,
                                 b ? b : a, out, c->n16, op, c->d_ex, st));
        if (!c->runs.n_int) return PFB_OK;
    }
    PFB_CUDA(int_ctx(c->d_jobs, c->d_ex, c->n, c->maxlog, a, b ? b : a, out, c->n16, out_stride, op, c->e->tw, st));
    return PFB_OK;
}

}  // namespace

static int ctx_create_on(pfb_mr_t *e, const uint64_t *N_all, int n_limbs, int n_batch, bool fft,
                         pfb_mr_ctx_t **out) {
    PFB_CUDA(cudaSetDevice(e->device));
    pfb_mr_ctx *c = new pfb_mr_ctx();
    c->e = e;
    c->n = n_batch;
    c->n16 = n_limbs;
    std::vector<uint16_t> n16((size_t)n_limbs * n_batch);
    for (size_t i = 0; i < n16.size(); i++) {
        if (N_all[i] > 0xFFFFu) {
            pfb::set_error("pfb_mr_ctx_create: limb %zu is not a 16-bit value", i);
            return ctx_fail(c, PFB_E_ARG);
        }
        n16[i] = (uint16_t)N_all[i];
    }
    std::vector<pfb_mr_number_t> nums(n_batch);
    for (int i = 0; i < n_batch; i++) nums[i] = pfb_mr_number_t{n16.data() + (size_t)i * n_limbs, n_limbs};
    // base 2 sizes R > 64 N: products of two reduced operands stay below 2N after REDC
    prep_all(nums.data(), n_batch, 2u, 1, nullptr, c->hp, false);
    std::vector<Layout> lay(n_batch);
    size_t words = 0;
    for (int i = 0; i < n_batch; i++) {
        if (!c->hp[i].ok) {
            pfb::set_error("pfb_mr_ctx_create: modulus %d is not odd, > 1 and at most %d bits", i, PFB_MR_MAX_BITS);
            return ctx_fail(c, PFB_E_ARG);
        }
        HostPrep &h = c->hp[i];
        for (int k = 0; k < fp::kClasses && fft && h.logl <= LOG_LCTA; k++)
            if (fp::class_points(k) == 1 << (h.logl - 1)) h.fpc = k + 1;
        lay[i] = h.fpc ? layout_fp(h.fpc - 1, 0, false, h.logl)
                       : layout_for(h.logl, 1, true, true);  // gy [2][L], spare H-word buffers, raw coefficients
        words += lay[i].total;
        c->maxlog = std::max(c->maxlog, c->hp[i].logl);
    }
    const size_t job_bytes = ((size_t)n_batch * sizeof(JobDev) + 255) & ~(size_t)255;
    const size_t ex_bytes = ((size_t)n_batch * sizeof(CtxExtra) + 255) & ~(size_t)255;
    const size_t v_bytes = (((size_t)n_batch * n_limbs * sizeof(uint64_t)) + 255) & ~(size_t)255;
    c->runs.build(n_batch, [](int) { return true; }, [&](int i) { return c->hp[i].fpc; });
    const size_t order_bytes = ((size_t)n_batch * sizeof(int) + 255) & ~(size_t)255;
    const size_t need = job_bytes + ex_bytes + 4 * v_bytes + order_bytes + words * sizeof(uint32_t);
    if (cudaMalloc(&c->d_arena, need) != cudaSuccess) {
        cudaGetLastError();
        pfb::set_error("pfb_mr_ctx_create: cannot allocate %zu bytes of device memory", need);
        return ctx_fail(c, PFB_E_NOMEM);
    }
    c->d_jobs = (JobDev *)c->d_arena;
    c->d_ex = (CtxExtra *)(c->d_arena + job_bytes);
    c->d_one = (uint64_t *)(c->d_arena + job_bytes + ex_bytes);
    c->d_nm1 = (uint64_t *)(c->d_arena + job_bytes + ex_bytes + v_bytes);
    c->d_tmp = (uint64_t *)(c->d_arena + job_bytes + ex_bytes + 2 * v_bytes);
    c->d_n = (uint64_t *)(c->d_arena + job_bytes + ex_bytes + 3 * v_bytes);
    c->d_order = (int *)(c->d_arena + job_bytes + ex_bytes + 4 * v_bytes);
    uint32_t *d_words = (uint32_t *)(c->d_arena + job_bytes + ex_bytes + 4 * v_bytes + order_bytes);
    std::vector<JobDev> jobs(n_batch);
    std::vector<CtxExtra> ex(n_batch);
    std::vector<uint64_t> one((size_t)n_batch * n_limbs), nm1((size_t)n_batch * n_limbs);
    size_t off = 0;
    for (int i = 0; i < n_batch; i++) {
        const HostPrep &h = c->hp[i];
        const Layout &l = lay[i];
        uint32_t *w = d_words + off;
        JobDev &j = jobs[i];
        memset(&j, 0, sizeof(j));
        j.nn = w + l.nn;
        j.nh = w + l.nh;
        j.npl = w + l.npl;
        j.nl = w + l.nl;
        if (!h.fpc) {
            j.x = w + l.x;
            j.res = w + l.res;
            if (h.logl > LOG_LCTA) j.ybuf = w + l.yb;
        }
        j.logl = h.logl;
        j.fpc = h.fpc;
        j.fbits = h.fpc ? LIMB_BITS / 2 : 0;
        j.phase = 0;
        ex[i].gy = w + l.gy;
        ex[i].yl = w + l.lt;
        ex[i].raw = (unsigned long long *)(w + l.raw);
        if (h.fpc) {
            ex[i].ys = w + l.gy;
            if (fp::spectrum_outside(h.fpc - 1)) j.sq = w + l.sq;
        }
        const size_t H = h.nl.size();
        std::vector<uint32_t> npl = h.npl, nl = h.nl;
        if (h.fpc) {  // two digits of 11 bits per limb: the radix R' is the same
            auto split = [](const std::vector<uint32_t> &v) {
                std::vector<uint32_t> d;
                for (uint32_t x : v) {
                    d.push_back(x & ((1u << LIMB_BITS / 2) - 1u));
                    d.push_back(x >> LIMB_BITS / 2);
                }
                return d;
            };
            npl = split(h.npl);
            nl = split(h.nl);
        }
        PFB_CUDA(cudaMemcpy((void *)j.npl, npl.data(), npl.size() * 4, cudaMemcpyHostToDevice));
        PFB_CUDA(cudaMemcpy((void *)j.nl, nl.data(), nl.size() * 4, cudaMemcpyHostToDevice));
        // working forms of 1 and N - 1: R mod N and N - (R mod N)
        const pfb::big::Words N = pfb::big::from_u16(nums[i].limbs, (size_t)n_limbs);
        const pfb::big::Words r = pfb::big::from_limbs(h.x0.data(), LIMB_BITS, H);
        const std::vector<uint64_t> o = widen16(r, (size_t)n_limbs), m = widen16(pfb::big::sub(N, r), (size_t)n_limbs);
        std::copy(o.begin(), o.end(), one.begin() + (size_t)i * n_limbs);
        std::copy(m.begin(), m.end(), nm1.begin() + (size_t)i * n_limbs);
        off += l.total;
    }
    PFB_CUDA(cudaMemcpy(c->d_jobs, jobs.data(), n_batch * sizeof(JobDev), cudaMemcpyHostToDevice));
    PFB_CUDA(cudaMemcpy(c->d_ex, ex.data(), n_batch * sizeof(CtxExtra), cudaMemcpyHostToDevice));
    PFB_CUDA(cudaMemcpy(c->d_one, one.data(), one.size() * 8, cudaMemcpyHostToDevice));
    PFB_CUDA(cudaMemcpy(c->d_nm1, nm1.data(), nm1.size() * 8, cudaMemcpyHostToDevice));
    const std::vector<uint64_t> nall(n16.begin(), n16.end());
    PFB_CUDA(cudaMemcpy(c->d_n, nall.data(), nall.size() * 8, cudaMemcpyHostToDevice));
    cudaError_t ce = cudaSuccess;
    if (!c->runs.order.empty())
        ce = cudaMemcpyAsync(c->d_order, c->runs.order.data(), c->runs.order.size() * sizeof(int),
                             cudaMemcpyHostToDevice, e->stream);
    for (int k = 0; k < fp::kClasses && ce == cudaSuccess; k++)
        if (c->runs.count[k])
            ce = fp::prep(e->fe, k, c->d_jobs, c->d_order + c->runs.first[k], c->runs.count[k], e->stream);
    if (ce == cudaSuccess && c->runs.n_int) ce = int_prep(c->d_jobs, nullptr, n_batch, c->maxlog, e->tw, e->stream);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(e->stream);
    if (ce != cudaSuccess) return ctx_fail(c, pfb::cuda_fail(ce, "pfb_mr_ctx_create", __FILE__, __LINE__));
    *out = c;
    return PFB_OK;
}

// As a batch: on the integer engine where the device cannot hold the
// floating-point engine's buffers (at most 22 words a point, against 21).
extern "C" int pfb_mr_ctx_create(pfb_mr_t *e, const uint64_t *N_all, int n_limbs, int n_batch, pfb_mr_ctx_t **out) {
    if (!out || !e || !N_all || n_limbs <= 0 || n_batch <= 0) {
        pfb::set_error("pfb_mr_ctx_create: bad argument");
        return PFB_E_ARG;
    }
    *out = nullptr;
    const int rc = ctx_create_on(e, N_all, n_limbs, n_batch, true, out);
    return rc == PFB_E_NOMEM ? ctx_create_on(e, N_all, n_limbs, n_batch, false, out) : rc;
}

extern "C" void pfb_mr_ctx_destroy(pfb_mr_ctx_t *c) {
    if (!c) return;
    cudaSetDevice(c->e->device);
    cudaDeviceSynchronize();
    ctx_fail(c, PFB_OK);
}

extern "C" int pfb_mr_ctx_n_sum(const pfb_mr_ctx_t *c) { return c ? 2 * c->n16 + 16 : -1; }

extern "C" int pfb_mr_ctx_buffers(const pfb_mr_ctx_t *c, const uint64_t **d_N, const uint64_t **d_one,
                                  const uint64_t **d_nm1) {
    if (!c) {
        pfb::set_error("pfb_mr_ctx_buffers: null context");
        return PFB_E_ARG;
    }
    if (d_N) *d_N = c->d_n;
    if (d_one) *d_one = c->d_one;
    if (d_nm1) *d_nm1 = c->d_nm1;
    return PFB_OK;
}

extern "C" int pfb_mr_ctx_to_residue(pfb_mr_ctx_t *c, const uint64_t *x_all, uint64_t *out_all) {
    if (!c || !x_all || !out_all) {
        pfb::set_error("pfb_mr_ctx_to_residue: bad argument");
        return PFB_E_ARG;
    }
    using namespace pfb::big;
    std::vector<uint16_t> t(c->n16);
    for (int i = 0; i < c->n; i++) {
        const size_t o = (size_t)i * c->n16;
        for (int k = 0; k < c->n16; k++) t[k] = (uint16_t)x_all[o + k];
        const Words x = from_u16(t.data(), (size_t)c->n16);
        const HostPrep &h = c->hp[i];
        const Words N = from_limbs(h.nl.data(), LIMB_BITS, h.nl.size());
        Words rem;
        divmod(add(shl(x, (size_t)LIMB_BITS * h.nl.size()), x), N, nullptr, &rem);  // x R' mod N, R' = 2^(22 H) + 1
        const std::vector<uint64_t> r = widen16(rem, (size_t)c->n16);
        std::copy(r.begin(), r.end(), out_all + o);
    }
    return PFB_OK;
}

extern "C" int pfb_mr_ctx_from_residue(pfb_mr_ctx_t *c, const uint64_t *d_x, uint64_t *out_all) {
    if (!out_all) {
        pfb::set_error("pfb_mr_ctx_from_residue: bad argument");
        return PFB_E_ARG;
    }
    const int rc = ctx_launch(c, d_x, nullptr, c ? c->d_tmp : nullptr, c ? c->n16 : 0, CTX_FROM, nullptr);
    if (rc) return rc;
    PFB_CUDA(cudaMemcpy(out_all, c->d_tmp, (size_t)c->n * c->n16 * 8, cudaMemcpyDeviceToHost));
    return PFB_OK;
}

extern "C" int pfb_mr_ctx_check_passed(pfb_mr_ctx_t *c, const uint64_t *d_r, uint8_t *d_passed, void *stream) {
    if (!c || !d_r || !d_passed) {
        pfb::set_error("pfb_mr_ctx_check_passed: bad argument");
        return PFB_E_ARG;
    }
    PFB_CUDA(cudaSetDevice(c->e->device));
    cudaStream_t st = stream ? (cudaStream_t)stream : cudaStreamLegacy;
    PFB_CUDA(int_ctx_check(d_r, c->d_one, c->d_nm1, d_passed, c->n, c->n16, st));
    return PFB_OK;
}

extern "C" int pfb_mr_ctx_modsq(pfb_mr_ctx_t *c, const uint64_t *d_a, uint64_t *d_out, void *stream) {
    return ctx_launch(c, d_a, nullptr, d_out, c ? c->n16 : 0, CTX_MODSQ, stream);
}

extern "C" int pfb_mr_ctx_modmul(pfb_mr_ctx_t *c, const uint64_t *d_a, const uint64_t *d_b, uint64_t *d_out,
                                 void *stream) {
    return ctx_launch(c, d_a, d_b, d_out, c ? c->n16 : 0, CTX_MODMUL, stream);
}

extern "C" int pfb_mr_ctx_sq_raw(pfb_mr_ctx_t *c, const uint64_t *d_a, uint64_t *d_out, void *stream) {
    return ctx_launch(c, d_a, nullptr, d_out, c ? 2 * c->n16 + 16 : 0, CTX_RAW_SQ, stream);
}

extern "C" int pfb_mr_ctx_mul_raw(pfb_mr_ctx_t *c, const uint64_t *d_a, const uint64_t *d_b, uint64_t *d_out,
                                  void *stream) {
    return ctx_launch(c, d_a, d_b, d_out, c ? 2 * c->n16 + 16 : 0, CTX_RAW_MUL, stream);
}
