// Runs the Miller-Rabin engine's host code (mr.cu) unchanged on the CPU
// against a stand-in CUDA runtime (tests/cpp/emul/cuda_runtime_api_fake.h)
// whose kernels only mark their candidates as finished, to see what the host
// does when device memory runs out.  Input lines:
//
//   server allow bits   one request of a random number of that many bits, with
//                       `allow` device allocations granted after the server's
//                       creation (-1: all) -> "verdict v" or "stopped rc",
//                       then the engine that ran it (fft, int, none)
//   mixed streams       a server with two requests of different length classes, that
//                       can (1) or cannot (0) create further streams -> as server
//   batch bytes bits n  strong tests of n numbers on a device of that many bytes
//                       beyond what the engine holds (-1: no limit) -> "rc c",
//                       device memory of the batch and the engine that ran it
//   ctx bytes bits n    a context of n moduli on a device of that many bytes beyond
//                       what the engine holds (-1: no limit) -> "rc c", its device
//                       memory in bytes and the engine that it was set up for
//   tune lg             autotune of one transform length -> "rc c", launches of the
//                       persistent kernel and the pair kept
#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <deque>
#include <iostream>
#include <random>
#include <sstream>
#include <string>
#include <thread>

#include <cuda_runtime.h>
#include <cuda_runtime_api_fake.h>

#include "mr.cu"

namespace pfb {
void set_error(const char *, ...) {}
int cuda_fail(cudaError_t, const char *, const char *, int) { return PFB_E_CUDA; }
}  // namespace pfb

static int n_fft, n_int;        // candidates that each engine has finished
static int prep_fft, prep_int;  // and that each has set up
static int launches;
static std::atomic<bool> held;  // the FFT kernels finish nothing while set
static int fn_fft, fn_int;

namespace pfb {
namespace mr {

int int_setup(const CrtConsts &, const WideTabs &) { return PFB_OK; }
void *int_persist_func() { return &fn_int; }
cudaError_t int_prep(JobDev *, const int *, int n, int, const Twiddles &, cudaStream_t) {
    prep_int += n;
    return cudaSuccess;
}
cudaError_t int_ctx(const JobDev *, const CtxExtra *, int, int, const uint64_t *, const uint64_t *, uint64_t *, int,
                    int, int, const Twiddles &, cudaStream_t) { return cudaSuccess; }
cudaError_t int_ctx_check(const uint64_t *, const uint64_t *, const uint64_t *, uint8_t *, int, int, cudaStream_t) {
    return cudaSuccess;
}

namespace fp {

int engine_create(Engine &e) {
    e = Engine{};
    return PFB_OK;
}
void engine_free(Engine &) {}
Launch persist_launch(const Engine &, bool, int, int n, int sms) {
    return Launch{&fn_fft, dim3((unsigned)std::min(n, sms)), dim3(32), 0};
}
cudaError_t ctx(const Engine &, int, const JobDev *, const int *, int, const uint64_t *, const uint64_t *, uint64_t *,
                int, int, const CtxExtra *, cudaStream_t) { return cudaSuccess; }
cudaError_t prep(const Engine &, int, JobDev *, const int *, int n, cudaStream_t) {
    prep_fft += n;
    return cudaSuccess;
}

}  // namespace fp
}  // namespace mr
}  // namespace pfb

static void finish(JobDev &j, int &count) {
    if (j.phase == 3) return;
    memset(j.res, 0, 4);  // (the kernels write it: it has to be there)
    j.phase = 3;
    j.verdict = 0;
    count++;
}

static std::function<void()> launch(void *func, void **a) {
    JobDev *jobs = *(JobDev **)a[0];
    if (func == &fn_int) {
        const int n = *(int *)a[1];
        return [=] {
            launches++;
            for (int i = 0; i < n; i++)
                if (!jobs[i].fpc) finish(jobs[i], n_int);
        };
    }
    const int *list = *(const int **)a[1], n = *(int *)a[2];
    return [=] {
        launches++;
        if (held) return;
        for (int i = 0; i < n; i++) finish(jobs[list[i]], n_fft);
    };
}

static std::vector<uint16_t> number(int bits) {
    std::mt19937 rng(bits);
    std::vector<uint16_t> l((bits + 15) / 16);
    for (auto &x : l) x = (uint16_t)rng();
    const int top = (bits - 1) % 16;
    l.back() = (uint16_t)((l.back() & ((1u << top) - 1u)) | (1u << top));
    l[0] |= 1u;
    return l;
}

static const char *engine(int fft, int integer) {
    return fft && integer ? "both" : fft ? "fft" : integer ? "int" : "none";
}

int main() {
    fake::launch = launch;
    pfb_mr_t *e = nullptr;
    if (pfb_mr_create(&e, 0)) return 2;
    std::string line;
    while (std::getline(std::cin, line)) {
        std::istringstream in(line);
        std::string op;
        in >> op;
        n_fft = n_int = prep_fft = prep_int = launches = 0;
        if (op == "server") {
            long allow;
            int bits;
            in >> allow >> bits;
            const std::vector<uint16_t> l = number(bits);
            pfb_mr_server_t *s = nullptr;
            if (pfb_mr_server_create(e, nullptr, &s)) return 2;
            fake::allow = allow;
            pfb_mr_server_submit(s, l.data(), (int)l.size(), 7, nullptr, 0);
            pfb_mr_result_t r{};
            int n = 0;
            for (int i = 0; i < 200 && n == 0; i++) n = pfb_mr_server_poll(s, &r, 1, 100);
            if (n == 1) std::cout << "verdict " << (int)r.verdict;
            else std::cout << "stopped " << n;
            fake::allow = -1;
            pfb_mr_server_destroy(s);
            std::cout << " " << engine(n_fft, n_int) << std::endl;
        } else if (op == "mixed") {
            int streams;
            in >> streams;
            pfb_mr_server_t *s = nullptr;
            if (pfb_mr_server_create(e, nullptr, &s)) return 2;
            fake::no_streams = !streams;
            held = true;
            for (int bits : {3000, 9000}) {
                const std::vector<uint16_t> l = number(bits);
                pfb_mr_server_submit(s, l.data(), (int)l.size(), (uint64_t)bits, nullptr, 0);
            }
            pfb_mr_server_stats_t st{};
            for (int i = 0; i < 200 && !st.error && st.resident < 2; i++) {
                std::this_thread::sleep_for(std::chrono::milliseconds(20));
                pfb_mr_server_stats(s, &st);
            }
            held = false;
            pfb_mr_result_t r[2];
            int n = 0;
            for (int i = 0; i < 50 && n >= 0 && n < 2; i++) {
                const int k = pfb_mr_server_poll(s, r + n, 2 - n, 100);
                n = k < 0 ? k : n + k;
            }
            if (n == 2) std::cout << "verdict " << (int)r[0].verdict << " " << (int)r[1].verdict;
            else std::cout << "stopped " << n;
            fake::no_streams = false;
            pfb_mr_server_destroy(s);
            std::cout << " " << engine(n_fft, n_int) << std::endl;
        } else if (op == "batch") {
            long long bytes;
            int bits, n;
            in >> bytes >> bits >> n;
            const std::vector<uint16_t> l = number(bits);
            const std::vector<pfb_mr_number_t> nums(n, pfb_mr_number_t{l.data(), (int)l.size()});
            std::vector<int8_t> verdict(n);
            const size_t held = fake::used;
            fake::limit = bytes < 0 ? ~(size_t)0 : held + (size_t)bytes;
            fake::peak = held;
            const int rc = pfb_mr_test(e, nums.data(), n, 2u, verdict.data(), nullptr, 0);
            std::cout << "rc " << rc << " " << fake::peak - held << " " << engine(n_fft, n_int) << std::endl;
            fake::limit = ~(size_t)0;
        } else if (op == "tune") {
            int lg, q = 0, ch = 0;
            in >> lg;
            const int rc = pfb_mr_autotune(e, lg, lg, nullptr, 0, nullptr);
            pfb_mr_get_tuning(e, lg, &q, &ch);
            std::cout << "rc " << rc << " " << launches << " " << q << " " << ch << std::endl;
        } else if (op == "ctx") {
            long long bytes;
            int bits, n;
            in >> bytes >> bits >> n;
            const std::vector<uint16_t> l = number(bits);
            std::vector<uint64_t> all;
            for (int i = 0; i < n; i++) all.insert(all.end(), l.begin(), l.end());
            const size_t held = fake::used;
            fake::limit = bytes < 0 ? ~(size_t)0 : held + (size_t)bytes;
            pfb_mr_ctx_t *c = nullptr;
            const int rc = pfb_mr_ctx_create(e, all.data(), (int)l.size(), n, &c);
            std::cout << "rc " << rc << " " << fake::used - held << " " << engine(prep_fft, prep_int) << std::endl;
            pfb_mr_ctx_destroy(c);
            fake::limit = ~(size_t)0;
        }
    }
    pfb_mr_destroy(e);
    std::cout << "left " << fake::used << std::endl;
    return 0;
}
