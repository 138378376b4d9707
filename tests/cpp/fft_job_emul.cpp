// Runs the floating-point Montgomery engine (fft_device.cuh, fft_kernels.cuh)
// unchanged on the CPU, one candidate per CTA of cooperative fibers
// (tests/cpp/emul/), with the engine's own host set-up (mr_prep_host.h) and
// roots (fft_tables_host.h).  Input lines:
//
//   job mode base N [E]        whole test (mode 1: strong test, 2: strong Lucas
//                              test) or base^E mod N (mode 0)
//                              -> class bits verdict residue
//   overlap base N E N2 E2     two modular powers of one length class, the second
//                              advanced a step at a time by a launch of its own
//                              that runs in the middle of the first one's steps
//                              -> class residue residue2
//   ctx cls op N a b           an operation of a modular context (mr_job.cuh:
//                              CtxOp) on plain numbers -> result
//   step cls bits dbl kind N   one squaring of limbs of a pattern: kind 0
//                              all B/2 + 40, 1 all -(B/2 + 40), 2 alternating,
//                              3 random signs, 4 random limbs (the top limbs
//                              zero so that |x| < N)
//                              -> x, result (signed hexadecimal), largest |limb|
#include <functional>
#include <iostream>
#include <random>
#include <sstream>
#include <string>
#include <vector>

#include "mr_kernels.cuh"

#include "fft_kernels.cuh"
#include "fft_tables_host.h"
#include "mr_prep_host.h"

using namespace pfb::mr;

void pfb::mr::fp::host_bar_sync(int id, int n) { emu::named_wait(id, n); }
using pfb::big::Words;

static Words from_hex(const std::string &h) {
    Words w;
    size_t end = h.size();
    while (end > 0) {
        const size_t start = end >= 16 ? end - 16 : 0;
        w.push_back(std::stoull(h.substr(start, end - start), nullptr, 16));
        end = start;
    }
    pfb::big::trim(w);
    return w;
}

static std::string to_hex(Words t) {
    pfb::big::trim(t);
    if (t.empty()) return "0";
    std::string s;
    char buf[24];
    snprintf(buf, sizeof buf, "%llx", (unsigned long long)t.back());
    s += buf;
    for (size_t i = t.size() - 1; i-- > 0;) {
        snprintf(buf, sizeof buf, "%016llx", (unsigned long long)t[i]);
        s += buf;
    }
    return s;
}

// Signed value of limbs of b bits.
static std::string limbs_hex(const std::vector<int> &l, int b) {
    std::vector<uint32_t> d(l.size());
    long long c = 0;
    auto digits = [&](int sign) {
        c = 0;
        for (size_t i = 0; i < l.size(); i++) {
            const long long v = (long long)sign * l[i] + c;
            d[i] = (uint32_t)(v & ((1ll << b) - 1));
            c = v >> b;
        }
    };
    digits(1);
    const bool neg = c < 0;
    if (neg) digits(-1);
    return (neg ? "-" : "") + to_hex(pfb::big::from_limbs(d.data(), b, d.size()));
}

template <class F>
static fp::Tab tables(std::vector<fp::Cplx> &mem) {
    size_t off[2][3] = {};
    mem = fp::class_roots<F>(off);
    fp::Tab t{};
    for (int m = 0; m < 2; m++)
        for (int p = 0; p < 3; p++) t.t[m][p] = mem.data() + off[m][p];
    return t;
}

template <class F>
static void prep_job(JobDev &j, const fp::Tab &tab) {
    const int list[1] = {0};
    emu::run_grid(1, 1, F::T, [&] { fp::fft_prep_kernel<F>(&j, list, tab); }, F::smem());
}

// One launch: `total` quanta of `quantum` steps.
template <class F>
static void launch_job(JobDev &j, const fp::Tab &tab, unsigned total, int quantum) {
    const int list[1] = {0};
    int locks[1] = {0};
    unsigned counter = 0;
    emu::run_grid(1, 1, F::T, [&] {
        if (j.mode == 2)
            fp::fft_persist_kernel<F, true>(&j, list, 1, locks, &counter, total, quantum, tab);
        else
            fp::fft_persist_kernel<F>(&j, list, 1, locks, &counter, total, quantum, tab);
    }, F::smem());
}

template <class F>
static void run_job_cls(JobDev &j) {
    std::vector<fp::Cplx> mem;
    const fp::Tab tab = tables<F>(mem);
    prep_job<F>(j, tab);
    for (int launch = 0; j.phase != 3 && launch < 1 << 20; launch++) launch_job<F>(j, tab, 8u, 64);
}

// j2 takes a step whenever j has passed another 13 barriers of the block (the
// first ones are the scheduler's own, whose shared variable the two share here).
template <class F>
static void run_overlap_cls(JobDev &j, JobDev &j2) {
    std::vector<fp::Cplx> mem;
    const fp::Tab tab = tables<F>(mem);
    prep_job<F>(j, tab);
    prep_job<F>(j2, tab);
    long barrier = 0;
    bool nested = false;
    emu::at_barrier = [&] {
        if (nested || ++barrier < 8 || barrier % 13 || j2.phase == 3) return;
        nested = true;
        launch_job<F>(j2, tab, 1u, 1);
        nested = false;
    };
    launch_job<F>(j, tab, 1u, 64);
    emu::at_barrier = nullptr;
}

template <class F>
static void run_step(int b, int dbl, int kind, const Words &N) {
    const size_t n = F::N;
    std::vector<fp::Cplx> mem, sq(F::C), nn(F::C), nh(F::C);
    std::vector<int> xs(n);
    const fp::Tab gtab = tables<F>(mem);
    Words inv;
    if (!neg_inv_radix(N, n * b, inv)) {
        std::cout << "none" << std::endl;
        return;
    }
    std::vector<uint32_t> npl(n), nl(n);
    pfb::big::to_limbs(inv, b, npl.data(), n);
    pfb::big::to_limbs(N, b, nl.data(), n);
    std::mt19937_64 rng(kind + 17);
    std::vector<int> x(n, 0), y(n);
    const int ext = (1 << (b - 1)) + 40;
    const size_t used = pfb::big::bit_length(N) / b;  // |x| < N
    for (size_t i = 0; i + 1 < used; i++)
        x[i] = kind == 0 ? ext : kind == 1 ? -ext : kind == 2 ? (i & 1 ? ext : -ext)
             : kind == 3 ? (rng() & 1 ? ext : -ext) : (int)(rng() % (2 * ext + 1)) - ext;
    emu::run_grid(1, 1, F::T, [&] {
        PFB_DYNAMIC_SMEM(unsigned char, raw);
        fp::View w;
        fp::carve<F>(raw, sq.data(), xs.data(), w);
        fp::Tab tab = gtab;
        const fp::Cplx *sn = nullptr, *sh = nullptr;
        fp::resident<F>(w, tab, sn, sh);
        int lo[F::R1], hi[F::R1];
        fp::balanced<F>([&](int i) { return npl[i]; }, b, lo, hi);
        fp::spectrum<F>(w, tab, 0, lo, hi, nn.data());
        fp::balanced<F>([&](int i) { return nl[i]; }, b, lo, hi);
        fp::spectrum<F>(w, tab, 1, lo, hi, nh.data());
        for (int e = 0; e < F::R1; e++) {
            lo[e] = x[fp::tid1<F>() + e * F::T1];
            hi[e] = x[F::C + fp::tid1<F>() + e * F::T1];
        }
        __syncthreads();  // the spectra are complete
        tab = gtab;
        sn = nn.data();
        sh = nh.data();
        fp::resident<F>(w, tab, sn, sh);
        fp::step<F>(w, tab, sn, sh, b, true, dbl, lo, hi);
        fp::put_limbs<F>(y.data(), lo, hi);
    }, F::smem());
    int big = 0;
    for (int v : y) big = std::max(big, v < 0 ? -v : v);
    std::cout << limbs_hex(x, b) << " " << limbs_hex(y, b) << " " << big << std::endl;
}

template <class F>
static void run_ctx(int op, const Words &N, const Words &a, const Words &b) {
    const size_t n = F::N;
    const int n16 = (int)((pfb::big::bit_length(N) + 15) / 16);
    std::vector<fp::Cplx> mem, sq(F::C), nn(F::C), nh(F::C), ys(2 * F::C);
    const fp::Tab tab = tables<F>(mem);
    Words inv;
    if (!neg_inv_radix(N, n * fp::kCtxBits, inv)) {
        std::cout << "none" << std::endl;
        return;
    }
    std::vector<uint32_t> npl(n), nl(n);
    pfb::big::to_limbs(inv, fp::kCtxBits, npl.data(), n);
    pfb::big::to_limbs(N, fp::kCtxBits, nl.data(), n);
    JobDev j{};
    j.nn = reinterpret_cast<uint32_t *>(nn.data());
    j.nh = reinterpret_cast<uint32_t *>(nh.data());
    j.npl = npl.data();
    j.nl = nl.data();
    j.fpc = F::ID + 1;
    j.fbits = fp::kCtxBits;
    CtxExtra ex{};
    ex.ys = reinterpret_cast<uint32_t *>(ys.data());
    j.sq = reinterpret_cast<uint32_t *>(sq.data());
    auto wide = [&](const Words &w) {
        std::vector<uint16_t> t(n16);
        pfb::big::to_u16(w, t.data(), n16);
        return std::vector<uint64_t>(t.begin(), t.end());
    };
    const std::vector<uint64_t> A = wide(a), B = wide(b);
    std::vector<uint64_t> out(n16);
    const int list[1] = {0};
    emu::run_grid(1, 1, F::T, [&] { fp::fft_prep_kernel<F>(&j, list, tab); }, F::smem());
    emu::run_grid(1, 1, F::T, [&] {
        fp::fft_ctx_kernel<F>(&j, list, A.data(), B.data(), out.data(), n16, op, tab, &ex);
    }, F::smem());
    std::vector<uint16_t> o(out.begin(), out.end());
    std::cout << to_hex(pfb::big::from_u16(o.data(), o.size())) << std::endl;
}

// A candidate's host set-up and memory, as the host code lays it out.
struct Job {
    HostPrep hp;
    std::vector<uint32_t> x, res, npl, nl, e, lv[5];
    std::vector<fp::Cplx> nn, nh, sq, gy;
    JobDev j{};
    LucasDev lc{};
    Job(const Job &) = delete;
    Job(int mode, uint32_t base, const Words &N, const Words &E) {
        std::vector<uint16_t> limbs(std::max<size_t>(1, (pfb::big::bit_length(N) + 15) / 16));
        pfb::big::to_u16(N, limbs.data(), limbs.size());
        std::vector<uint16_t> el(std::max<size_t>(1, (pfb::big::bit_length(E) + 15) / 16));
        pfb::big::to_u16(E, el.data(), el.size());
        const pfb_mr_number_t num{limbs.data(), (int)limbs.size()}, ex{el.data(), (int)el.size()};
        host_prep(num, base, mode, mode ? nullptr : &ex, hp, true);
        if (!runs()) return;
        const size_t n = hp.x0.size();
        x = hp.x0;
        npl = hp.npl;
        nl = hp.nl;
        e = hp.exp;
        res.resize(n);
        nn.resize(n / 2);
        nh.resize(n / 2);
        j.x = x.data();
        j.res = res.data();
        j.nn = reinterpret_cast<uint32_t *>(nn.data());
        j.nh = reinterpret_cast<uint32_t *>(nh.data());
        j.npl = npl.data();
        j.nl = nl.data();
        j.exp = e.data();
        j.logl = hp.logl;
        j.fpc = hp.fpc;
        j.fbits = hp.fbits;
        if (fp::spectrum_outside(hp.fpc - 1)) {  // N'' lies at its start, as in the engine's layout
            sq.resize(n / 2);
            std::copy(npl.begin(), npl.end(), reinterpret_cast<uint32_t *>(sq.data()));
            j.npl = j.sq = reinterpret_cast<uint32_t *>(sq.data());
        }
        j.cursor = hp.cursor;
        j.extra = mode >= 1 ? hp.s - 1 : 0;
        j.base = base;
        j.mode = mode;
        if (mode == 2) {
            for (auto &v : lv) v.resize(n);
            gy.resize(n);
            lc.lv0 = lv[0].data();
            lc.lv1 = lv[1].data();
            lc.lqk = lv[2].data();
            lc.lt = lv[3].data();
            lc.lone = lv[4].data();
            lc.gy = reinterpret_cast<uint32_t *>(gy.data());
            lc.q = hp.q;
            lc.lb = hp.lb;
            j.lucas = &lc;
        }
    }
    bool runs() const { return hp.ok && hp.decided < 0 && hp.fpc; }
    std::string residue() const { return to_hex(pfb::big::from_limbs(res.data(), hp.fbits, res.size())); }
};

int main() {
    fp::c_first = fp::first_roots();
    std::string line;
    while (std::getline(std::cin, line)) {
        std::istringstream in(line);
        std::string op, sn, se;
        in >> op;
        if (op == "step") {
            int cls, b, dbl, kind;
            in >> cls >> b >> dbl >> kind >> sn;
            const Words N = from_hex(sn);
            switch (cls) {
#define PFB_CLS(F) \
    case fp::F::ID: run_step<fp::F>(b, dbl, kind, N); break;
                PFB_FP_CLASSES(PFB_CLS)
#undef PFB_CLS
            }
            continue;
        }
        if (op == "ctx") {
            int cls, o;
            std::string sa, sb;
            in >> cls >> o >> sn >> sa >> sb;
            switch (cls) {
#define PFB_CLS(F) \
    case fp::F::ID: run_ctx<fp::F>(o, from_hex(sn), from_hex(sa), from_hex(sb)); break;
                PFB_FP_CLASSES(PFB_CLS)
#undef PFB_CLS
            }
            continue;
        }
        if (op == "overlap") {
            uint32_t base = 2;
            std::string sn2, se2;
            in >> base >> sn >> se >> sn2 >> se2;
            Job a(0, base, from_hex(sn), from_hex(se)), b(0, base, from_hex(sn2), from_hex(se2));
            switch (a.hp.fpc - 1) {
#define PFB_CLS(F) \
    case fp::F::ID: run_overlap_cls<fp::F>(a.j, b.j); break;
                PFB_FP_CLASSES(PFB_CLS)
#undef PFB_CLS
            }
            std::cout << a.hp.fpc - 1 << " " << a.residue() << " " << b.residue() << std::endl;
            continue;
        }
        int mode = 1;
        uint32_t base = 2;
        in >> mode >> base >> sn >> se;
        Job job(mode, base, from_hex(sn), from_hex(se));
        const HostPrep &hp = job.hp;
        if (!job.runs()) {
            std::cout << "- 0 " << (hp.ok && hp.decided >= 0 ? hp.decided : -1) << " 0" << std::endl;
            continue;
        }
        switch (hp.fpc - 1) {
#define PFB_CLS(F) \
    case fp::F::ID: run_job_cls<fp::F>(job.j); break;
            PFB_FP_CLASSES(PFB_CLS)
#undef PFB_CLS
        }
        std::cout << hp.fpc - 1 << " " << hp.fbits << " " << (job.j.phase == 3 ? job.j.verdict : -2) << " "
                  << job.residue() << std::endl;
    }
    return 0;
}
