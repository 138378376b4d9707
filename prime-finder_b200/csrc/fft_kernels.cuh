// Kernels of the floating-point Montgomery engine (fft_device.cuh): set-up
// of a candidate, its exponent ladder and the persistent scheduler, one
// instance per length class.  The jobs are those of mr_job.cuh.
//
// Bound: the double-precision pipe (64 fused multiply-adds per clock and SM)
// for long numbers, the chain of passes and block barriers for short ones.
// Measured per squaring of one candidate on one SM, integer engine -> this
// one: 600 digits 14 -> 3.2 us, 9800 digits 33 -> 8.0 us, 50 000 digits
// 98.6 -> 43 us, 100 000 digits 186 -> 79 us.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "fft_device.cuh"
#include "mr_job.cuh"

namespace pfb {
namespace mr {
namespace fp {

// Set-up of the listed jobs, one CTA each: the spectra of N'' and N, and x's
// digits to balanced limbs.
template <class F>
__global__ void __launch_bounds__(F::T, F::MINB) fft_prep_kernel(JobDev *jobs, const int *list, Tab tab) {
    PFB_DYNAMIC_SMEM(unsigned char, raw);
    const JobDev jb = jobs[list[blockIdx.x]];
    View w;
    carve<F>(raw, nullptr, nullptr, w);
    const Cplx *none = nullptr, *none2 = nullptr;
    resident<F>(w, tab, none, none2);
    int lo[F::R1], hi[F::R1];
    balanced<F>([&](int i) { return jb.npl[i]; }, jb.fbits, lo, hi);
    spectrum<F>(w, tab, 0, lo, hi, reinterpret_cast<Cplx *>(jb.nn));
    balanced<F>([&](int i) { return jb.nl[i]; }, jb.fbits, lo, hi);
    spectrum<F>(w, tab, 1, lo, hi, reinterpret_cast<Cplx *>(jb.nh));
    if (!jb.x) return;  // (a modulus of a context)
    balanced<F>([&](int i) { return jb.x[i]; }, jb.fbits, lo, hi);
    cta_sync<F>();
    if (jb.mode == 2) {  // V_0 = 2, V_1 = 1, Q^0 = 1 and 1 itself, in Montgomery form
        const LucasDev lc = *jb.lucas;
        put_limbs<F>(lc.lv1, lo, hi);
        put_limbs<F>(lc.lqk, lo, hi);
        put_limbs<F>(lc.lone, lo, hi);
        int l2[F::R1], h2[F::R1];
#pragma unroll
        for (int e = 0; e < F::R1; e++) {
            l2[e] = lo[e];
            h2[e] = hi[e];
        }
        add_mul<F>(w, jb.fbits, 1, l2, h2, lo, hi);
        put_limbs<F>(lc.lv0, lo, hi);
    } else {
        put_limbs<F>(jb.x, lo, hi);
    }
}

// The job's state, which another SM may have written earlier in the launch.
__device__ __forceinline__ JobDev load_job(const JobDev *jp) {
    JobDev jb;
    const unsigned long long *src = reinterpret_cast<const unsigned long long *>(jp);
    unsigned long long *dst = reinterpret_cast<unsigned long long *>(&jb);
#pragma unroll
    for (int i = 0; i < (int)(sizeof(JobDev) / 8); i++) dst[i] = __ldcg(src + i);
    return jb;
}

// Runs up to max_steps steps of one candidate (strong test or modular power).
template <class F>
__device__ void run_fft_job(JobDev *jp, int max_steps, Tab tab, unsigned char *raw) {
    const JobDev jb = load_job(jp);
    View w;
    carve<F>(raw, reinterpret_cast<Cplx *>(jb.sq), reinterpret_cast<int *>(jb.x), w);
    const Cplx *nn = reinterpret_cast<const Cplx *>(jb.nn), *nh = reinterpret_cast<const Cplx *>(jb.nh);
    resident<F>(w, tab, nn, nh);
    const int b = jb.fbits;
    int cursor = jb.cursor, phase = jb.phase, extra = jb.extra, verdict = jb.verdict, steps = 0;
    int lo[F::R1], hi[F::R1];
    get_limbs<F>(jb.x, lo, hi);
    while (steps < max_steps && phase != 3) {
        // phase 0 and 2 square; phases 1 and 2 then compare the residue
        bool square = phase != 1;
        uint32_t bit = 0;
        if (phase == 0) bit = (__ldg(jb.exp + (cursor >> 5)) >> (cursor & 31)) & 1u;
        for (;;) {
            step<F>(w, tab, nn, nh, b, square, bit && jb.base == 2u && square ? 1 : 0, lo, hi);
            if (!square || phase != 2) break;
            square = false;
        }
        if (phase == 0) {
            if (bit && jb.base != 2u) add_mul<F>(w, b, (int)jb.base - 1, lo, hi, lo, hi);
            cursor--;
            if (cursor < 0) phase = 1;
        } else {
            if (phase == 2) extra--;
            // (lo, hi) is x / R' = the plain residue; x itself is still in w.xs
            int *L = reinterpret_cast<int *>(w.A);
            to_digits<F>(w, b, jb.nl, lo, hi, L);
            bool one = true, nm1 = true;  // N odd: N - 1 differs from N in digit 0 only
            for (int i = threadIdx.x; i < F::N; i += F::T) {
                const uint32_t y = (uint32_t)L[lpos<F>(i)], n = jb.nl[i];
                one = one && (y == (i == 0 ? 1u : 0u));
                nm1 = nm1 && (y == (i == 0 ? n - 1u : n));
                if (phase == 1) jb.res[i] = y;
            }
            const bool all_one = vote_and<F>(one), all_nm1 = vote_and<F>(nm1);
            if (jb.mode == 0) {
                phase = 3;
            } else if (all_nm1 || (phase == 1 && all_one)) {
                verdict = 1;
                phase = 3;
            } else if (extra <= 0) {
                verdict = 0;
                phase = 3;
            } else {
                phase = 2;
            }
            load_x<F>(w, lo, hi);
        }
        steps++;
    }
    put_limbs<F>(jb.x, lo, hi);
    if (threadIdx.x == 0) {
        jp->cursor = cursor;
        jp->phase = phase;
        jp->extra = extra;
        jp->verdict = verdict;
        jp->steps = jb.steps + steps;
    }
    __syncthreads();
}

// Strong Lucas test (the ladder of mr_kernels.cuh: run_lucas): V_k, V_(k+1)
// and Q^k are kept as limb arrays, each thread reading and writing its own.
// Up to max_steps ladder bits or final steps.  Every Montgomery step of the
// ladder goes through one copy of the code: `todo` lists what is left of the
// current bit.
template <class F>
__device__ void run_fft_lucas(JobDev *jp, int max_steps, Tab tab, unsigned char *raw) {
    const JobDev jb = load_job(jp);
    const LucasDev lc = *jb.lucas;
    View w;
    carve<F>(raw, reinterpret_cast<Cplx *>(jb.sq), reinterpret_cast<int *>(jb.x), w);
    Cplx *ys = reinterpret_cast<Cplx *>(lc.gy);
    const Cplx *nn = reinterpret_cast<const Cplx *>(jb.nn), *nh = reinterpret_cast<const Cplx *>(jb.nh);
    resident<F>(w, tab, nn, nh);
    const int b = jb.fbits, aq = lc.q < 0 ? -lc.q : lc.q;
    int cursor = jb.cursor, phase = jb.phase, extra = jb.extra, verdict = jb.verdict, steps = 0;
    int lo[F::R1], hi[F::R1], yl[F::R1], yh[F::R1];
    // a bit: PRODUCT (V_k V_(k+1)), SQUARE (V_2k or V_2k+2), QPOW; after the
    // last one the checks U_d == 0, then V_(d 2^r) == 0, each on a plain
    // residue; a doubling: SQUARE, QPOW, then the second check
    enum { PRODUCT, SQUARE, QPOW, CHECK_U, CHECK_V };
    while (steps < max_steps && phase != 3) {
        uint32_t bit = 0;
        if (phase == 0) bit = (__ldg(jb.exp + (cursor >> 5)) >> (cursor & 31)) & 1u;
        int first = phase == 0 ? PRODUCT : (phase == 1 ? CHECK_U : SQUARE), last = phase == 0 ? QPOW : CHECK_V;
        bool hit = false;
        for (int op = first; op <= last && !hit; op++) {
            if (phase == 2 && op == CHECK_U) continue;
            if (op == QPOW && aq == 1) {  // Q = -1: Q^k = (-1)^k
                get_limbs<F>(lc.lone, lo, hi);
                if (bit) {
#pragma unroll
                    for (int e = 0; e < F::R1; e++) {
                        lo[e] = -lo[e];
                        hi[e] = -hi[e];
                    }
                }
                put_limbs<F>(lc.lqk, lo, hi);
                continue;
            }
            const Cplx *y = nullptr;
            if (op == PRODUCT) {
                get_limbs<F>(lc.lv1, lo, hi);
                spectrum<F>(w, tab, 0, lo, hi, ys);
                spectrum<F>(w, tab, 1, lo, hi, ys + F::C);
                y = ys;
            }
            get_limbs<F>(op == QPOW ? lc.lqk : (op == SQUARE && bit ? lc.lv1 : lc.lv0), lo, hi);
            if (op == CHECK_U) {  // V_d - 2 V_(d+1)
                get_limbs<F>(lc.lv1, yl, yh);
                add_mul<F>(w, b, -2, yl, yh, lo, hi);
            }
            step<F>(w, tab, nn, nh, b, op <= QPOW, 0, lo, hi, y);
            if (op == PRODUCT) {
                put_limbs<F>(lc.lt, lo, hi);
            } else if (op == SQUARE) {
                get_limbs<F>(lc.lqk, yl, yh);
                // V_2k = T2 - 2 Q^k, V_2k+2 = T2 - 2 Q Q^k, V_2k+1 = T1 - Q^k
                add_mul<F>(w, b, bit ? -2 * lc.q : -2, yl, yh, lo, hi);
                put_limbs<F>(bit ? lc.lv1 : lc.lv0, lo, hi);
                if (phase == 0) {
                    get_limbs<F>(lc.lt, lo, hi);
                    add_mul<F>(w, b, -1, yl, yh, lo, hi);
                    put_limbs<F>(bit ? lc.lv0 : lc.lv1, lo, hi);
                }
            } else if (op == QPOW) {
                if (bit) add_mul<F>(w, b, lc.q - 1, lo, hi, lo, hi);
                put_limbs<F>(lc.lqk, lo, hi);
            } else {
                int *L = reinterpret_cast<int *>(w.A);
                to_digits<F>(w, b, jb.nl, lo, hi, L);
                bool z = true;
                for (int i = threadIdx.x; i < F::N; i += F::T) z = z && L[lpos<F>(i)] == 0;
                hit = vote_and<F>(z);
            }
        }
        if (phase == 0) {
            cursor--;
            if (cursor < 0) phase = 1;
        } else {
            if (phase == 2) extra--;
            verdict = hit ? 1 : 0;
            phase = hit || extra <= 0 ? 3 : 2;
        }
        steps++;
    }
    if (threadIdx.x == 0) {
        jp->cursor = cursor;
        jp->phase = phase;
        jp->extra = extra;
        jp->verdict = verdict;
        jp->steps = jb.steps + steps;
    }
    __syncthreads();
}

// Persistent scheduler over the n listed jobs, all of class F: CTAs take
// quanta (`quantum` steps of one job) until `total` are handed out; quantum q
// goes to the first unfinished, unlocked job at or after position q mod n.
// One warp looks at 32 jobs at a time.  Nothing waits: a CTA that finds every
// job locked or finished leaves.  LUCAS: all jobs are Lucas tests.
template <class F, bool LUCAS = false>
__global__ void __launch_bounds__(F::T, F::MINB)
fft_persist_kernel(JobDev *jobs, const int *list, int n, int *locks, unsigned int *counter, unsigned int total,
                   int quantum, Tab tab) {
    PFB_DYNAMIC_SMEM(unsigned char, raw);
    __shared__ int s_job;
    const unsigned FULL = 0xffffffffu;
    for (;;) {
        if (threadIdx.x < 32) {
            const int lane = (int)threadIdx.x;
            unsigned int q = 0;
            if (lane == 0) q = atomicAdd(counter, 1u);
            q = __shfl_sync(FULL, q, 0);
            int job = -1;
            for (int base = 0; q < total && base < n && job < 0; base += 32) {
                int j = -1;
                bool live = false;
                if (base + lane < n) {
                    j = list[(q + (unsigned int)(base + lane)) % (unsigned int)n];
                    live = __ldcg(&jobs[j].phase) != 3;
                }
                unsigned cand = __ballot_sync(FULL, live);
                while (cand && job < 0) {
                    const int src = __ffs((int)cand) - 1;
                    cand &= cand - 1u;
                    int got = 0;
                    if (lane == src && atomicCAS(&locks[j], 0, 1) == 0) {
                        __threadfence();
                        got = __ldcg(&jobs[j].phase) != 3;
                        if (!got) atomicExch(&locks[j], 0);
                    }
                    got = __shfl_sync(FULL, got, src);
                    const int jj = __shfl_sync(FULL, j, src);
                    if (got) job = jj;
                }
            }
            if (lane == 0) s_job = job;
        }
        __syncthreads();
        const int j = s_job;
        __syncthreads();
        if (j < 0) break;
        if constexpr (LUCAS) run_fft_lucas<F>(jobs + j, quantum, tab, raw);
        else run_fft_job<F>(jobs + j, quantum, tab, raw);
        if (threadIdx.x == 0) {
            __threadfence();
            atomicExch(&locks[j], 0);
        }
    }
}

// One operation of a modular context (mr_job.cuh: CtxOp, without the raw
// products) on the listed moduli, one CTA each: operands and results in 16-bit
// limbs, one per uint64, at A + m n16 and so on for modulus m; digits of 11
// bits (n = 2 H: the integer engine's radix R' = 2^(22 H) + 1, so the working
// form is the same).  Operands, results and the modulus' own buffers are all
// that a CTA touches.
constexpr int kCtxBits = 11;
template <class F>
__global__ void __launch_bounds__(F::T, F::MINB)
fft_ctx_kernel(const JobDev *jobs, const int *list, const uint64_t *A, const uint64_t *B, uint64_t *out, int n16,
               int op, Tab tab, const CtxExtra *ex) {
    PFB_DYNAMIC_SMEM(unsigned char, raw);
    const int m = list[blockIdx.x];
    const JobDev jb = jobs[m];
    View w;
    carve<F>(raw, reinterpret_cast<Cplx *>(jb.sq), nullptr, w);
    const Cplx *nn = reinterpret_cast<const Cplx *>(jb.nn), *nh = reinterpret_cast<const Cplx *>(jb.nh);
    resident<F>(w, tab, nn, nh);
    auto digit = [&](const uint64_t *src) {
        return [=](int i) {
            const int bit = kCtxBits * i, q = bit >> 4, off = bit & 15;
            const uint32_t v = (q < n16 ? (uint32_t)(src[q] & 0xFFFFull) : 0u) |
                               (q + 1 < n16 ? (uint32_t)(src[q + 1] & 0xFFFFull) << 16 : 0u);
            return (v >> off) & ((1u << kCtxBits) - 1u);
        };
    };
    int lo[F::R1], hi[F::R1];
    const Cplx *y = nullptr;
    if (op == CTX_MODMUL) {
        Cplx *yo = reinterpret_cast<Cplx *>(ex[m].ys);
        balanced<F>(digit(B + (size_t)m * n16), kCtxBits, lo, hi);
        spectrum<F>(w, tab, 0, lo, hi, yo);
        spectrum<F>(w, tab, 1, lo, hi, yo + F::C);
        y = yo;
    }
    balanced<F>(digit(A + (size_t)m * n16), kCtxBits, lo, hi);
    step<F>(w, tab, nn, nh, kCtxBits, op != CTX_FROM, 0, lo, hi, y);
    int *L = reinterpret_cast<int *>(w.A);
    to_digits<F>(w, kCtxBits, jb.nl, lo, hi, L);
    uint64_t *o = out + (size_t)m * n16;
    for (int k = threadIdx.x; k < n16; k += F::T) {
        const int bit = 16 * k, i = bit / kCtxBits, off = bit - kCtxBits * i;
        unsigned long long v = 0;
#pragma unroll
        for (int q = 0; q < 3; q++)
            if (i + q < F::N) v |= (unsigned long long)(uint32_t)L[lpos<F>(i + q)] << (kCtxBits * q);
        o[k] = (v >> off) & 0xFFFFull;
    }
}

}  // namespace fp
}  // namespace mr
}  // namespace pfb
