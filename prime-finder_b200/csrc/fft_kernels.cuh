// Kernels of the floating-point Montgomery engine (fft_device.cuh): set-up
// of a candidate, its exponent ladder and the persistent scheduler, one
// instance per length class.  The jobs are those of mr_job.cuh.
//
// Bound: the double-precision pipe (64 fused multiply-adds per clock and SM)
// for long numbers, the chain of passes and block barriers for short ones.
// Measured per squaring of one candidate on one SM, integer engine -> this
// one: 600 digits 14 -> 3.4 us, 10 000 digits 33 -> 8.3 us, 50 000 digits
// 98.6 -> 53.4 us.
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
    carve<F>(raw, nullptr, w);
    int lo[F::R1], hi[F::R1];
    balanced<F>(jb.npl, jb.fbits, lo, hi);
    spectrum<F>(w, tab, 0, lo, hi, reinterpret_cast<Cplx *>(jb.nn));
    balanced<F>(jb.nl, jb.fbits, lo, hi);
    spectrum<F>(w, tab, 1, lo, hi, reinterpret_cast<Cplx *>(jb.nh));
    balanced<F>(jb.x, jb.fbits, lo, hi);
    cta_sync<F>();
#pragma unroll
    for (int e = 0; e < F::R1; e++) {
        jb.x[threadIdx.x + e * F::T] = (uint32_t)lo[e];
        jb.x[F::C + threadIdx.x + e * F::T] = (uint32_t)hi[e];
    }
}

// Runs up to max_steps steps of one candidate (strong test or modular power).
template <class F>
__device__ void run_fft_job(JobDev *jp, int max_steps, const Tab &tab, unsigned char *raw, Cplx *gscratch) {
    JobDev jb;
    {
        const unsigned long long *src = reinterpret_cast<const unsigned long long *>(jp);
        unsigned long long *dst = reinterpret_cast<unsigned long long *>(&jb);
#pragma unroll
        for (int i = 0; i < (int)(sizeof(JobDev) / 8); i++) dst[i] = __ldcg(src + i);
    }
    View w;
    carve<F>(raw, gscratch, w);
    const Cplx *nn = reinterpret_cast<const Cplx *>(jb.nn), *nh = reinterpret_cast<const Cplx *>(jb.nh);
    const int b = jb.fbits;
    int cursor = jb.cursor, phase = jb.phase, extra = jb.extra, verdict = jb.verdict, steps = 0;
    int lo[F::R1], hi[F::R1];
#pragma unroll
    for (int e = 0; e < F::R1; e++) {
        lo[e] = (int)__ldcg(jb.x + threadIdx.x + e * F::T);
        hi[e] = (int)__ldcg(jb.x + F::C + threadIdx.x + e * F::T);
    }
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
            if (bit && jb.base != 2u) mul_small<F>(w, b, jb.base, lo, hi);
            cursor--;
            if (cursor < 0) phase = 1;
        } else {
            if (phase == 2) extra--;
            // (lo, hi) is x / R' = the plain residue; x itself is still in w.xs
            int *L = reinterpret_cast<int *>(w.A);
            to_digits<F>(w, b, jb.nl, lo, hi, L);
            bool one = true, nm1 = true;  // N odd: N - 1 differs from N in digit 0 only
            for (int i = threadIdx.x; i < F::N; i += F::T) {
                const uint32_t y = (uint32_t)L[i], n = jb.nl[i];
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
#pragma unroll
            for (int e = 0; e < F::R1; e++) {
                lo[e] = w.xs[(2 * e) * F::T + threadIdx.x];
                hi[e] = w.xs[(2 * e + 1) * F::T + threadIdx.x];
            }
        }
        steps++;
    }
#pragma unroll
    for (int e = 0; e < F::R1; e++) {
        jb.x[threadIdx.x + e * F::T] = (uint32_t)lo[e];
        jb.x[F::C + threadIdx.x + e * F::T] = (uint32_t)hi[e];
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
// job locked or finished leaves.  scratch: C points per CTA (classes whose
// spectrum of x^2 does not fit in shared memory).
template <class F>
__global__ void __launch_bounds__(F::T, F::MINB)
fft_persist_kernel(JobDev *jobs, const int *list, int n, int *locks, unsigned int *counter, unsigned int total,
                   int quantum, Tab tab, Cplx *scratch) {
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
        run_fft_job<F>(jobs + j, quantum, tab, raw, F::SQS ? nullptr : scratch + (size_t)blockIdx.x * F::C);
        if (threadIdx.x == 0) {
            __threadfence();
            atomicExch(&locks[j], 0);
        }
    }
}

}  // namespace fp
}  // namespace mr
}  // namespace pfb
