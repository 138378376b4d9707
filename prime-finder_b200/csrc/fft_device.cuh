// Floating-point form of the Montgomery step (the strong test's and the
// modular powers' squarings): exact integer products by weighted complex
// FFTs in double precision, one CTA per candidate.
//
// x is held as n = 2 C signed limbs of b bits (B = 2^b), limb j and limb
// j + C together one complex point.  With the Montgomery radix R' = B^n + 1:
//
//   D  = x^2 mod (B^n + 1)
//   m  = D N'' mod (B^n + 1)                 N'' = -N^-1 mod R', spectrum stored
//   U  = (x^2 + m N) / R'                    spectrum of N stored
//
// U is found modulo M2 = B^n + B^(n/2) + 1, where R' = -B^(n/2) has the
// inverse B^(n/2) + 1: the sum x^2 + m N is formed on the spectra (one
// inverse transform for both), and division by R' is a linear map of the two
// halves.  Seven complex transforms of length C per squaring, where the
// integer form (mr_device.cuh) takes eight of length 2 C for each of two
// primes.
//
//   B^n + 1:             z_j = x_j + i x_(j+C)      modulo y^C - i
//   B^n + B^(n/2) + 1:   z_j = x_j + w x_(j+C)      modulo y^C - w, w = e^(2 pi i/3)
//
// The transform is the remainder tree of y^C - e^(i phi): a node y^(2m) - r^2
// has the children y^m - r and y^m + r, so a butterfly is (lo + r hi, lo - r
// hi) with one r per node: no weighting sweeps, and the first pass has the
// same few constants in every thread.
//
// Limbs are signed and redundant (|limb| <= B/2 + 40): the coefficients are
// brought back to limbs by three local carry steps, with no carry chain over
// the number.  |U| < 0.7 N is a signed residue; B^n is far above it, so the
// limbs found modulo M2 are U itself and not U plus a multiple of M2.
//
// Exactness.  A product of two operands z, z' of C points by these transforms
// has an error below |z| |z'| (3 levels + 4) 5 2^-53 in every coefficient
// (2-norms; the argument of Percival, "Rapid multiplication modulo the sum
// and difference of highly composite numbers", Math. Comp. 72 (2003), with 5
// units for a level: a fused forward butterfly with its rounded root makes
// at most 3.8 of the norm it hands on, an inverse one 3.8).  With |limb| at
// most B/2 + 40, |z|^2 <= 1.5 n limb^2 modulo M2 (z = x + w y); U adds two
// products, and its halves are re -+ im / sqrt(3): 3.5 n limb^2 in all.
// limb_bits() keeps that below 0.4, so the rounding to integers is exact for
// all inputs, not only for likely ones.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

namespace pfb {
namespace mr {
namespace fp {

struct alignas(16) Cplx {
    double re, im;
};

// ---- length classes --------------------------------------------------------
// C = 2^k or 3 2^k complex points, passes of radix R1 (with the factor 3), R2,
// R3, R4 (R4 = 1: three passes), T threads.  Each holds one group of the first
// pass (T = T1 = C / R1; the second half of a warp repeats the first when T1 =
// 16): the last inverse pass, the carries and the next first pass stay in
// registers.  SQS: x^2's spectrum waits in
// shared memory, XSS: so do x's limbs (else in the candidate's global memory:
// jb.sq, jb.x); PADL: one unused point per 2^PADL in shared memory against
// bank conflicts of the last pass.
constexpr int kResident = 1024;
template <int ID_, int C_, int R1_, int R2_, int R3_, int R4_, int T_, bool SQS_, bool XSS_, int MINB_>
struct Cls {
    static constexpr int ID = ID_, C = C_, R1 = R1_, R2 = R2_, R3 = R3_, R4 = R4_, T = T_, T1 = C_ / R1_, N = 2 * C_;
    static constexpr bool SQS = SQS_, XSS = XSS_;
    static constexpr int MINB = MINB_;
    static constexpr int NPASS = R4_ > 1 ? 4 : 3;
    static constexpr int RM = R4_ > 1 ? R4_ : R3_;  // radix of the middle sweep
    static constexpr int PADL = RM >= 16 ? 4 : 3;
    static constexpr int WARPS = T / 32;
    // After the first pass the R1 blocks are transforms of their own: each team
    // of warps keeps to its share of them (C / TEAMS consecutive points) until
    // the last inverse pass, so only its own warps wait for one another there.
    // Where that leaves a team's lanes idle, or saves a barrier of 128 threads
    // at most (1024 and 2048 points: 8 and 11 % slower), all warps are one team.
    static constexpr int TEAMS = C_ == 1024 || C_ == 2048                    ? 1
                                 : R1_ % WARPS == 0                          ? WARPS
                                 : WARPS % 2 == 0 && R1_ % (WARPS / 2) == 0 ? WARPS / 2
                                 : WARPS % 4 == 0 && R1_ % (WARPS / 4) == 0 ? WARPS / 4
                                                                            : 1;
    static constexpr int TT = T / TEAMS;  // threads of a team
    // short numbers, whose steps are a chain of latencies: the roots and the
    // spectra of N'' and N are copied to shared memory for a quantum
    static constexpr bool RES = C_ <= kResident;
    static constexpr int ROOTS = 2 * (R2_ / 2 * R1_ + R3_ / 2 * R1_ * R2_ + (R4_ > 1 ? R4_ / 2 * R1_ * R2_ * R3_ : 0));
    static_assert(R1_ * R2_ * R3_ * R4_ == C_ && T % 32 == 0 && N % T == 0, "passes");
    static_assert(T1 == T || (T1 == 16 && T == 32), "one group of the first pass per thread");
    // shared memory: points (padded), x^2's spectrum, x's limbs, carries
    // between warps, scratch words
    static constexpr int A_PTS = C_ + (C_ >> PADL);
    static constexpr size_t smem() {
        return (size_t)A_PTS * 16 + (SQS_ ? (size_t)C_ * 16 : 0) + (XSS_ ? (size_t)C_ * 8 : 0) +
               (size_t)2 * WARPS * R1_ * 8 + 256 + (RES ? (size_t)(2 * C_ + ROOTS) * 16 : 0);
    }
};

constexpr int kClasses = 16;
using Cls0 = Cls<0, 64, 4, 4, 4, 1, 32, true, true, 8>;
using Cls1 = Cls<1, 96, 3, 8, 4, 1, 32, true, true, 8>;
using Cls2 = Cls<2, 128, 4, 8, 4, 1, 32, true, true, 8>;
using Cls3 = Cls<3, 192, 3, 4, 4, 4, 64, true, true, 6>;
using Cls4 = Cls<4, 256, 4, 4, 4, 4, 64, true, true, 6>;
using Cls5 = Cls<5, 384, 6, 8, 8, 1, 64, true, true, 6>;
using Cls6 = Cls<6, 512, 8, 8, 8, 1, 64, true, true, 6>;
using Cls7 = Cls<7, 768, 6, 16, 8, 1, 128, true, true, 4>;
using Cls8 = Cls<8, 1024, 8, 16, 8, 1, 128, true, true, 3>;
using Cls9 = Cls<9, 1536, 12, 8, 16, 1, 128, true, true, 2>;
using Cls10 = Cls<10, 2048, 16, 16, 8, 1, 128, true, true, 2>;
using Cls11 = Cls<11, 3072, 12, 16, 16, 1, 256, true, true, 1>;
using Cls12 = Cls<12, 4096, 16, 16, 16, 1, 256, true, true, 1>;
using Cls13 = Cls<13, 6144, 24, 16, 16, 1, 256, false, true, 1>;
using Cls14 = Cls<14, 8192, 16, 8, 8, 8, 512, false, true, 1>;
using Cls15 = Cls<15, 12288, 24, 8, 8, 8, 512, false, false, 1>;
#define PFB_FP_CLASSES(F)                                                                                     \
    F(Cls0) F(Cls1) F(Cls2) F(Cls3) F(Cls4) F(Cls5) F(Cls6) F(Cls7) F(Cls8) F(Cls9) F(Cls10) F(Cls11) F(Cls12) \
        F(Cls13) F(Cls14) F(Cls15)

// Whether x^2's spectrum of a class lies in global memory (C points).
inline bool spectrum_outside(int cls) {
#define PFB_CLS(F) !F::SQS,
    static const bool o[kClasses] = {PFB_FP_CLASSES(PFB_CLS)};
#undef PFB_CLS
    return o[cls];
}

inline int class_points(int cls) {
#define PFB_CLS(F) F::C,
    static const int c[kClasses] = {PFB_FP_CLASSES(PFB_CLS)};
#undef PFB_CLS
    return c[cls];
}

// Largest b for which every coefficient is provably rounded to the right
// integer (see the head of the file).
inline int limb_bits(int cls) {
    const int C = class_points(cls);
    int lv = 0;
    while ((1 << lv) < C) lv++;
    for (int b = 24;; b--) {
        const double limb = ldexp(1.0, b - 1) + 40.0;
        const double err = 3.5 * (2.0 * C) * limb * limb * (3.0 * lv + 4.0) * 5.0 * ldexp(1.0, -53);
        if (err < 0.4) return b;
    }
}

// ---- tables ----------------------------------------------------------------
// Roots of the passes after the first: [modulus][pass - 2] planes [q][node],
// R/2 planes per pass (level 0: 1 root, level s: 2^(s-1) roots; the others
// are i times those).
struct Tab {
    const Cplx *t[2][3];
};

// The first pass' roots, the same for every length: entry q of a radix-32
// group at the root of the tree.
// (tree of binary levels), and for a radix 3 r group the root r and r^2 of
// the ternary level, then for each child the roots of a radix-8 group.
struct First {
    Cplx r[2][16];
    Cplx t[2][2 + 3 * 4];
};
__constant__ First c_first;

#ifdef __CUDA_ARCH__
__device__ __forceinline__ Cplx ldg(const Cplx *p) {
    const double2 v = __ldg(reinterpret_cast<const double2 *>(p));
    return Cplx{v.x, v.y};
}
__device__ __forceinline__ Cplx ldcg(const Cplx *p) {
    const double2 v = __ldcg(reinterpret_cast<const double2 *>(p));
    return Cplx{v.x, v.y};
}
// Barrier id of the block's named barriers, for N threads.
template <int N>
__device__ __forceinline__ void bar_sync(int id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(N) : "memory"); }
__device__ __forceinline__ long long bits_of(double d) { return __double_as_longlong(d); }
__device__ __forceinline__ double from_bits(long long v) { return __longlong_as_double(v); }
#else
void host_bar_sync(int id, int n);  // (the CPU emulation's)
template <int N>
inline void bar_sync(int id) { host_bar_sync(id, N); }
inline Cplx ldg(const Cplx *p) { return *p; }
inline Cplx ldcg(const Cplx *p) { return *p; }
inline long long bits_of(double d) {
    long long v;
    memcpy(&v, &d, 8);
    return v;
}
inline double from_bits(long long v) {
    double d;
    memcpy(&d, &v, 8);
    return d;
}
#endif

template <class F>
__device__ __forceinline__ void cta_sync() {
    if (F::T == 32) __syncwarp();
    else __syncthreads();
}

// The threads of this thread's team.
template <class F>
__device__ __forceinline__ void team_sync() {
    if (F::TT == 32) __syncwarp();
    else if (F::TEAMS == 1) __syncthreads();
    else bar_sync<F::TT>(1 + (int)threadIdx.x / F::TT);
}

template <class F>
__device__ __forceinline__ int padx(int i) {
    return i + (i >> F::PADL);
}

// int (|v| < 2^31) to double without the conversion unit: 2^52 + 2^31 + v has
// v + 2^31 in its low word.
__device__ __forceinline__ double to_double(int v) {
    const unsigned u = (unsigned)v ^ 0x80000000u;
    return from_bits((long long)((0x43300000ull << 32) | u)) - 4503601774854144.0;
}

// ---- butterflies -----------------------------------------------------------
// (a, b) <- (a + r b, a - r b), r replaced by i r when ROT.
template <bool ROT>
__device__ __forceinline__ void bf_fwd(Cplx &a, Cplx &b, const Cplx &r) {
    const double br = ROT ? -b.im : b.re, bi = ROT ? b.re : b.im;
    const double tr = fma(-r.im, bi, fma(r.re, br, a.re));
    const double ti = fma(r.re, bi, fma(r.im, br, a.im));
    b.re = fma(2.0, a.re, -tr);
    b.im = fma(2.0, a.im, -ti);
    a.re = tr;
    a.im = ti;
}

// The inverse, twice it: (p, q) <- (p + q, (p - q) conj(r)).
template <bool ROT>
__device__ __forceinline__ void bf_inv(Cplx &p, Cplx &q, const Cplx &r) {
    const double dr0 = p.re - q.re, di0 = p.im - q.im;
    p.re += q.re;
    p.im += q.im;
    const double dr = ROT ? di0 : dr0, di = ROT ? -dr0 : di0;  // times conj(i) = -i
    q.re = fma(dr, r.re, di * r.im);
    q.im = fma(di, r.re, -(dr * r.im));
}

// A group's levels; tw[0] the root of the first level, tw[2^(s-1) + u] that
// of node 2u of level s.
template <int R>
__device__ __forceinline__ void fwd_group(Cplx *v, const Cplx *tw) {
#pragma unroll
    for (int half = R / 2, nodes = 1; half >= 1; half >>= 1, nodes <<= 1) {
#pragma unroll
        for (int nd = 0; nd < nodes; nd++) {
            const Cplx &r = tw[nodes == 1 ? 0 : nodes / 2 + nd / 2];
#pragma unroll
            for (int e = 0; e < half; e++) {
                const int at = nd * 2 * half + e;
                if (nd & 1) bf_fwd<true>(v[at], v[at + half], r);
                else bf_fwd<false>(v[at], v[at + half], r);
            }
        }
    }
}

template <int R>
__device__ __forceinline__ void inv_group(Cplx *v, const Cplx *tw) {
#pragma unroll
    for (int half = 1, nodes = R / 2; half < R; half <<= 1, nodes >>= 1) {
#pragma unroll
        for (int nd = 0; nd < nodes; nd++) {
            const Cplx &r = tw[nodes == 1 ? 0 : nodes / 2 + nd / 2];
#pragma unroll
            for (int e = 0; e < half; e++) {
                const int at = nd * 2 * half + e;
                if (nd & 1) bf_inv<true>(v[at], v[at + half], r);
                else bf_inv<false>(v[at], v[at + half], r);
            }
        }
    }
}

// A group of the first pass, radix 2^k or 3 2^k.  The ternary level takes
// y^(3m) - r^3 to y^m - r, y^m - r z, y^m - r z^2, z = e^(2 pi i / 3).
template <int R, int MOD>
__device__ __forceinline__ void fwd_first(Cplx *v) {
    if constexpr (R % 3 == 0) {
        constexpr int Q = R / 3;
        constexpr double H = 0.86602540378443864676;
        const Cplx *w = c_first.t[MOD];
#pragma unroll
        for (int e = 0; e < Q; e++) {
            const Cplx f = v[e], g = v[e + Q], h = v[e + 2 * Q];
            const Cplx b{fma(w[0].re, g.re, -(w[0].im * g.im)), fma(w[0].re, g.im, w[0].im * g.re)};
            const Cplx s{fma(-w[1].im, h.im, fma(w[1].re, h.re, b.re)), fma(w[1].re, h.im, fma(w[1].im, h.re, b.im))};
            const Cplx d{fma(2.0, b.re, -s.re), fma(2.0, b.im, -s.im)};  // b - c
            const double tr = fma(-0.5, s.re, f.re), ti = fma(-0.5, s.im, f.im);
            v[e] = Cplx{f.re + s.re, f.im + s.im};
            v[e + Q] = Cplx{fma(-H, d.im, tr), fma(H, d.re, ti)};
            v[e + 2 * Q] = Cplx{fma(H, d.im, tr), fma(-H, d.re, ti)};
        }
        if constexpr (Q > 1) {
#pragma unroll
            for (int k = 0; k < 3; k++) fwd_group<Q>(v + k * Q, w + 2 + 4 * k);
        }
    } else {
        fwd_group<R>(v, c_first.r[MOD]);
    }
}

template <int R, int MOD>
__device__ __forceinline__ void inv_last(Cplx *v) {
    if constexpr (R % 3 == 0) {
        constexpr int Q = R / 3;
        constexpr double H = 0.86602540378443864676;
        const Cplx *w = c_first.t[MOD];
        if constexpr (Q > 1) {
#pragma unroll
            for (int k = 0; k < 3; k++) inv_group<Q>(v + k * Q, w + 2 + 4 * k);
        }
#pragma unroll
        for (int e = 0; e < Q; e++) {
            const Cplx f = v[e], g = v[e + Q], h = v[e + 2 * Q];
            const Cplx s{g.re + h.re, g.im + h.im}, d{g.re - h.re, g.im - h.im};
            const double tr = fma(-0.5, s.re, f.re), ti = fma(-0.5, s.im, f.im);
            v[e] = Cplx{f.re + s.re, f.im + s.im};
            const Cplx b{fma(H, d.im, tr), fma(-H, d.re, ti)}, c{fma(-H, d.im, tr), fma(H, d.re, ti)};
            v[e + Q] = Cplx{fma(b.re, w[0].re, b.im * w[0].im), fma(b.im, w[0].re, -(b.re * w[0].im))};
            v[e + 2 * Q] = Cplx{fma(c.re, w[1].re, c.im * w[1].im), fma(c.im, w[1].re, -(c.re * w[1].im))};
        }
    } else {
        inv_group<R>(v, c_first.r[MOD]);
    }
}

template <class F, int R>
__device__ __forceinline__ void load_roots(Cplx *tw, const Cplx *tab, int nodes, int node) {
#pragma unroll
    for (int q = 0; q < R / 2; q++) tw[q] = F::RES ? tab[q * nodes + node] : ldg(tab + q * nodes + node);
}

// One pass of radix R over the C points in A: NODES nodes of C / NODES
// points, element stride SUB.  ALL: the next pass is not the team's own.
template <class F, int R, int NODES, bool INV, bool ALL>
__device__ __forceinline__ void pass(Cplx *A, const Cplx *tab) {
    constexpr int SUB = F::C / NODES / R, G = F::C / R / F::TEAMS;  // groups of a team
    const int g0 = ((int)threadIdx.x / F::TT) * G;
#pragma unroll 1
    for (int i = (int)threadIdx.x % F::TT; i < G; i += F::TT) {
        const int g = g0 + i;
        const int node = g / SUB, j0 = g % SUB, base = node * (R * SUB) + j0;
        Cplx tw[R / 2], v[R];
        load_roots<F, R>(tw, tab, NODES, node);
#pragma unroll
        for (int e = 0; e < R; e++) v[e] = A[padx<F>(base + e * SUB)];
        if constexpr (INV) inv_group<R>(v, tw);
        else fwd_group<R>(v, tw);
#pragma unroll
        for (int e = 0; e < R; e++) A[padx<F>(base + e * SUB)] = v[e];
    }
    if (ALL) cta_sync<F>();
    else team_sync<F>();
}

enum MidOp { MID_STORE_SQ, MID_STORE_MUL, MID_STORE, MID_SQ, MID_MUL, MID_MULADD };

// The last forward pass, the pointwise operation and the first inverse pass
// on groups of RM consecutive points.  Spectra outside A are laid out
// [element][group], so a warp reads and writes them contiguously, and S is
// read back by the thread that wrote it.
// G may have been written earlier in the launch, by the same thread; res: it
// is in shared memory.
//   MID_STORE_SQ, MID_STORE_MUL, MID_STORE: S <- v^2, v G, v; no inverse
//   MID_SQ: v^2    MID_MUL: v G    MID_MULADD: v G + S
template <class F>
__device__ __forceinline__ void mid(Cplx *A, const Cplx *tab, int op, const Cplx *Gs, Cplx *S, bool res = false) {
    constexpr int R = F::RM, G = F::C / R, GT = G / F::TEAMS;
    const int g0 = ((int)threadIdx.x / F::TT) * GT;
#pragma unroll 1
    for (int i = (int)threadIdx.x % F::TT; i < GT; i += F::TT) {
        const int g = g0 + i;
        Cplx tw[R / 2], v[R];
        load_roots<F, R>(tw, tab, G, g);
        const int base = padx<F>(g * R);
#pragma unroll
        for (int e = 0; e < R; e++) v[e] = A[R <= (1 << F::PADL) ? base + e : padx<F>(g * R + e)];
        fwd_group<R>(v, tw);
        if (op == MID_MUL || op == MID_MULADD || op == MID_STORE_MUL) {
#pragma unroll
            for (int e = 0; e < R; e++) {
                const Cplx c = res ? Gs[e * G + g] : ldcg(Gs + e * G + g);
                Cplx s{0.0, 0.0};
                if (op == MID_MULADD) s = F::SQS ? S[e * G + g] : ldcg(S + e * G + g);
                const double re = fma(v[e].re, c.re, fma(-v[e].im, c.im, s.re));
                const double im = fma(v[e].re, c.im, fma(v[e].im, c.re, s.im));
                v[e].re = re;
                v[e].im = im;
            }
        } else if (op == MID_STORE) {
#pragma unroll
            for (int e = 0; e < R; e++) S[e * G + g] = v[e];
            continue;
        } else {
#pragma unroll
            for (int e = 0; e < R; e++) {
                const double re = fma(v[e].re, v[e].re, -(v[e].im * v[e].im));
                const double im = (v[e].re + v[e].re) * v[e].im;
                v[e].re = re;
                v[e].im = im;
            }
        }
        if (op == MID_STORE_SQ || op == MID_STORE_MUL) {
#pragma unroll
            for (int e = 0; e < R; e++) S[e * G + g] = v[e];
            continue;
        }
        inv_group<R>(v, tw);
#pragma unroll
        for (int e = 0; e < R; e++) A[R <= (1 << F::PADL) ? base + e : padx<F>(g * R + e)] = v[e];
    }
    if (op == MID_STORE_SQ || op == MID_STORE_MUL || op == MID_STORE) cta_sync<F>();
    else team_sync<F>();
}

// ---- one candidate's working set -------------------------------------------
struct View {
    Cplx *A;       // points, padded
    Cplx *S;       // a spectrum, [element][group]
    int *xs;       // limbs of x, [half][e][thread]: n words, each thread its own
    int *bnd;      // carries between warps
    uint32_t *sc;  // scratch words of the carry scan and of votes
    Cplx *res;     // RES: roots, then the spectra of N'' and N
};

// sq (C points), xs (n limbs): where S and xs lie when they are not in shared
// memory: the candidate's own, so that launches which overlap, on other
// candidates as the locks see to, share nothing.
template <class F>
__device__ __forceinline__ void carve(unsigned char *raw, Cplx *sq, int *xs, View &w) {
    w.A = reinterpret_cast<Cplx *>(raw);
    raw += (size_t)F::A_PTS * 16;
    if (F::SQS) {
        w.S = reinterpret_cast<Cplx *>(raw);
        raw += (size_t)F::C * 16;
    } else {
        w.S = sq;
    }
    w.res = reinterpret_cast<Cplx *>(raw);
    if (F::RES) raw += (size_t)(2 * F::C + F::ROOTS) * 16;
    if (F::XSS) {
        w.xs = reinterpret_cast<int *>(raw);
        raw += (size_t)F::C * 8;
    } else {
        w.xs = xs;
    }
    w.bnd = reinterpret_cast<int *>(raw);
    raw += (size_t)2 * F::WARPS * F::R1 * 8;
    w.sc = reinterpret_cast<uint32_t *>(raw);
}

// This thread's group of the first pass.
template <class F>
__device__ __forceinline__ int tid1() {
    return F::T1 == F::T ? (int)threadIdx.x : (int)threadIdx.x & (F::T1 - 1);
}

// The roots (and with nn, nh the spectra) in shared memory, where the class
// keeps them there: tab, nn and nh then point to the copies.
template <class F>
__device__ __forceinline__ void resident(const View &w, Tab &tab, const Cplx *&nn, const Cplx *&nh) {
    if (!F::RES) return;
    const Cplx *src = tab.t[0][0];
    for (int i = threadIdx.x; i < F::ROOTS; i += F::T) w.res[i] = ldg(src + i);
    if (nn)
        for (int i = threadIdx.x; i < F::C; i += F::T) {
            w.res[F::ROOTS + i] = ldg(nn + i);
            w.res[F::ROOTS + F::C + i] = ldg(nh + i);
        }
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int p = 0; p < 3; p++) tab.t[m][p] = w.res + (tab.t[m][p] - src);
    nn = w.res + F::ROOTS;
    nh = nn + F::C;
    cta_sync<F>();
}

// First forward pass from the limbs in registers: modulus MOD (0: B^n + 1,
// 1: M2), into A.
template <class F, int MOD>
__device__ __forceinline__ void first_pass(Cplx *A, const int *lo, const int *hi) {
    Cplx v[F::R1];
#pragma unroll
    for (int e = 0; e < F::R1; e++) {
        const double a = to_double(lo[e]), c = to_double(hi[e]);
        if (MOD == 0) {
            v[e].re = a;
            v[e].im = c;
        } else {
            v[e].re = fma(-0.5, c, a);
            v[e].im = 0.86602540378443864676 * c;
        }
    }
    fwd_first<F::R1, MOD>(v);
#pragma unroll
    for (int e = 0; e < F::R1; e++) A[padx<F>(tid1<F>() + e * F::T1)] = v[e];
    cta_sync<F>();
}

// Carries of every limb to the next one: k in, the neighbour's carry out.
// Limb order: thread t + T1 e, then the second half; the carry out of the top
// limb comes back negated (B^n = -1), modulo M2 at limbs 0 and n/2.
template <class F, int MOD>
__device__ __forceinline__ void exchange(int *kl, int *kh, int *buf) {
    constexpr int R = F::R1;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if constexpr (F::WARPS > 1) {
        if (lane == 31) {
#pragma unroll
            for (int e = 0; e < R; e++) {
                buf[(warp * R + e) * 2] = kl[e];
                buf[(warp * R + e) * 2 + 1] = kh[e];
            }
        }
        __syncthreads();
    }
    [[maybe_unused]] const int wl = kl[R - 1], wh = kh[R - 1];  // the top limbs' carries
    // descending e: the first thread takes the last thread's carry of e - 1
#pragma unroll
    for (int e = R - 1; e >= 0; e--) {
        int pl, ph;
        if constexpr (F::WARPS > 1) {
            pl = __shfl_up_sync(FULL, kl[e], 1);
            ph = __shfl_up_sync(FULL, kh[e], 1);
            if (lane == 0) {
                const int at = warp ? (warp - 1) * R + e : (F::WARPS - 1) * R + (e ? e - 1 : R - 1);
                pl = buf[at * 2];
                ph = buf[at * 2 + 1];
            }
        } else {
            constexpr int M = F::T1 - 1;  // T1 = 32 or 16 lanes in a ring
            const int from = (lane & ~M) | ((lane + M) & M);
            pl = (lane & M) != M ? kl[e] : (e ? kl[e ? e - 1 : 0] : wl);
            ph = (lane & M) != M ? kh[e] : (e ? kh[e ? e - 1 : 0] : wh);
            pl = __shfl_sync(FULL, pl, from);
            ph = __shfl_sync(FULL, ph, from);
        }
        if (e == 0 && tid1<F>() == 0) {
            const int tl = pl, th = ph;
            pl = -th;
            ph = MOD == 0 ? tl : tl - th;
        }
        kl[e] = pl;
        kh[e] = ph;
    }
}

// Two more local carry steps after the carries k of the first split: limbs
// of at most B/2 + 40 in magnitude.
template <class F, int MOD>
__device__ __forceinline__ void settle(const View &w, int b, int *kl, int *kh, int *lo, int *hi) {
    constexpr int R = F::R1;
    const int mask = (1 << b) - 1, half = 1 << (b - 1);
    exchange<F, MOD>(kl, kh, w.bnd);
#pragma unroll
    for (int turn = 1; turn <= 2; turn++) {
#pragma unroll
        for (int e = 0; e < R; e++) {
            const int cl = lo[e] + kl[e] + half, ch = hi[e] + kh[e] + half;
            kl[e] = cl >> b;
            kh[e] = ch >> b;
            lo[e] = (cl & mask) - half;
            hi[e] = (ch & mask) - half;
        }
        exchange<F, MOD>(kl, kh, w.bnd + (turn & 1) * 2 * F::WARPS * R);
    }
#pragma unroll
    for (int e = 0; e < R; e++) {
        lo[e] += kl[e];
        hi[e] += kh[e];
    }
}

// Last inverse pass, rounding and carries: the C points in A to limbs, times
// two when dbl.  MOD 1: the value found is that of the points divided by R'.
template <class F, int MOD>
__device__ __forceinline__ void last_pass(const View &w, int b, int dbl, int *lo, int *hi) {
    constexpr int R = F::R1;
    constexpr double S0 = 1.0 / F::C;
    const int mask = (1 << b) - 1, half = 1 << (b - 1), bs = b - dbl;
    // 1.5 2^52 + B/2 (B/4 when doubled): the sum's low 51 bits are the rounded
    // coefficient plus that offset
    const double magic = 6755399441055744.0 + (double)(half >> dbl);
    int kl[R], kh[R];
    {
        Cplx v[R];
#pragma unroll
        for (int e = 0; e < R; e++) v[e] = w.A[padx<F>(tid1<F>() + e * F::T1)];
        inv_last<R, MOD>(v);
#pragma unroll
        for (int e = 0; e < R; e++) {
            long long ql, qh;
            if (MOD == 0) {
                ql = bits_of(fma(v[e].re, S0, magic));
                qh = bits_of(fma(v[e].im, S0, magic));
            } else {
                // u + w v = re + i im: v = 2/sqrt(3) im, u = re + v / 2; times
                // (1 + y) with y^2 = -y - 1: (u - v) + u y
                const double h = v[e].im * 0.57735026918962576451;  // v / 2
                ql = bits_of(fma(v[e].re - h, S0, magic));
                qh = bits_of(fma(v[e].re + h, S0, magic));
            }
            ql -= 0x4338000000000000ll;
            qh -= 0x4338000000000000ll;
            kl[e] = (int)(ql >> bs);
            kh[e] = (int)(qh >> bs);
            lo[e] = (int)(((unsigned)ql << dbl) & (unsigned)mask) - half;
            hi[e] = (int)(((unsigned)qh << dbl) & (unsigned)mask) - half;
        }
    }
    settle<F, MOD>(w, b, kl, kh, lo, hi);
}

// The passes between the first and the middle one.
template <class F>
__device__ __forceinline__ void fwd_inner(Cplx *A, const Cplx *const *t) {
    pass<F, F::R2, F::R1, false, false>(A, t[0]);
    if constexpr (F::NPASS == 4) pass<F, F::R3, F::R1 * F::R2, false, false>(A, t[1]);
}
template <class F>
__device__ __forceinline__ void inv_inner(Cplx *A, const Cplx *const *t) {
    if constexpr (F::NPASS == 4) pass<F, F::R3, F::R1 * F::R2, true, false>(A, t[1]);
    pass<F, F::R2, F::R1, true, true>(A, t[0]);
}

// x's limbs as the last step found them.
template <class F>
__device__ __forceinline__ void load_x(const View &w, int *lo, int *hi) {
#pragma unroll
    for (int e = 0; e < F::R1; e++) {
        lo[e] = w.xs[e * F::T1 + tid1<F>()];
        hi[e] = w.xs[F::C + e * F::T1 + tid1<F>()];
    }
}

// One Montgomery step on the limbs (lo, hi) of x (mod N; times two when dbl):
//   square: x <- x^2 / R', or x y / R' given y's spectra (2 C points: modulo
//   B^n + 1, then M2)    else: x <- x / R'
// nn, nh: spectra of N'' (modulo B^n + 1) and N (modulo M2), from resident().
template <class F>
__device__ __forceinline__ void step(const View &w, const Tab &tab, const Cplx *nn, const Cplx *nh, int b,
                                     bool square, int dbl, int *lo, int *hi, const Cplx *y = nullptr) {
    constexpr int R = F::R1, MT = F::NPASS - 2;
#pragma unroll
    for (int e = 0; e < R; e++) {
        w.xs[e * F::T1 + tid1<F>()] = lo[e];
        w.xs[F::C + e * F::T1 + tid1<F>()] = hi[e];
    }
    // phases: 0 spectrum of x (of its square, of x y) modulo M2 into S, 1 D, 2 m, 3 U
#pragma unroll 1
    for (int ph = 0; ph < 4; ph++) {
        if (ph == 1 && !square) continue;  // D = x
        const int mod = (ph == 0 || ph == 3) ? 1 : 0;
        if (mod) first_pass<F, 1>(w.A, lo, hi);
        else first_pass<F, 0>(w.A, lo, hi);
        const Cplx *t[3] = {mod ? tab.t[1][0] : tab.t[0][0], mod ? tab.t[1][1] : tab.t[0][1],
                            mod ? tab.t[1][2] : tab.t[0][2]};
        fwd_inner<F>(w.A, t);
        const int op = ph == 0 ? (!square ? MID_STORE : (y ? MID_STORE_MUL : MID_STORE_SQ))
                               : (ph == 1 ? (y ? MID_MUL : MID_SQ) : (ph == 2 ? MID_MUL : MID_MULADD));
        mid<F>(w.A, t[MT], op, ph == 0 ? y + F::C : (ph == 1 ? y : (ph == 2 ? nn : nh)), w.S,
               F::RES && ph >= 2);
        if (ph == 0) {
            load_x<F>(w, lo, hi);
            continue;
        }
        inv_inner<F>(w.A, t);
        if (mod) last_pass<F, 1>(w, b, dbl, lo, hi);
        else last_pass<F, 0>(w, b, 0, lo, hi);
    }
}

// lo, hi <- limbs + c (ylo, yhi), carried locally; |c| < 2^16, and the value
// stays below B^n / 4.
template <class F>
__device__ void add_mul(const View &w, int b, int c, const int *ylo, const int *yhi, int *lo, int *hi) {
    constexpr int R = F::R1;
    const int mask = (1 << b) - 1, half = 1 << (b - 1);
    int kl[R], kh[R];
#pragma unroll
    for (int e = 0; e < R; e++) {
        const long long ql = lo[e] + (long long)c * ylo[e] + half, qh = hi[e] + (long long)c * yhi[e] + half;
        kl[e] = (int)(ql >> b);
        kh[e] = (int)(qh >> b);
        lo[e] = (int)(ql & mask) - half;
        hi[e] = (int)(qh & mask) - half;
    }
    cta_sync<F>();
    settle<F, 0>(w, b, kl, kh, lo, hi);
}

// This thread's limbs from an array of n words written earlier in the launch.
template <class F>
__device__ __forceinline__ void get_limbs(const uint32_t *src, int *lo, int *hi) {
#pragma unroll
    for (int e = 0; e < F::R1; e++) {
        lo[e] = (int)__ldcg(src + tid1<F>() + e * F::T1);
        hi[e] = (int)__ldcg(src + F::C + tid1<F>() + e * F::T1);
    }
}

// ---- canonical form --------------------------------------------------------
// Carry function of a run of limbs, (f(-1), f(0), f(1)) + 1 in two bits each.
__device__ __forceinline__ uint32_t fn_at(uint32_t f, uint32_t c) { return (f >> (2u * c)) & 3u; }
__device__ __forceinline__ uint32_t fn_then(uint32_t f, uint32_t g) {  // g after f
    return fn_at(g, fn_at(f, 0u)) | (fn_at(g, fn_at(f, 1u)) << 2) | (fn_at(g, fn_at(f, 2u)) << 4);
}

// Where limb i lies in such an array: a thread's run of n / T limbs is followed
// by one unused word, so that the runs of a warp start in different banks.
template <class F>
__device__ __forceinline__ int lpos(int i) {
    return i + i / (F::N / F::T);
}

// The n limbs L (at lpos; each within (-3B/4, 2B)) to digits in [0, B); returns the carry
// out of the top limb (-1: the number is negative).
template <class F>
__device__ int normalize(int *L, int b, uint32_t *sc) {
    constexpr int W = F::N / F::T;
    const unsigned FULL = 0xffffffffu;
    const int mask = (1 << b) - 1, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    int c = 0;
    bool zero = true, ones = true;
    for (int q = 0; q < W; q++) {
        const int v = L[t * (W + 1) + q] + c, d = v & mask;
        c = v >> b;
        L[t * (W + 1) + q] = d;
        zero = zero && d == 0;
        ones = ones && d == mask;
    }
    uint32_t f = (uint32_t)(c + 1 - (zero ? 1 : 0)) | ((uint32_t)(c + 1) << 2) | ((uint32_t)(c + 1 + (ones ? 1 : 0)) << 4);
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t g = __shfl_up_sync(FULL, f, o);
        if (lane >= o) f = fn_then(g, f);
    }
    if (lane == 31) sc[warp] = f;
    cta_sync<F>();
    uint32_t cin = 1u;  // carry + 1 into this warp
    for (int v = 0; v < warp; v++) cin = fn_at(sc[v], cin);
    uint32_t tot = 1u;
    for (int v = 0; v < F::WARPS; v++) tot = fn_at(sc[v], tot);
    const uint32_t before = __shfl_up_sync(FULL, f, 1);
    int carry = (int)(lane ? fn_at(before, cin) : cin) - 1;
    for (int q = 0; q < W && carry; q++) {
        const int v = L[t * (W + 1) + q] + carry;
        carry = v >> b;
        L[t * (W + 1) + q] = v & mask;
    }
    cta_sync<F>();
    return (int)tot - 1;
}

// This thread's limbs to and from an array of n words.
template <class F, class W>
__device__ __forceinline__ void put_limbs(W *L, const int *lo, const int *hi) {
#pragma unroll
    for (int e = 0; e < F::R1; e++) {
        L[tid1<F>() + e * F::T1] = (W)lo[e];
        L[F::C + tid1<F>() + e * F::T1] = (W)hi[e];
    }
}

// L (at lpos) <- the canonical digits (base B) of the value of the limbs modulo
// N, for a value in (-N, N); nl: N's digits.  L overlays A.
template <class F>
__device__ void to_digits(const View &w, int b, const uint32_t *nl, const int *lo, const int *hi, int *L) {
    cta_sync<F>();
#pragma unroll
    for (int e = 0; e < F::R1; e++) {
        L[lpos<F>(tid1<F>() + e * F::T1)] = lo[e];
        L[lpos<F>(F::C + tid1<F>() + e * F::T1)] = hi[e];
    }
    cta_sync<F>();
    if (normalize<F>(L, b, w.sc) < 0) {
        for (int i = threadIdx.x; i < F::N; i += F::T) L[lpos<F>(i)] += (int)nl[i];
        cta_sync<F>();
        normalize<F>(L, b, w.sc);
    }
}

// Block-wide AND of a vote.
template <class F>
__device__ __forceinline__ bool vote_and(bool v) {
    return __syncthreads_and(v ? 1 : 0) != 0;
}

// Balanced limbs (|limb| <= B/2) from canonical digits d(i), at the positions
// of this thread; a carry out of the top limb wraps to -1 at limb 0 (B^n =
// -1; it cannot happen for a number below B^n / 2).
template <class F, class Digit>
__device__ __forceinline__ void balanced(Digit d, int b, int *lo, int *hi) {
    const int B = 1 << b, half = B >> 1;
    auto at = [&](int i) {
        const int v = (int)d(i);
        const int top = (int)d(i ? i - 1 : F::N - 1) >= half ? 1 : 0;
        return (v >= half ? v - B : v) + (i ? top : -top);
    };
#pragma unroll
    for (int e = 0; e < F::R1; e++) {
        lo[e] = at(tid1<F>() + e * F::T1);
        hi[e] = at(F::C + tid1<F>() + e * F::T1);
    }
}

// out <- the spectrum (modulus mod) of the limbs, [element][group].
template <class F>
__device__ void spectrum(const View &w, const Tab &tab, int mod, const int *lo, const int *hi, Cplx *out) {
    const Cplx *t[3] = {tab.t[mod][0], tab.t[mod][1], tab.t[mod][2]};
    if (mod) first_pass<F, 1>(w.A, lo, hi);
    else first_pass<F, 0>(w.A, lo, hi);
    fwd_inner<F>(w.A, t);
    mid<F>(w.A, t[F::NPASS - 2], MID_STORE, nullptr, out);
}

}  // namespace fp
}  // namespace mr
}  // namespace pfb
