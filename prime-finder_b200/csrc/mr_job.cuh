// The per-candidate state that the engine's kernels and its host side share.
#pragma once
#include <stdint.h>

namespace pfb {
namespace mr {

// State of one candidate in device memory.
struct JobDev {
    uint32_t *x;          // H limbs: Montgomery residue (working value)
    uint32_t *res;        // H limbs: canonical residue a^E mod N (output)
    uint32_t *nn;         // [2][H] negacyclic NTT_H(N''), N'' = -N^-1 mod (B^H + 1)
    uint32_t *nh;         // [2][H] NTT_H(N)
    const uint32_t *npl;  // H limbs of N'' (set-up input)
    const uint32_t *nl;   // H limbs of N
    const uint32_t *exp;  // exponent, 32-bit words, little-endian
    uint32_t *ybuf;       // H + H/32 words (L = 2^15 only: the residue Y, padded)
    struct LucasDev *lucas;  // strong Lucas test (mode 2) only
    int logl;
    int cursor;   // next exponent bit (MSB first); phase 0 while >= 0
    int extra;    // squarings left in phase 2 (s - 1 for a strong test)
    int phase;    // 0 exponent loop, 1 first check, 2 squarings r < s, 3 done
    uint32_t base;
    int mode;     // 0 modular power only, 1 strong test, 2 strong Lucas test
    int verdict;  // 1 probable prime, 0 composite
    int steps;    // steps taken (diagnostics)
    // floating-point engine (fft_device.cuh): its length class + 1, else 0;
    // bits of a limb.  Then x, res, npl, nl hold 2 C words (x signed limbs,
    // the others digits), nn and nh C complex points.
    int fpc;
    int fbits;
    uint32_t *sq;  // x^2's spectrum of the classes that keep it in global memory (C points)
};

// Strong Lucas state of one candidate: H limbs each, Montgomery form: V_k,
// V_(k+1), Q^k, a product, R mod N; gy the [2][L] spectrum of V_(k+1)
// (floating-point engine: its two spectra, 2 C points).
struct LucasDev {
    uint32_t *lv0, *lv1, *lqk, *lt, *lone, *gy;
    int q;        // Selfridge Q = (1 - D) / 4
    uint32_t lb;  // every stored value is < lb * N
};

// Operations of the modular context (pfb_mr_ctx_*).
enum CtxOp : int {
    CTX_MODSQ = 0,    // out = REDC(A^2)         (working form in, working form out)
    CTX_MODMUL = 1,   // out = REDC(A B)
    CTX_RAW_SQ = 2,   // out = A^2, n_sum limbs  (no reduction)
    CTX_RAW_MUL = 3,  // out = A B, n_sum limbs
    CTX_FROM = 4,     // out = A R^-1 mod N      (working form -> plain residue)
};

// Per-modulus buffers beyond the engine's own (JobDev: spectra of N' and N,
// limbs of N, spill buffers of the longest transform).
struct CtxExtra {
    uint32_t *gy;              // [2][L] spectrum of the second factor
    uint32_t *yl;              // H limbs of the second factor
    unsigned long long *raw;   // L coefficients of a raw product
    uint32_t *ys;              // floating-point engine: spectra of the second factor, 2 C points (over gy and raw)
};

}  // namespace mr
}  // namespace pfb
