// Host construction of the roots of the floating-point transforms
// (fft_device.cuh): plain host computations, so that the same tables can be
// built where no GPU is present.
#pragma once
#include <math.h>
#include <stdint.h>

#include <vector>

#include "fft_device.cuh"

namespace pfb {
namespace mr {
namespace fp {

// Angles are kept as integers in units of a full turn / kTurn, which every
// halving below divides exactly.
constexpr long long kTurn = 36ll << 34;

// e^(2 pi i num / kTurn), each part correctly rounded but for the rare tie
// of the extended-precision value; the argument is reduced to an eighth turn.
inline Cplx unit_root(long long num) {
    num %= kTurn;
    if (num < 0) num += kTurn;
    const int oct = (int)(8 * num / kTurn);
    long long r = num - (long long)oct * (kTurn / 8);
    if (oct & 1) r = kTurn / 8 - r;
    const long double a = 6.283185307179586476925286766559L * (long double)r / (long double)kTurn;
    long double c = cosl(a), s = sinl(a);
    static const int swap[8] = {0, 1, 1, 0, 0, 1, 1, 0}, sc[8] = {1, 1, -1, -1, -1, -1, 1, 1},
                     ss[8] = {1, 1, 1, 1, -1, -1, -1, -1};
    if (swap[oct]) {
        const long double t = c;
        c = s;
        s = t;
    }
    return Cplx{(double)(sc[oct] * c), (double)(ss[oct] * s)};
}

// Angle (in turns / kTurn) of the root r of node `node` at level `lv` of the
// tree of y^C - e^(i phi0): half the node's own angle.
inline long long node_angle(long long phi0, int lv, long long node) {
    long long phi = phi0;
    for (int d = lv - 1; d >= 0; d--) phi = phi / 2 + (((node >> d) & 1) ? kTurn / 2 : 0);
    return phi / 2;
}

// Root angle of the moduli: y^C = i (B^n + 1), y^C = e^(2 pi i / 3) (M2).
inline long long top_angle(int mod) { return mod ? kTurn / 3 : kTurn / 4; }

// The roots of a radix-R group at node `node` of (binary) level `lv` under
// the angle phi0.
inline Cplx group_root(long long phi0, int lv, long long node, int q) {
    int s = 0;
    while (q >= (1 << s)) s++;  // q = 0: level 0; else q in [2^(s-1), 2^s): level s
    const int u = s ? q - (1 << (s - 1)) : 0;
    return unit_root(node_angle(phi0, lv + s, (node << s) + 2 * u));
}

// Angle of child k of the ternary level at the root of the tree.
inline long long child_angle(int mod, int k) { return top_angle(mod) / 3 + kTurn / 3 * k; }

inline First first_roots() {
    First f{};
    for (int mod = 0; mod < 2; mod++) {
        for (int q = 0; q < 16; q++) f.r[mod][q] = group_root(top_angle(mod), 0, 0, q);
        f.t[mod][0] = unit_root(child_angle(mod, 0));
        f.t[mod][1] = unit_root(2 * child_angle(mod, 0));
        for (int k = 0; k < 3; k++)
            for (int q = 0; q < 4; q++) f.t[mod][2 + 4 * k + q] = group_root(child_angle(mod, k), 0, 0, q);
    }
    return f;
}

inline int ilog2(int v) {
    int l = 0;
    while ((1 << l) < v) l++;
    return l;
}

// The planes of one class: t.t[mod][pass] as offsets into the returned points.
template <class F>
std::vector<Cplx> class_roots(size_t off[2][3]) {
    std::vector<Cplx> v;
    const int radix[4] = {F::R1, F::R2, F::R3, F::R4};
    for (int mod = 0; mod < 2; mod++) {
        int nodes = F::R1;
        for (int p = 1; p < F::NPASS; p++) {
            off[mod][p - 1] = v.size();
            for (int q = 0; q < radix[p] / 2; q++)
                for (int nd = 0; nd < nodes; nd++) {
                    if (nodes % 3 == 0) {
                        const int sub = nodes / 3;
                        v.push_back(group_root(child_angle(mod, nd / sub), ilog2(sub), nd % sub, q));
                    } else {
                        v.push_back(group_root(top_angle(mod), ilog2(nodes), nd, q));
                    }
                }
            nodes *= radix[p];
        }
    }
    return v;
}

}  // namespace fp
}  // namespace mr
}  // namespace pfb
