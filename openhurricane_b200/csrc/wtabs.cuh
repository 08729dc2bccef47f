// Mechanism tables of the warp-per-cell (wcell.cuh, kernel 6) and
// segment-per-cell (scell.cuh, kernel 7) integrators, mechanisms of
// N = nsp + 1 <= 16 unknowns; packed on the host by pack_w (capi.cu).
#pragma once

#include "integrator.cuh"
#include "t3_base.cuh"

namespace hc {

// reaction fields of WMech::rd (doubles) and ::ri (ints), field-major over reactions
enum WRD : int {
    kWA = 0, kWb, kWTa, kWA0, kWb0, kWTa0, kWalpha, kWiTsss, kWiTs, kWTss, kWTsss, kWTs, kWs,
    kWnu,                      // nu[8]: -fnu (reactants) then +bnu (products)
    kWord = kWnu + 8,          // ord[8]
    kWRDn = kWord + 8
};
// kWxj: the reaction's first extra exponential job (fall-off: k0, then the Troe
// centering terms exp(-T/T***), exp(-T/T*), exp(-T**/T))
enum WRI : int { kWtype = 0, kWrev, kWnf, kWnb, kWxj, kWidx, kWRIn = kWidx + 8 };
// species fields of WMech::th, field-major over 32 species slots
enum WTH : int {
    kWtl = 0, kWtc, kWth,
    kWrange = 3,               // then 2 ranges of 21: h[5], h5, s0, s[4], s6, cp[5], dcp[4]
    kWRangeN = 21,
    kWW = kWrange + 2 * kWRangeN,   // molecular weight
    kWTHn = kWW + 1
};

// Reactions come in rounds of 32 (reaction r = 32 * round + slot); the
// reaction tables and the records are round-major, [round][field][32], so
// that lane `slot` reads field f of its reaction at a fixed offset.
// Exponential jobs (round-major [round][3][32]: alpha, beta, gamma): job j
// is exp(alpha ln T + beta / T + gamma T); job r < nrc is reaction r's
// Arrhenius factor, the fall-off reactions' extra terms follow.
struct WMech {
    int32_t nsp, nrc, nrc32, ntb, nent, njob, njob32;
    const double *xj;     // [njob32 / 32][3][32]
    const double *th;     // [kWTHn][32]
    const double *rd;     // [nrc32 / 32][kWRDn][32]
    const int32_t *ri;    // [nrc32 / 32][kWRIn][32]
    const double *eff;    // [nrc][nsp] efficiencies (third-body / fall-off rows)
    const int32_t *lptr;  // [nsp + 1] participation lists of the species
    const int32_t *lent;  // [3 * nent] per entry: reaction | pos << 16 | np << 20 | third-body << 24,
                          // then the participants' columns packed 8 bits each (two words)
    const double *lnu;    // [nent] the species' signed coefficient in the entry's reaction
    const int32_t *tbl;   // [ntb] third-body / fall-off reactions
    const double *raw;    // [nsp][2][7] mass-basis NASA-7 (out-of-range forms)
    double glim;          // |G0/(Ru T)| bound of the product form of 1/Kc
    // kernel 6 only: two words per reaction of the direct form (kWX*, round-major
    // [round][2][32]) and the species' participation lists in lock step,
    // [gE][16] reaction slots and signed coefficients (zero past a list's end)
    int32_t gE;
    const int32_t *rx;
    const int32_t *gslot;
    const double *gnu;
};

// WMech::rx word 0: the species of up to three unit-order factors a side (4
// bits each, kWOne where there is none), whether the reaction needs the
// general form, is reversible, its change in moles + 1, and the multiplicity
// of each side's first factor; word 1: the column (5 bits) that each factor's
// derivative goes to (N + 1, which nothing reads, for none)
enum WRX : int {
    kWXf = 0, kWXb = 12, kWXgeneral = 24, kWXrev = 25, kWXs = 26, kWXmf = 28, kWXmb = 30
};
constexpr int kWOne = 15;   // the species slot that holds c = 1, exp(+-g) = 1, h = cp = 0

// parts that kernel 6 splits a sum over the reactions into (one lane each)
__host__ __device__ constexpr int w_parts(int N) { return N <= 10 ? 2 : 1; }

constexpr int kWRec = 12;   // kernel 7's record: q, dq/dT, g, dH, d[8]

// the mechanism tables as copied into the block's shared memory
struct WTabs {
    const double *th, *rd, *eff, *lnu, *xj;
    const int32_t *ri, *lptr, *lent, *tbl;
};

// shared memory of the block's table copy (bytes, 8-byte aligned parts)
__host__ __device__ inline size_t w_tables_bytes(int nsp, int nrc, int nrc32, int nent, int ntb, int njob32) {
    const size_t d = (size_t)kWTHn * 32 + (size_t)kWRDn * nrc32 + (size_t)(nrc > 0 ? nrc : 1) * nsp + nent +
                     3 * (size_t)njob32;
    const size_t i = (size_t)kWRIn * nrc32 + (nsp + 1) + 3 * (size_t)nent + (ntb > 0 ? ntb : 1);
    return sizeof(double) * d + ((sizeof(int32_t) * i + 7) & ~(size_t)7);
}

}  // namespace hc
