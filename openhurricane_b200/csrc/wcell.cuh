// Warp-per-cell implicit-Euler integrator (kernel 6) for mechanisms of
// N = nsp + 1 <= 16 unknowns, FP64, constant-pressure and constant-volume
// reactors.
//
// One warp integrates one cell at a time and takes the next cell from the
// device work queue (the grid is persistent). The per-cell control flow is
// the reference's (chemistrySource.cpp:1511-1555, ImplicitEuler.cpp:101-342,
// ODEsSolver.cpp:148-225), uniform across the warp, with one evaluation site.
//
// What bounds it: a flow step lasts as long as its stiffest cell (10 to 100
// times the mean number of Newton iterations), so the time of ONE Newton
// iteration of one warp counts, a chain of dependent FP64 and shuffle
// latencies, and the instruction fetch of its code. The split below is made
// to shorten that chain and to keep the hot loop small:
//
//  * species: lane i evaluates species i (NASA-7, molar, from coefficients
//    pre-multiplied on the host); every exp(a ln T + b/T + c T) of the rate
//    laws is one batched pass, one lane each;
//  * reactions: lane r evaluates reaction r (r = lane + 32 k) without
//    loops over its participants: up to three unit-order factors
//    a side, padded with a species slot that reads 1, 1/Kc as the product of
//    the species' exp(+-G0/(Ru T)). It writes row r of the DENSE matrix
//    D[r][j] = dq_r/dc_j (third-body and fall-off rows included), dq_r/dT, q_r;
//    the columns no participant touches stay zero and are never rewritten.
//    Other orders, more factors or an out-of-range thermo take the
//    out-of-line general form;
//  * rows: W lanes share a row of the Newton matrix, lane (i, h) owns row i and
//    C columns of [I - dt J | rhs]. It walks species i's participation list
//    (all lists in lock step) and adds nu D[r][its columns] to registers: J never
//    goes through memory. The temperature row is a set of plain dot products
//    over the reactions (dH_r with each column of D), one lane each, in the
//    same loop;
//  * Gaussian elimination with partial pivoting on the registers, the right-hand
//    side along with the matrix: the pivot is the largest |a(k)| by its upper 27
//    bits (one warp max reduction of a key that carries the row; ties and
//    near-ties to the first row; the solutions' errors in the solver's norm against 80-bit
//    arithmetic are those of the full magnitudes, geometric means 2.924e-8 and 2.928e-8 over
//    6000 Newton matrices of 9 species, 1.95e-2 and 1.99e-2 over 600 of 53), every lane has the reciprocal of its own
//    candidate ready before the pivot is known, the next pivot column is updated
//    first and searched while the others follow. Then one back substitution.
//    (Gauss-Jordan would save it, 450 cycles, but is not backward stable on these
//    badly scaled matrices: the reference's step sequence came out different, with
//    2786 Newton iterations instead of 4191 on two of the 4096 Dirichlet cells);
//  * norms: warp max reductions of the bit patterns.
//
// With autoUpdateJacobian the factors stay in shared memory and an iteration that keeps the
// Jacobian sums f alone and substitutes. That is a build of its own: as an option of one
// build it made every iteration 6 % longer, and before the factors were kept it saved nothing
// (1001 Dirichlet cells at 1e-7 s, a Jacobian every ten iterations: 61.7 -> 50.2 ms).
//
// Measured (B200, 9 species / 21 reactions): one Newton iteration of the stiffest
// cell takes 4.5 us (before: 13.9 us with lane i holding row i, the reactions' lists
// walked and the LU's rows broadcast one by one). Flow steps: 4096 Dirichlet cells at
// 1e-7 s 277 -> 92 ms, 12,288 mixed cells at 1e-5 s 641 -> 335 ms, 1001 cells of the
// constant-volume reactor 684 -> 86 ms (there against the cell group).
#pragma once

#include "fastmath.cuh"
#include "stepctl.cuh"
#include "wtabs.cuh"

namespace hc {

// The block's shared memory: the tables kernel 6 copies into it, then the warps'
// parts. Everything is named by its place in it (one register instead of a
// 64-bit pointer's two, in a kernel that is short of registers).
__device__ __forceinline__ double *w_smem() {
    extern __shared__ __align__(16) double smem_w[];
    return smem_w;
}

struct WTabs6 {
    int rd, eff, gnu, xj;        // places in doubles (the species table is at 0)
    int ri, rx, gslot;           // places in 32-bit words
    __device__ __forceinline__ const double *d(int at) const { return w_smem() + at; }
    __device__ __forceinline__ const int32_t *i(int at) const { return reinterpret_cast<const int32_t *>(w_smem()) + at; }
};

__host__ __device__ inline size_t w6_tables_doubles(const WMech &m) {
    const size_t d = (size_t)kWTHn * 32 + (size_t)kWRDn * m.nrc32 + (size_t)(m.nrc > 0 ? m.nrc : 1) * m.nsp +
                     16 * (size_t)m.gE + 3 * (size_t)m.njob32;
    const size_t i = (size_t)kWRIn * m.nrc32 + 2 * (size_t)m.nrc32 + 16 * (size_t)m.gE;
    return (d + (i + 1) / 2 + 1) & ~(size_t)1;   // the warps' parts start on 16 bytes
}

template <int N>
struct WLayout {
    static constexpr int R = (N <= 10) ? 10 : 16;   // lanes (rows) of one column block
    static constexpr int W = 32 / R;                // column blocks: lanes sharing a row
    static constexpr int C = 2 * ((N + 1 + 2 * W - 1) / (2 * W));   // columns per lane (even: 16-byte loads)
    static constexpr int COLS = W * C;              // N unknowns, the right-hand side, padding
    static constexpr int LD = COLS + 2;             // row stride of D (the rows' banks spread)
    static constexpr int P = w_parts(N);            // parts of a sum over the reactions
    static constexpr int TI = N - 1;                // column of T; column N is q / the right-hand side
    static constexpr int hN = N / C, cN = N % C;    // owner and place of column N
    static_assert(N + 1 < COLS + 1 && P * (N + 2) + 2 <= 32, "layout");
    // per-warp shared memory (doubles)
    static constexpr int kA1 = 0;                   // {c, h} of 16 species slots
    static constexpr int kA2 = 32;                  // {exp(-g), cp}
    static constexpr int kA3 = 64;                  // {exp(g), cp}
    static constexpr int kY = 96, kCP = 112, kDCP = 128;   // y, cp (cv) and dcp/dT
    static constexpr int kG = 144;                  // g, dG/dT - G/T
    static constexpr int kTS = 176;                 // the dot products
    static constexpr int kDH = 208;                 // dH_r (dE_r) [nrc32], then dCp_r, the exponentials, D
    __host__ __device__ static size_t doubles(int nrc, int nrc32, int njob32) {
        return (size_t)kDH + 2 * nrc32 + njob32 + (size_t)LD * (nrc > 0 ? nrc : 1);
    }
    // autoUpdateJacobian's factors behind it: U, then the multipliers by row (odd strides)
    static constexpr int kLU = COLS + 1, kLM = N + 1, kFactors = N * (kLU + kLM);
};

// One reaction in the general form (any orders, up to four participants a
// side, and the clamped equilibrium constant when `slow`): row r of D by
// accumulation, dH and dCp. reactionTypes q / Kc / DqDci / DqDT
// (reactionTypes.cpp:178-445, 843-876), unimolecularFallOffRR, fallOffFunctions.
template <int N>
static __device__ HC_NOINLINE void w_reaction_general(double *s, const double *x, const int32_t *xi, const double *er,
                                                      int nsp, double T, double logT, double invT, double invRuT,
                                                      bool slow, const double *cM, double kx, const double *X,
                                                      double cvRu, double *D, double *dHp, double *dCp) {
    using L = WLayout<N>;
    auto cc = [s](int i) { return s[L::kA1 + 2 * i]; };
    const int type = xi[kWtype * 32], rev = xi[kWrev * 32], nf = xi[kWnf * 32], nb = xi[kWnb * 32];
    double pf[kMaxSide], pb[kMaxSide];
#pragma unroll
    for (int k = 0; k < kMaxSide; ++k) {
        pf[k] = (k < nf) ? conc_pow(cc(xi[(kWidx + k) * 32]), x[(kWord + k) * 32]) : 1.0;
        pb[k] = (k < nb) ? conc_pow(cc(xi[(kWidx + nf + k) * 32]), x[(kWord + nf + k) * 32]) : 1.0;
    }
    double M = 0.0;
    if (type != kArrhenius)
        for (int j = 0; j < nsp; ++j) M += er[j] * cM[j * (cM == s + L::kA1 ? 2 : 1)];
    const double b = x[kWb * 32], Ta = x[kWTa * 32];
    double kf, k0 = 0.0, Pr = 0.0, Ff = 1.0, logPr = 0.0;
    T3Cent cent{0.0, 0.0};
    if (type == kArrhenius) {
        kf = kx;
    } else if (type == kThirdBody) {
        kf = M * kx;
    } else {
        const int xj = xi[kWxj * 32];
        k0 = x[kWA0 * 32] * X[xj];
        Pr = fdiv(k0, notZeroD(kx)) * M;
        if (type != kLindemann) {
            cent = t3_troe_cent(type == kTroe4, x[kWalpha * 32], x[kWiTsss * 32], x[kWiTs * 32], x[kWTss * 32],
                                X[xj + 1], X[xj + 2], (type == kTroe4) ? X[xj + 3] : 0.0, invT);
            logPr = log10(hmax(Pr, kTiny));
            Ff = t3_troe_F(cent.lf, logPr);
        }
        kf = kx * (Pr / (1.0 + Pr)) * Ff;
    }
    double dH = 0.0, dC = 0.0;
    for (int k = 0; k < nf + nb; ++k) {
        const double nu = x[(kWnu + k) * 32];
        const int i = xi[(kWidx + k) * 32];
        dH += nu * s[L::kA1 + 2 * i + 1];
        dC += nu * s[L::kA2 + 2 * i + 1];
    }
    double krf = 0.0, ra = 0.0, rb = 0.0;
    const double s_ = x[kWs * 32];
    if (rev) {
        if (!slow) {
            double ik = 1.0;
            for (int k = 0; k < nf; ++k) ik *= pow_small(s[L::kA2 + 2 * xi[(kWidx + k) * 32]], -x[(kWnu + k) * 32]);
            for (int k = nf; k < nf + nb; ++k) ik *= pow_small(s[L::kA3 + 2 * xi[(kWidx + k) * 32]], x[(kWnu + k) * 32]);
            if (s_ == -1.0) ik *= (kPatm / kRu) * invT;
            else if (s_ == 1.0) ik *= T * (kRu / kPatm);
            else if (s_ != 0.0) ik *= exp(-s_ * (log(kPatm / kRu) - logT));
            krf = ik;
            ra = ik;
            rb = ik * (-dH * invT * invRuT - s_ * invT);
        } else {
            double kp = 0.0, dk = 0.0;
            for (int k = 0; k < nf + nb; ++k) {
                const int i = xi[(kWidx + k) * 32];
                const double nu = x[(kWnu + k) * 32];
                kp += nu * s[L::kG + i];
                dk += nu * s[L::kG + 16 + i];
            }
            dk *= invRuT;
            const double lik = kp - s_ * (log(kPatm / kRu) - logT);
            if (fabs(lik) < 650.0) {
                ra = exp(lik);
                krf = ra;
                rb = ra * (dk - s_ * invT);
            } else {
                double Kc, DKcDT;
                t3_kc_slow(kp, dk, s_, T, Kc, DKcDT);
                krf = (fabs(Kc) > kVeryTiny) ? 1.0 / Kc : 0.0;
                const double den = hmax(Kc, kVeryTiny);
                ra = 1.0 / den;
                rb = krf * DKcDT / den;
            }
        }
    }
    const double kr = kf * krf;
    double qf = kf, qr = kr;
#pragma unroll
    for (int k = 0; k < kMaxSide; ++k) {
        qf *= pf[k];
        qr *= pb[k];
    }
    const double q = qf - (rev ? qr : 0.0);
    double dkf = (type >= kLindemann) ? (Pr / (1.0 + Pr)) * Ff * (kx * invT * (b + Ta * invT))
                                      : kf * invT * (b + Ta * invT);
    double dkr = rev ? dkf * ra - kf * rb : 0.0;
#pragma unroll
    for (int k = 0; k < kMaxSide; ++k) {
        dkf *= pf[k];
        dkr *= pb[k];
    }
    double dq = dkf - dkr;
    if (!finite(dq)) dq = 0.0;
    double g = 0.0;
    if (type == kThirdBody) {
        g = fdiv(q, hmax(M, kTiny));
    } else if (type >= kLindemann) {
        double dgdT;
        t3_falloff_jac_fast(type != kLindemann, cent, Ff, logPr, k0, kx, x[kWb0 * 32], x[kWTa0 * 32], b, Ta, M, q,
                            invT, g, dgdT);
        dq += dgdT;
    }
    for (int j = 0; j < L::COLS; ++j) D[j] = (j < nsp && type != kArrhenius) ? g * er[j] : 0.0;
    D[L::TI] = dq;
    D[N] = q;
    *dHp = dH - cvRu * T * s_;
    *dCp = dC - cvRu * s_;
    // d q / d c_k: forward products for the reactants, minus the reverse ones
    for (int side = 0; side < 2; ++side) {
        const int n = side ? nb : nf, off = side ? nf : 0;
        const double K = side ? (rev ? -kr : 0.0) : kf;
        for (int k = 0; k < n; ++k) {
            double d = K;
#pragma unroll
            for (int l = 0; l < kMaxSide; ++l) {
                if (l >= n) break;
                if (l == k) {
                    const double o = x[(kWord + off + k) * 32];
                    if (o == 1.0) continue;
                    const double cj = cc(xi[(kWidx + off + k) * 32]);
                    if (o < 1.0) d *= (cj > kTiny) ? o * pow_n(cj, o - 1.0) : 0.0;
                    else d *= o * pow_n(hmax(cj, 0.0), o - 1.0);
                } else {
                    d *= side ? pb[l] : pf[l];
                }
            }
            D[xi[(kWidx + off + k) * 32]] += d;
        }
    }
}

// AUTO: autoUpdateJacobian; a build of its own, so that the other carries none of it
template <int N, bool AUTO>
struct WCell {
    using L = WLayout<N>;
    static constexpr bool kAuto = AUTO;
    static constexpr int E = 1;       // every lane of a row carries the row's element
    static constexpr unsigned full = 0xffffffffu;
    const WMech &m;
    const WTabs6 tb;
    const IntegratorParams &P;
    const int so;     // this warp's shared memory
    int lane, nsp;
    int row, h;       // this lane's row of the Newton matrix and its column block
    bool act;         // the lane owns a row
    int rl;           // row lane of column block 0 (this lane's own index when it owns none)
    double cvRu;      // Ru in the constant-volume reactor, else 0
    int da, sa, db, sb, dn;   // the dot product this lane evaluates: places, strides, length
    double a[L::C];   // this lane's columns of [I - dt J | rhs]
    double pinv;      // this row's reciprocal pivot
    unsigned long long order;   // row of pivot k, 4 bits each
    double f[1];      // this row's right-hand side (where f_here())

    __device__ WCell(const WMech &mm, const WTabs6 &t, const IntegratorParams &pp, int at, int l)
        : m(mm), tb(t), P(pp), so(at), lane(l), nsp(mm.nsp) {
        h = l / L::R;
        act = h < L::W;
        row = act ? l - h * L::R : 15;
        rl = act ? row : l;
        cvRu = (pp.reactor == 1) ? kRu : 0.0;
        const int dH = L::kDH, dC = dH + m.nrc32, D = dC + m.nrc32 + m.njob32;
        // columns 0 .. N of D with dH, then q with dCp, each in P parts; y with cp and with dcp/dT
        const int q = l % (N + 2), part = l / (N + 2);
        da = (q == N + 1 ? dC : dH) + part;
        sa = L::P;
        db = D + part * L::LD + (q == N + 1 ? N : q);
        sb = L::P * L::LD;
        dn = (part < L::P) ? (m.nrc - part + L::P - 1) / L::P : 0;
        if (l == L::P * (N + 2) || l == L::P * (N + 2) + 1) {
            da = L::kY;
            db = (l == L::P * (N + 2)) ? L::kCP : L::kDCP;
            sa = sb = 1;
            dn = nsp;
        }
        if (dn <= 0) da = db = sa = sb = dn = 0;   // nothing to sum, and nothing to read past the end
    }

    __device__ __forceinline__ double sum(double v) const {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(full, v, o);
        return v;
    }
    // the largest of non-negative values: their bit patterns order like them
    __device__ __forceinline__ double max_nonneg(double v) const {
        const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
        const unsigned mh = __reduce_max_sync(full, hi);
        const unsigned ml = __reduce_max_sync(full, hi == mh ? lo : 0u);
        return __hiloint2double((int)mh, (int)ml);
    }

    __device__ __forceinline__ bool has(int) const { return act; }
    __device__ __forceinline__ int elem(int) const { return row; }
    __device__ __forceinline__ bool f_here() const { return h == L::hN; }
    __device__ __forceinline__ double T_of(const double (&y)[1]) const { return __shfl_sync(full, y[0], L::TI); }
    // the first element that is not finite (1 << 30: none)
    __device__ __forceinline__ int first_bad(const double (&x)[1]) const {
        const unsigned bad = __ballot_sync(full, act && h == 0 && !finite(x[0]));
        return bad ? __ffs(bad) - 1 : 1 << 30;
    }
    // One reaction's row of D (lanes past the last reaction write nothing); FULL: the
    // round has third-body or fall-off reactions.
    template <bool FULL>
    __device__ __forceinline__ void reaction(int r, double T, double logT, double invT, double invRuT, bool wslow,
                                             const double *cM, int sM, const double *X, double *D) {
        double *s = w_smem() + so;
        const int32_t *rx = tb.i(tb.rx + (r >> 5) * 64 + (r & 31));
        const double *x = tb.d(tb.rd + (r >> 5) * (kWRDn * 32) + (r & 31));
        const int32_t *xi = tb.i(tb.ri + (r >> 5) * (kWRIn * 32) + (r & 31));
        const unsigned w0 = (unsigned)rx[0], w1 = (unsigned)rx[32];
        const double kx = x[kWA * 32] * X[r];
        const int rc = r < m.nrc ? r : 0;
        const double *er = tb.d(tb.eff + rc * nsp);
        double *Dr = D + rc * L::LD;
        const bool general = wslow || ((w0 >> kWXgeneral) & 1u);
        if (r < m.nrc && general)
            w_reaction_general<N>(s, x, xi, er, nsp, T, logT, invT, invRuT, wslow, cM, kx, X, cvRu, Dr, &s[L::kDH + r],
                                  &s[L::kDH + m.nrc32 + r]);
        const bool live = r < m.nrc && !general;
        const double2 *A1 = reinterpret_cast<const double2 *>(s + L::kA1);
        const double2 *A2 = reinterpret_cast<const double2 *>(s + L::kA2);
        const double2 *A3 = reinterpret_cast<const double2 *>(s + L::kA3);
        const int f0 = (w0 >> kWXf) & 15, f1 = (w0 >> (kWXf + 4)) & 15, f2 = (w0 >> (kWXf + 8)) & 15;
        const int b0 = (w0 >> kWXb) & 15, b1 = (w0 >> (kWXb + 4)) & 15, b2 = (w0 >> (kWXb + 8)) & 15;
        const double2 u0 = A1[f0], u1 = A1[f1], u2 = A1[f2], v0 = A1[b0], v1 = A1[b1], v2 = A1[b2];
        const double2 m0 = A2[f0], m1 = A2[f1], m2 = A2[f2], n0 = A3[b0], n1 = A3[b1], n2 = A3[b2];
        const int type = xi[kWtype * 32];
        const double b = x[kWb * 32], Ta = x[kWTa * 32];
        const double tk = (b + Ta * invT) * invT;          // d ln k / dT
        double kf = kx, M = 0.0;
        FallOff fo{1.0, 0.0, 0.0};
        if (FULL && type != kArrhenius) {
#pragma unroll
            for (int j = 0; j < N - 1; ++j)      // in the reference's order
                if (j < nsp) M += er[j] * cM[sM * j];
            if (type == kThirdBody) {
                kf = M * kx;
            } else {
                const int xj = xi[kWxj * 32];
                const bool troe = type != kLindemann;
                fo = fall_off<true>(troe, x[kWalpha * 32], x[kWiTsss * 32], x[kWiTs * 32], x[kWTss * 32],
                                           troe ? X[xj + 1] : 0.0, troe ? X[xj + 2] : 0.0,
                                           (type == kTroe4) ? X[xj + 3] : 0.0,
                                           x[kWA0 * 32] * X[xj] * frcp(notZeroD(kx)), M,
                                           (x[kWb0 * 32] + x[kWTa0 * 32] * invT) * invT - tk, invT);
                kf = kx * fo.w;
            }
        }
        const int sx = (int)((w0 >> kWXs) & 3u) - 1;
        const double s_ = (sx == 0) ? 0.0 : (sx < 0) ? -1.0 : 1.0;
        const double fs = (sx == 0) ? 1.0 : (sx < 0) ? (kPatm / kRu) * invT : T * (kRu / kPatm);
        const double ik = ((w0 >> kWXrev) & 1u) ? ((m0.x * m1.x) * (m2.x * n0.x)) * ((n1.x * n2.x) * fs) : 0.0;
        const double dH = ((v0.y + v1.y) + v2.y) - ((u0.y + u1.y) + u2.y);
        const double dC = ((n0.y + n1.y) + n2.y) - ((m0.y + m1.y) + m2.y);
        // products in the reference's order: net rates are small differences near equilibrium
        const double f12 = u1.x * u2.x, b12 = v1.x * v2.x;
        const double kr = kf * ik, kfu = kf * u0.x, krv = kr * v0.x;
        const double qf = kfu * f12, qr = krv * b12, q = qf - qr;
        // dkr/dT = kr (d ln kf/dT + dH/(Ru T^2) + s/T), the reference's derivative of Kc
        double dq = qf * tk - qr * (tk + (dH * invRuT + s_) * invT);
        dq = finite(dq) ? dq : 0.0;
        auto mult = [](unsigned c) { return (c == 1u) ? 1.0 : (c == 2u) ? 2.0 : 3.0; };
        double d0 = (kf * f12) * mult((w0 >> kWXmf) & 3u), d1 = kfu * u2.x, d2 = kfu * u1.x;
        double d3 = -(kr * b12) * mult((w0 >> kWXmb) & 3u), d4 = -(krv * v2.x), d5 = -(krv * v1.x);
        const int c0 = w1 & 31, c1 = (w1 >> 5) & 31, c2 = (w1 >> 10) & 31;
        const int c3 = (w1 >> 15) & 31, c4 = (w1 >> 20) & 31, c5 = (w1 >> 25) & 31;
        if (FULL && type != kArrhenius) {
            double g;
            if (type == kThirdBody) {
                g = q * fast_rcp(hmax(M, kTiny));
            } else {
                const double dT = q * fo.wT;
                g = q * fo.gM;
                g = finite(g) ? g : 0.0;
                dq += finite(dT) ? dT : 0.0;
            }
            // columns rank one in the efficiencies; a participant's own comes on top
            auto e = [&](int c) { return (c < nsp) ? er[c] * g : 0.0; };
            d0 += e(c0), d1 += e(c1), d2 += e(c2), d3 += e(c3), d4 += e(c4), d5 += e(c5);
            if (live) {
#pragma unroll
                for (int j = 0; j < N - 1; ++j)
                    if (j < nsp) Dr[j] = er[j] * g;
            }
        }
        if (live) {
            Dr[c0] = d0;
            Dr[c1] = d1;
            Dr[c2] = d2;
            Dr[c3] = d3;
            Dr[c4] = d4;
            Dr[c5] = d5;
            Dr[L::TI] = dq;
            Dr[N] = q;
            s[L::kDH + r] = dH - cvRu * T * s_;
            s[L::kDH + m.nrc32 + r] = dC - cvRu * s_;
        }
    }

    // ---------------------------------------------------------------------
    // f(y) and [I - dt J | (y0 - y) + dt f] in this warp's registers; y is
    // this lane's row's element. rhs_only: only f is used, and the
    // constant-volume right-hand side takes c as given for the third bodies.
    __device__ __forceinline__ void evaluate(const double (&yv)[1], const double (&y0)[1], double dt, bool rhs_only) {
        double *s = w_smem() + so;
        const double y = yv[0];
        const double T = T_of(yv);
        const double invT = fast_rcp(hmax(T, kTiny));
        const double logT = fast_log(T);
        const double invRuT = invT * (1.0 / kRu);
        // ---- species (lane i) and the exponentials of the rate laws (one per lane), the
        // two in one stretch of code without branches so that their chains overlap; the
        // lanes past the last species work on zero tables
        double *X = s + L::kDH + 2 * m.nrc32;
        const double *ts = tb.d(lane);
        const double tl = ts[kWtl * 32], tc = ts[kWtc * 32], thh = ts[kWth * 32];
        const double *tr = ts + (kWrange + ((T < tc) ? 0 : kWRangeN)) * 32;
        const double *xj = tb.d(tb.xj + lane);
        const double xarg = xj[0] * logT + xj[32] * invT + xj[64] * T;
        double h_ = T * (tr[0] + T * (tr[32] + T * (tr[64] + T * (tr[96] + T * tr[128])))) + tr[160];
        const double s0 = tr[192] * logT +
                          (T * (tr[224] + T * (tr[256] + T * (tr[288] + T * tr[320]))) + tr[352]);
        double g = (h_ - T * s0) * invRuT;
        double dgt = -h_ * invT;
        double cp = tr[384] + T * (tr[416] + T * (tr[448] + T * (tr[480] + T * tr[512])));
        double dcp = tr[544] + T * (tr[576] + T * (tr[608] + T * tr[640]));
        const bool sp = lane < nsp, out = sp && !(T >= tl && T <= thh);
        if (out)
            t3_thermo_slow(&m.raw[14 * lane + ((T < tc) ? 0 : 7)], tl, thh, ts[kWW * 32], T, logT, invRuT, cp, h_,
                           dcp, g, dgt);
        const bool slow = sp && (out || !(fabs(g) < m.glim));
        const double e = fast_exp(hmin(hmax(g, -m.glim), m.glim));
        X[lane] = fast_exp(xarg);
        if (sp) {
            reinterpret_cast<double2 *>(s + L::kA1)[lane] = make_double2(hmax(y, 0.0), h_);
            reinterpret_cast<double2 *>(s + L::kA2)[lane] = make_double2(fast_rcp(e), cp);
            reinterpret_cast<double2 *>(s + L::kA3)[lane] = make_double2(e, cp);
            s[L::kY + lane] = y;
            s[L::kCP + lane] = cp - cvRu;
            s[L::kDCP + lane] = dcp;
            s[L::kG + lane] = g;
            s[L::kG + 16 + lane] = dgt;
        }
        for (int j = lane + 32; j < m.njob; j += 32) {
            const double *xq = tb.d(tb.xj + (j >> 5) * 96 + (j & 31));
            X[j] = fast_exp(xq[0] * logT + xq[32] * invT + xq[64] * T);
        }
        const bool wslow = __any_sync(full, slow);
        __syncwarp();
        // ---- reactions: one row of D each
        double *D = X + m.njob32;
        // the third bodies' concentrations: clamped, or as given (see above)
        const double *cM = (rhs_only && cvRu != 0.0) ? s + L::kY : s + L::kA1;
        const int sM = (rhs_only && cvRu != 0.0) ? 1 : 2;
        for (int r0 = 0; r0 < m.nrc; r0 += 32) {
            const int r = r0 + lane;
            // plain Arrhenius rounds skip the third-body and fall-off code
            if (__any_sync(full, *tb.i(tb.ri + (r0 >> 5) * (kWRIn * 32) + kWtype * 32 + lane) != kArrhenius))
                reaction<true>(r, T, logT, invT, invRuT, wslow, cM, sM, X, D);
            else
                reaction<false>(r, T, logT, invT, invRuT, wslow, cM, sM, X, D);
        }
        __syncwarp();
        // ---- species rows (all lists in lock step) and the temperature row's dot products
        double acc[L::C];
#pragma unroll
        for (int c = 0; c < L::C; ++c) acc[c] = 0.0;
        double dot = 0.0;
        const double *Dh = D + (act ? h : 0) * L::C;
        // four entries at a time, so that their table and record loads overlap
        for (int e = 0; AUTO && rhs_only && e < m.gE; e += 4) {      // column N alone
            double nu[4], q[4], da_[4], db_[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                nu[k] = *tb.d(tb.gnu + 16 * (e + k) + row);
                q[k] = D[*tb.i(tb.gslot + 16 * (e + k) + row) * L::LD + N];
                const int p = (e + k < dn) ? e + k : 0;
                da_[k] = (e + k < dn) ? s[da + p * sa] : 0.0;
                db_[k] = s[db + p * sb];
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                dot += da_[k] * db_[k];
                acc[L::cN] += nu[k] * q[k];
            }
        }
        for (int e = 0; !(AUTO && rhs_only) && e < m.gE; e += 4) {
            double nu[4], da_[4], db_[4];
            const double2 *d2[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                nu[k] = *tb.d(tb.gnu + 16 * (e + k) + row);
                d2[k] = reinterpret_cast<const double2 *>(Dh + *tb.i(tb.gslot + 16 * (e + k) + row) * L::LD);
                const int p = (e + k < dn) ? e + k : 0;
                da_[k] = (e + k < dn) ? s[da + p * sa] : 0.0;
                db_[k] = s[db + p * sb];
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                dot += da_[k] * db_[k];
#pragma unroll
                for (int c = 0; c < L::C; c += 2) {
                    const double2 d = d2[k][c / 2];
                    acc[c] += nu[k] * d.x;
                    acc[c + 1] += nu[k] * d.y;
                }
            }
        }
        s[L::kTS + lane] = dot;
        __syncwarp();
        // ---- temperature equation (chemistrySource.cpp:863-906, 975-1055)
        const double *td = s + L::kTS;
        const double icCp = frcp(td[L::P * (N + 2)]), dcCp = td[L::P * (N + 2) + 1];
        auto dots = [td](int q) { return L::P == 2 ? td[q] + td[N + 2 + q] : td[q]; };
        const double DT = dots(N) * icCp;      // sum_r q_r dH_r / C = sum_i f_i h_i / C
        if (row == L::TI) {
#pragma unroll
            for (int c = 0; c < L::C; ++c) {
                const int j = h * L::C + c;
                const double cpj = (j < L::TI) ? s[L::kCP + j] : (j == L::TI) ? dcCp : 0.0;
                double S = dots(j < N ? j : N);
                if (j == L::TI) S += dots(N + 1);
                acc[c] = (cpj * DT - S) * icCp;
            }
        }
        f[0] = acc[L::cN];
#pragma unroll
        for (int c = 0; c < L::C; ++c) a[c] = ((h * L::C + c == row) ? 1.0 : 0.0) - dt * acc[c];
        if (h == L::hN) a[L::cN] = (-y + y0[0]) + dt * f[0];
    }

    // x of [A | b] in the registers a[]; every lane gets its row's element. reuse (AUTO): with
    // the factors of the last call and the right-hand side in a[]; step by step what the
    // elimination does to it, so that x is the same to the last bit
    __device__ __forceinline__ void solve(double (&x)[1], bool reuse) {
        double *U = w_smem() + so + L::doubles(m.nrc, m.nrc32, m.njob32), *M = U + N * L::kLU;
        if (AUTO && reuse) {
            double b = a[L::cN];
#pragma unroll
            for (int k = 0; k < N; ++k) {
                const double u = __shfl_sync(full, b, L::hN * L::R + ((int)(order >> (4 * k)) & 15));
                b -= M[(act ? row : 0) * L::kLM + k] * u;
            }
#pragma unroll
            for (int c = 0; c < L::C; ++c) a[c] = U[(act ? row : 0) * L::kLU + h * (act ? L::C : 0) + c];
            substitute(x, b);
            return;
        }
        eliminate(M);
        if (AUTO) {
            if (act) {
#pragma unroll
                for (int c = 0; c < L::C; ++c) U[row * L::kLU + h * L::C + c] = a[c];
            }
            __syncwarp();
        }
        substitute(x, a[L::cN]);
    }

    // M (AUTO): the multipliers
    __device__ __forceinline__ void eliminate(double *M) {
        // the pivot's key carries its row; a zero pivot makes the reciprocal, and x, not finite
        constexpr int R = L::R;
        pinv = 0.0;
        bool used = !act;
        order = 0ull;
        auto key = [&](double v, int hk) {
            const unsigned hi = (unsigned)__double2hiint(v) & 0x7fffffffu;
            return (h == hk && !used) ? ((hi & ~31u) | (unsigned)(31 - row)) : 0u;
        };
        unsigned top = __reduce_max_sync(full, key(a[0], 0));
        double own = fast_rcp(a[0]);
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const int hk = k / L::C, ck = k % L::C;
            const int hn = (k + 1) / L::C, cn = (k + 1) % L::C;
            const double mine = __shfl_sync(full, a[ck], hk * R + rl);
            const int pr = 31 - (int)(top & 31u);
            const double inv = __shfl_sync(full, own, hk * R + pr);
            const bool piv = row == pr;
            const int from = h * R + pr;
            used = used || piv;
            const double l = used ? 0.0 : mine * inv;
            if (AUTO && act && h == 0) M[row * L::kLM + k] = l;
            pinv = piv ? inv : pinv;
            order |= (unsigned long long)pr << (4 * k);
            // the next pivot column first: its search and reciprocals run under the other columns
            const double un = __shfl_sync(full, a[cn], from);
            a[cn] -= l * un;
            if (k + 1 < N) {
                top = __reduce_max_sync(full, key(a[cn], hn));
                own = fast_rcp(a[cn]);
            }
#pragma unroll
            for (int c = 0; c < L::C; ++c) {
                if (c == cn || (hk == L::W - 1 && c <= ck)) continue;
                const double u = __shfl_sync(full, a[c], from);
                a[c] -= l * u;
            }
        }
    }

    // back substitution along the pivot order; b: the eliminated right-hand side, in column block hN
    __device__ __forceinline__ void substitute(double (&x)[1], double b) {
        x[0] = 0.0;
#pragma unroll
        for (int k = N - 1; k >= 0; --k) {
            const int pr = (int)(order >> (4 * k)) & 15;
            const double u = __shfl_sync(full, a[k % L::C], (k / L::C) * L::R + rl);
            const double xk = __shfl_sync(full, b * pinv, L::hN * L::R + pr);
            x[0] = (row == k) ? xk : x[0];
            b -= u * xk;
        }
    }
};

constexpr int kWWarps = 8;  // most warps (cells in flight) per block

// shared memory of a block of `warps` warps (bytes)
template <int N>
size_t w6_smem_bytes(const WMech &m, int warps, bool keepJ) {
    using L = WLayout<N>;
    const size_t w = L::doubles(m.nrc, m.nrc32, m.njob32) + (keepJ ? (size_t)L::kFactors : 0);
    return sizeof(double) * (w6_tables_doubles(m) + w * warps);
}

// BLOCKS an SM: 1 (up to 255 registers a thread, nothing spilled: the shorter Newton
// iteration) or 2 (128 registers: more cells in flight); variant_w.cu chooses
template <int N, int BLOCKS, bool AUTO>
__global__ void __launch_bounds__(32 * kWWarps, BLOCKS)
integrate_w_kernel(const __grid_constant__ WMech m, const __grid_constant__ IntegratorParams P,
                   const __grid_constant__ CellIO io) {
    using L = WLayout<N>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int nsp = m.nsp;
    const unsigned full = 0xffffffffu;
    // the mechanism tables into the block's shared memory, once
    WTabs6 tb;
    {
        int d = 0;
        auto copy = [&](const double *src, int n) {
            for (int i = threadIdx.x; i < n; i += blockDim.x) w_smem()[d + i] = src[i];
            d += n;
            return d - n;
        };
        copy(m.th, kWTHn * 32);
        tb.rd = copy(m.rd, kWRDn * m.nrc32);
        tb.eff = copy(m.eff, (m.nrc > 0 ? m.nrc : 1) * nsp);
        tb.gnu = copy(m.gnu, 16 * m.gE);
        tb.xj = copy(m.xj, 3 * m.njob32);
        int q = 2 * d;
        auto copyi = [&](const int32_t *src, int n) {
            for (int i = threadIdx.x; i < n; i += blockDim.x) reinterpret_cast<int32_t *>(w_smem())[q + i] = src[i];
            q += n;
            return q - n;
        };
        tb.ri = copyi(m.ri, kWRIn * m.nrc32);
        tb.rx = copyi(m.rx, 2 * m.nrc32);
        tb.gslot = copyi(m.gslot, 16 * m.gE);
    }
    const size_t wd = L::doubles(m.nrc, m.nrc32, m.njob32) + (AUTO ? (size_t)L::kFactors : 0);
    const int so = (int)(w6_tables_doubles(m) + (size_t)warp * wd);
    double *s = w_smem() + so;
    for (int i = lane; i < (int)wd; i += 32) s[i] = 0.0;
    __syncwarp();
    if (lane == 0) {
        // the slot that absent factors read
        s[L::kA1 + 2 * kWOne] = 1.0;
        s[L::kA2 + 2 * kWOne] = 1.0;
        s[L::kA3 + 2 * kWOne] = 1.0;
    }
    __syncthreads();
    StepControl<WCell<N, AUTO>> ci(m, tb, P, so, lane);
    const int row = ci.row;
    const bool sp = ci.act && row < nsp, own = sp && ci.h == 0;
    const double W = sp ? *tb.d(kWW * 32 + row) : 1.0;
    // the first cells go round the blocks (one warp per SM while they last), the rest by the queue
    const long long first = (long long)gridDim.x * warps;
    auto next = [&]() {
        long long q = 0;
        if (lane == 0) q = first + (long long)atomicAdd(io.queue_head, 1ULL);
        return __shfl_sync(full, q, 0);
    };
    for (long long k = (long long)warp * gridDim.x + blockIdx.x; k < io.nqueue; k = next()) {
        const int64_t cell = io.order ? (int64_t)io.order[k] : (int64_t)k;
        ci.start();
        const double Ti = io.T[cell];
        const double tstep = io.dt[cell] * io.dt_factor;
        const double rho0 = io.rho[cell];
        double y = 0.0;
        if (sp) y = rho0 * io.Y[(int64_t)row * io.ncells + cell] * frcp(W);
        const double c0 = y;
        if (Ti < P.T_threshold) {
            if (lane == 0) {
                io.subdt[cell] = tstep;
                if (io.status) io.status[cell] = 1;  // HC_CELL_SKIPPED
                if (io.cost) io.cost[cell] = 0;
            }
            if (io.Ri && own) io.Ri[(int64_t)row * io.ncells + cell] = 0.0;
            continue;
        }
        double sub = hmin(tstep, hmin(io.subdt[cell], P.dt_max));
        double yv[1] = {(ci.act && row == N - 1) ? Ti : y};
        ci.cell(tstep, sub, yv);
        y = yv[0];
        // ciToYi (chemistrySource.cpp:1225-1246) and rho = p / (Rm T)
        const double Tn = __shfl_sync(full, y, N - 1);
        double yi = own ? hmax(0.0, y) : 0.0;
        const double rr = ci.sum(own ? yi * W : 0.0);
        yi = own ? yi * W * frcp(hmax(rr, kTiny)) : 0.0;
        const double ys = ci.sum(yi);
        if (ys != 1.0) yi *= frcp(ys);
        const double wsum = ci.sum(own ? yi * frcp(W) : 0.0);
        const double Rm = kRu * hmax(wsum, kVeryTiny);
        if (own) {
            io.Y[(int64_t)row * io.ncells + cell] = yi;
            if (io.Ri) io.Ri[(int64_t)row * io.ncells + cell] = (y - c0) * frcp(tstep) * W;
        }
        if (lane == 0) {
            ci.store(io, cell, Tn, sub);
            // constant volume keeps the density (chemistrySource.cpp:1317-1323)
            if (P.reactor != 1) io.rho[cell] = fdiv(io.p[cell], Rm * Tn);
        }
    }
}

}  // namespace hc
