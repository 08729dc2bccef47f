// Tables of the lanes-per-cell rate kernels (rates.cu): explicit and
// point-implicit source terms of mechanisms whose reactions all have the
// direct form (unit-order factors, at most three a side, no species twice
// but for a repeated factor, none of the rarer rate laws).
#pragma once

#include <cuda_runtime.h>

#include <string>

#include "fastmath.cuh"
#include "mech.cuh"
#include "t3_base.cuh"

namespace hc {

// code.x: species of the forward factors (8 bits each, nsp for none) | rate type << 24
// code.y: species of the reverse factors
// code.z: kR* fields; code.w: first efficiency entry | fall-off row << 16
enum RFlags : int {
    kRfirst = 0,      // 6 bits: factor k is its species' first occurrence
    kRmf = 6,         // multiplicity of forward factor 0 (2 bits), of reverse factor 0
    kRmb = 8,
    kRrev = 10,
    kRlast = 11,      // factor that is the last species (7: none)
    kRall = 14,       // third body: every species counts 1, the entries hold the differences
    kRneff = 16       // number of efficiency entries (8 bits)
};
constexpr int kRFall = 8;   // A0, b0, Ta0, alpha, 1/T***, 1/T*, T**, unused

struct RMech {
    int32_t nsp, nrc;
    const int4 *code;       // [nrc]
    const double4 *rate;    // [nrc] A, b, Ta, change in moles
    const double *th;       // [nsp][kRTh]
    const int32_t *eidx;    // third-body entries: species, efficiency (less 1 where kRall)
    const double *eval;
    const double *fall;     // [..][kRFall]
};

// th: per species Tl, Tc, Th, W, 1/W, then per range a0 .. a5 of the molar NASA-7
// polynomial over Ru and the terms of the Gibbs energy per mass (kRG), as the
// reference divides them
constexpr int kRange = 6 + 7, kRG = 6;
constexpr int kRTh = 5 + 2 * kRange;

// the range's coefficients at T
__device__ __forceinline__ const double *species_range(const double *t, double T) {
    return t + ((T < ldg(&t[1])) ? 5 : 5 + kRange);
}

// molar G0 in the reference's order of operations (JANAF::g0, JANAF.cpp:201-213): its
// rounding is then the reference's, which the small net rates near equilibrium magnify
__device__ __forceinline__ double species_gibbs(const double *t, const double *a, double T, double lT) {
    const double *g = a + kRG;
    const double g0 = ((((-ldg(&g[4]) * T - ldg(&g[3])) * T - ldg(&g[2])) * T - ldg(&g[1])) * T + ldg(&g[0]) * (1 - lT) -
                       ldg(&g[6])) * T + ldg(&g[5]);
    return g0 * ldg(&t[3]);
}

// H / Ru and Cp / Ru as the reference evaluates them: outside the fitted range cp at
// the range's end, h extrapolated from there (JANAF.cpp:142-199)
__device__ __forceinline__ void species_hcp(const double *t, double T, double &h, double &cp) {
    const double *a = species_range(t, T);
    const double a0 = ldg(&a[0]), a1 = ldg(&a[1]), a2 = ldg(&a[2]), a3 = ldg(&a[3]), a4 = ldg(&a[4]);
    const double Tc = hmin(hmax(T, ldg(&t[0])), ldg(&t[2]));
    cp = a0 + Tc * (a1 + Tc * (a2 + Tc * (a3 + Tc * a4)));
    h = Tc * (a0 + Tc * (a1 * 0.5 + Tc * (a2 * (1.0 / 3.0) + Tc * (a3 * 0.25 + Tc * (a4 * 0.2))))) + ldg(&a[5]);
    h += cp * (T - Tc);
}

constexpr double kLnRuPatm = -2.5003366899611787;   // ln(Ru / p_atm)

// One reaction at a state (reactionTypes q / Kc / DqDci / DqDT, reactionTypes.cpp:178-445,
// 843-876, unimolecularFallOffRR, fallOffFunctions).
struct RxnVals {
    double q;
    // JAC only: dq/dT, the factor of the efficiencies in dq/dc, dq/dc of each factor's species
    double dq, g, d[6];
};

// The species by slot (slot nsp: c = 1, g = d = 0): cg(i) = {c clamped, g = G0},
// dd(i) = (dG0/dT - G0/T) / Ru, cm(i) the third bodies' concentrations with their sum
// ctot. 1/Kc is one exponential of the reaction's change in g, so that no species'
// exp(+-g) has to be held or can overflow on its own. k4: A, b, Ta, change in moles.
// LEAN: lean_exp (throughput) instead of fast_exp (latency).
template <bool JAC, bool LEAN, class CG, class CM, class DD>
__device__ __forceinline__ RxnVals rxn_eval(const RMech &m, const int4 w, const double4 k4, CG cg, CM cm, DD dd,
                                            double T, double invT, double logT, double ctot) {
    const double invRuT = invT * (1.0 / kRu);
    RxnVals o;
    auto ex = [](double x) { return LEAN ? lean_exp(x) : fast_exp(x); };
    const int nsp = m.nsp;
    const int i0 = w.x & 255, i1 = (w.x >> 8) & 255, i2 = (w.x >> 16) & 255, type = w.x >> 24;
    const int j0 = w.y & 255, j1 = (w.y >> 8) & 255, j2 = (w.y >> 16) & 255;
    const double sm = k4.w, lRTp = kLnRuPatm + logT;
    const double kx = k4.x * ex(k4.y * logT - k4.z * invT);
    const double2 U0 = cg(i0), U1 = cg(i1), V0 = cg(j0), V1 = cg(j1);
    const double u0 = U0.x, u1 = U1.x, v0 = V0.x, v1 = V1.x;
    double dG = -U0.y - U1.y;
    double u2 = 1.0, v2 = 1.0;
    if (i2 != nsp) {
        const double2 U2 = cg(i2);
        u2 = U2.x;
        dG -= U2.y;
    }
    dG = (dG + V0.y) + V1.y;
    if (j2 != nsp) {
        const double2 V2 = cg(j2);
        v2 = V2.x;
        dG += V2.y;
    }
    const double arg = dG * invRuT + sm * lRTp;
    double dk = 0.0;
    if (JAC) {
        dk = (dd(j0) + dd(j1)) - (dd(i0) + dd(i1));
        if (i2 != nsp) dk -= dd(i2);
        if (j2 != nsp) dk += dd(j2);
        dk *= invT;
    }
    // kr = kf krf, dkr/dT = dkf/dT ra - kf rb (reactionTypes::Kc, ::DKcDT)
    double krf = 0.0, ra = 0.0, rb = 0.0;
    if ((w.z >> kRrev) & 1) {
        if (fabs(arg) < 650.0) {
            krf = ra = ex(arg);
            rb = krf * (dk - sm * invT);
        } else {
            double Kc, DKcDT;
            t3_kc_slow(arg - sm * lRTp, dk, sm, T, Kc, DKcDT);
            krf = (fabs(Kc) > kVeryTiny) ? 1.0 / Kc : 0.0;
            const double den = hmax(Kc, kVeryTiny);
            ra = 1.0 / den;
            rb = krf * DKcDT / den;
        }
    }
    double kf = kx, M = 0.0;
    const double tk = (k4.y + k4.z * invT) * invT;         // d ln k / dT
    FallOff fo{1.0, 0.0, 0.0};
    if (type != kArrhenius) {
        const int e0 = w.w & 0xffff, ne = (w.z >> kRneff) & 255;
        M = ((w.z >> kRall) & 1) ? ctot : 0.0;
        for (int e = e0; e < e0 + ne; ++e) M += ldg(&m.eval[e]) * cm(ldg(&m.eidx[e]));
        if (type == kThirdBody) {
            kf = M * kx;
        } else {
            const double *fl = m.fall + (w.w >> 16) * kRFall;
            const double b0 = ldg(&fl[1]), Ta0 = ldg(&fl[2]);
            const double k0 = ldg(&fl[0]) * ex(b0 * logT - Ta0 * invT);
            const double up = (fabs(kx) < 1e-290) ? 0x1p200 : 1.0;   // frcp takes no subnormal kx
            const bool troe = type != kLindemann;
            double e1 = 0.0, e2 = 0.0, e3 = 0.0, iT3 = 0.0, iT1 = 0.0, T2 = 0.0;
            if (troe) {
                iT3 = ldg(&fl[4]);
                iT1 = ldg(&fl[5]);
                T2 = ldg(&fl[6]);
                e1 = ex(-T * iT3);
                e2 = ex(-T * iT1);
                if (type == kTroe4) e3 = ex(-T2 * invT);
            }
            fo = fall_off<JAC>(troe, ldg(&fl[3]), iT3, iT1, T2, e1, e2, e3, (k0 * up) * frcp(notZeroD(kx) * up), M,
                               (b0 + Ta0 * invT) * invT - tk, invT);
            kf = kx * fo.w;
        }
    }
    const double kr = kf * krf;
    // products in the reference's order: net rates are small differences near equilibrium
    o.q = ((kf * u0) * u1) * u2 - ((kr * v0) * v1) * v2;
    if (JAC) {
        // in this order too: a product of concentrations alone underflows where the large
        // reverse rate at low T brings it back
        const double dkf = kf * tk;
        o.dq = ((dkf * u0) * u1) * u2 - (((dkf * ra - kf * rb) * v0) * v1) * v2;
        if (!finite(o.dq)) o.dq = 0.0;
        o.g = 0.0;
        if (type == kThirdBody) {
            o.g = fdiv(o.q, hmax(M, kTiny));
        } else if (type >= kLindemann) {
            const double g = o.q * fo.gM, dT = o.q * fo.wT;
            o.g = finite(g) ? g : 0.0;
            o.dq += finite(dT) ? dT : 0.0;
        }
        const int mf = (w.z >> kRmf) & 3, mb = (w.z >> kRmb) & 3;
        o.d[0] = ((mf == 1) ? 1.0 : (mf == 2) ? 2.0 : 3.0) * ((kf * u1) * u2);
        o.d[1] = (kf * u0) * u2;
        o.d[2] = (kf * u0) * u1;
        o.d[3] = ((mb == 1) ? -1.0 : (mb == 2) ? -2.0 : -3.0) * ((kr * v1) * v2);
        o.d[4] = -(kr * v0) * v2;
        o.d[5] = -(kr * v0) * v1;
    }
    return o;
}

// diag null: the explicit terms only
int launch_rates(const RMech &m, const DevMech &dm, int num_sms, int64_t n, const double *T, const double *rho,
                 const double *Y, double *Ri, double *diag, cudaStream_t st, std::string &err);
// whether some launch's shared memory holds the mechanism
bool rates_fit(int nsp, int nrc, bool implicit);

}  // namespace hc
