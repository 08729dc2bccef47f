// Mixture property kernel: per-species enthalpy, mixture cp, Wilke viscosity
// and conductivity, mixture-averaged diffusion coefficients.
//
//   h_i, cp        thermo/src/JANAF.cpp:155-199, thermoList.cpp:165-190
//   mu_i, kappa_i  transport/src/kineticTheory.cpp:37-57, kineticTheory.inl:32-34
//   mu, kappa      transport/src/transportList.cpp:238-284 (muKappa, Wilke)
//   x_i            species/src/speciesList.cpp:208-224 (Yi2Xi)
//   D_i            transport/src/kineticTheory.cpp:118-163 (Di), T^1.5 = T sqrt(T)
//
// Lanes per cell: a block holds up to 128 cells in shared memory (mole
// fractions x and 1/S, see below) and the pair tables, and L threads share a
// cell's blocks of four rows i. What bounds it is the FP64 pipe: the O(nsp^2)
// pair loop, 12 FP64 instructions a pair, no division and no square root.
//
//  * Wilke: sqrt(mu_i / mu_j sqrt(W_j / W_i)) = S_i / S_j with S = sqrt(mu / sqrt(W)),
//    so sum_j phi_ij x_j = A_i + 2 S_i B_i + S_i^2 C_i with A, B, C the products of
//    the constant matrix c_ij = 1 / sqrt(8 (1 + W_i / W_j)) with x, x / S and
//    x / S^2 (all terms positive);
//  * diffusion: sum_j x_j / D_ij = p / T^1.5 sum_j x_j Omega_ij / d_ij, Omega_ij =
//    T^-0.145 e_ij + 1 / (T / sqrt(eps_i eps_j) + 1/2)^2: one reciprocal a pair
//    (hardware approximation and one cubic step); the tables are zero for j = i;
//  * four rows per thread, so that x_j and 1/S_j are read once for four pairs and
//    the tables come as 16-byte broadcast loads.
//
// Rounding: the constants come from the host's extended precision, quotients are corrected
// to half an ulp (near_div), mu_i is formed again for its row instead of squaring 1 / R:
// the errors against extended precision are those of the divisions and square roots it
// replaced (mu of 9 species 1.58e-16, without these steps 2.18e-16), at the same time.
// The pair sums stay one chain: partial sums of 16 columns cost 10 us for one cell (their
// registers) and gain nothing over the former kernel, which had one chain too.
//
// Measured (B200, 65,536 cells of 53 species): 1911 us before (a warp per cell, a
// division and a square root a pair), 280 us now.
#include <cuda_runtime.h>

#include <string>

#include "../../include/hurchem_b200.h"
#include "fastmath.cuh"
#include "launch.cuh"
#include "variants.h"

namespace hc {

constexpr int kPropMaxSp = 64;
constexpr int kPropThreads = 512;   // most threads of a block
constexpr int kPropCells = 128;     // most cells of a block
constexpr int kPropSp = 7;          // constants per species at the end of DevMech::ptab

// a / b from a and r, nearly 1 / b, to within little more than half an ulp, without the
// division's slow path: b normal and not zero
__device__ __forceinline__ double near_div(double a, double b, double r) {
    const double q = a * r;
    return fma(fma(-q, b, a), r, q);
}

// a sum in four chains, taken in turn: one chain of nsp / L additions rounds as often
struct Sum4 {
    double a = 0.0, b = 0.0, c = 0.0, d = 0.0;
    __device__ __forceinline__ void add(double y) {
        const double t = a + y;
        a = b;
        b = c;
        c = d;
        d = t;
    }
    __device__ __forceinline__ double value() const { return (a + b) + (c + d); }
};

// viscosity of the species with constants q (kineticTheory.cpp:37-57): q[2] sqrt(T) over this
__device__ __forceinline__ double species_omega(const double *q, double T, double Tpow) {
    const double rt = fast_rcp(T * q[0] + 0.5);                  // 1 / (T / eps_i + 1/2)
    return 1.147 * (Tpow * q[1]) + rt * rt;
}

__global__ void __launch_bounds__(kPropThreads, 1)
properties_kernel(const __grid_constant__ DevMech m, int64_t n, const double *__restrict__ T_,
                  const double *__restrict__ p_, const double *__restrict__ Y, double *ha,
                  double *cpm, double *mu, double *kappa, double *D, int L, int64_t tiles) {
    extern __shared__ __align__(16) double smem_p[];
    const int nsp = m.nsp, NB = (nsp + 3) / 4, B = blockDim.x / L;
    const int tab = 4 * NB * nsp;
    double *pc = smem_p;                        // c, 1/d, e: [row block][j][4 rows] each
    double *pi = pc + tab, *pe = pi + tab, *se = pe + tab;   // then 1/sqrt(eps) per species
    const int cl = threadIdx.x % B, l = threadIdx.x / B;
    const double *sp = se + 4 * NB;             // and kPropSp constants per species
    double *x = se + 4 * NB + kPropSp * nsp + cl, *R = x + nsp * B, *part = R + nsp * B;
#pragma unroll 8
    for (int i = threadIdx.x; i < 3 * tab + 4 * NB + kPropSp * nsp; i += blockDim.x) smem_p[i] = ldg(&m.ptab[i]);
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        __syncthreads();
        const int64_t cell0 = tile * B + cl;
        const bool live = cell0 < n;
        const int64_t cell = live ? cell0 : n - 1;
        const double T = T_[cell], p = p_[cell];
        // Yi2Xi
        double wsum = 0.0;
        Sum4 cps;
        for (int i = l; i < nsp; i += L) {
            const double w = near_div(Y[(int64_t)i * n + cell], sp[kPropSp * i + 4], sp[kPropSp * i + 5]);
            x[i * B] = w;
            wsum += w;
        }
        part[l * B] = wsum;
        __syncthreads();
        wsum = 0.0;
        for (int k = 0; k < L; ++k) wsum += part[k * B];
        const double Wmean = 1.0 / hmax(wsum, kVeryTiny);
        // T^-0.145 with what the product rounds off: every coefficient of the cell has its error
        const double sqT = sqrt(T), lT = fast_log(T), arg = -0.145 * lT, pw = fast_exp(arg);
        const double Tpow = fma(pw, fma(-0.145, lT, -arg), pw);
        double xt = 0.0;
        for (int i = l; i < nsp; i += L) {
            const double xi = hmax(0.0, hmin(1.0, x[i * B] * Wmean));
            x[i * B] = xi;
            xt += xi;
            // species enthalpy, viscosity
            double cp0, h0;
            species_cp_h(m, i, T, cp0, h0);
            if (ha && live) ha[(int64_t)i * n + cell] = h0;
            cps.add(cp0 * Y[(int64_t)i * n + cell]);
            const double *q = sp + kPropSp * i;
            const double om = species_omega(q, T, Tpow);
            R[i * B] = rsqrt(near_div(q[2] * sqT, om, fast_rcp(om)) * q[3]);   // 1 / S
        }
        part[(L + l) * B] = xt;
        part[(2 * L + l) * B] = cps.value();
        __syncthreads();
        xt = 0.0;
        for (int k = 0; k < L; ++k) xt += part[(L + k) * B];
        if (xt != 1.0) {
            const double ixt = 1.0 / xt;
            for (int i = l; i < nsp; i += L) x[i * B] = near_div(x[i * B], xt, ixt);
        }
        __syncthreads();
        // Wilke mixing (transportList::muKappa) and mixture-averaged D_i
        double mum = 0.0, kappam = 0.0;
        const double scale = T * sqT / p;
        for (int ib = l; ib < NB; ib += L) {
            double A[4], Bs[4], Cs[4], Ds[4], Te[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                A[q] = Bs[q] = Cs[q] = Ds[q] = 0.0;
                Te[q] = T * se[4 * ib + q];
            }
            const double2 *c2 = reinterpret_cast<const double2 *>(pc + 4 * ib * nsp);
            const double2 *i2 = reinterpret_cast<const double2 *>(pi + 4 * ib * nsp);
            const double2 *e2 = reinterpret_cast<const double2 *>(pe + 4 * ib * nsp);
            for (int j = 0; j < nsp; ++j) {
                const double xj = x[j * B], Rj = R[j * B], ej = se[j];
                const double xr = xj * Rj, xrr = xr * Rj;
                double c[4], d[4], e[4];
                *reinterpret_cast<double2 *>(c) = c2[2 * j];
                *reinterpret_cast<double2 *>(c + 2) = c2[2 * j + 1];
                *reinterpret_cast<double2 *>(d) = i2[2 * j];
                *reinterpret_cast<double2 *>(d + 2) = i2[2 * j + 1];
                *reinterpret_cast<double2 *>(e) = e2[2 * j];
                *reinterpret_cast<double2 *>(e + 2) = e2[2 * j + 1];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    A[q] = fma(c[q], xj, A[q]);
                    Bs[q] = fma(c[q], xr, Bs[q]);
                    Cs[q] = fma(c[q], xrr, Cs[q]);
                    const double inv = fast_rcp(fma(Te[q], ej, 0.5));
                    Ds[q] = fma(xj * d[q], fma(inv, inv, Tpow * e[q]), Ds[q]);
                }
            }
            double wm[4] = {0.0, 0.0, 0.0, 0.0}, wk[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int i = 4 * ib + q;
                if (i >= nsp) break;
                const double *c = sp + kPropSp * i;
                // mu_i again, not the square of 1 / R, which would double its rounding errors
                const double Si = fast_rcp(R[i * B]), phi = A[q] + Si * (2.0 * Bs[q] + Si * Cs[q]);
                const double den = species_omega(c, T, Tpow) * phi;
                double cp0, h0;
                species_cp_h(m, i, T, cp0, h0);
                const double xi = x[i * B];
                wm[q] = near_div(c[2] * sqT * xi, den, fast_rcp(den));
                wk[q] = wm[q] * (cp0 + 1.25 * c[6]);
                if (D && live) {
                    double Dim = 0.0;
                    if (xi < 1.0 - kVeryTiny)     // a lone species has Ds = 0
                        Dim = (Ds[q] > 1e-280 && Ds[q] < 1e280)
                                  ? near_div(1.0 - xi, Ds[q], fast_rcp(Ds[q])) * scale
                                  : (1.0 - xi) * scale / Ds[q];
                    if (isinf(Dim)) Dim = 0.0;
                    D[(int64_t)i * n + cell] = Dim;
                }
            }
            mum += (wm[0] + wm[1]) + (wm[2] + wm[3]);
            kappam += (wk[0] + wk[1]) + (wk[2] + wk[3]);
        }
        part[l * B] = mum;
        part[(L + l) * B] = kappam;
        __syncthreads();
        if (l == 0 && live) {
            double mum = 0.0, kappam = 0.0, cp = 0.0;
            for (int k = 0; k < L; ++k) {
                mum += part[k * B];
                kappam += part[(L + k) * B];
                cp += part[(2 * L + k) * B];
            }
            if (mu) mu[cell] = mum;
            if (kappa) kappa[cell] = kappam;
            if (cpm) cpm[cell] = cp;
        }
    }
}

int launch_properties(const DevMech &m, int64_t n, const double *T, const double *p,
                      const double *Y, double *ha, double *cp, double *mu, double *kappa,
                      double *D, cudaStream_t st, std::string &err) {
    if (m.nsp > kPropMaxSp) {
        err = "property kernel is built for at most 64 species";
        return HC_E_UNSUPPORTED;
    }
    if (!m.ptab) {
        err = "mechanism has no transport pair tables";
        return HC_E_INVALID;
    }
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // up to four threads a cell (fewer where the mechanism has fewer row blocks);
    // the widest block that fits and leaves no SM without cells
    const int NB = (m.nsp + 3) / 4, L = std::min(4, NB);
    int B = kPropCells;
    auto smem = [&](int b) { return sizeof(double) * (12 * (size_t)NB * m.nsp + 4 * NB + kPropSp * m.nsp + (2 * m.nsp + 3 * L) * (size_t)b); };
    while (B > 32 && (smem(B) > kMaxSmem || (n + B - 1) / B < sms)) B /= 2;
    const size_t sm = smem(B);
    if (int rc = allow_smem<properties_kernel>(err)) return rc;
    int per_sm = 0;
    HC_LCUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, properties_kernel, B * L, sm));
    if (per_sm < 1) {
        err = "property kernel does not fit on an SM";
        return HC_E_UNSUPPORTED;
    }
    const int64_t tiles = (n + B - 1) / B;
    const int64_t blocks = std::min<int64_t>(tiles, (int64_t)sms * per_sm);
    properties_kernel<<<(unsigned)blocks, B * L, sm, st>>>(m, n, T, p, Y, ha, cp, mu, kappa, D, L, tiles);
    HC_LCUDA(cudaGetLastError());
    return HC_OK;
}

// Temperature from the mixture's mass enthalpy at constant pressure,
// thermoList::THa_p (thermoList.cpp:501-533): Newton steps
// T <- limit(T - (h(T) - ha) / cp(T)) from T0 until |dT| <= T0 tol, at most
// max_iter + 1 steps; limit clamps to [TLow, THigh] and sets the flag
// (0 below, 1 inside, 2 above; thermoList.cpp:152-163). Thread per cell.
__global__ void t_from_ha_kernel(const __grid_constant__ DevMech m, int64_t n,
                                 const double *__restrict__ ha, const double *__restrict__ Y,
                                 const double *__restrict__ T0, double TLow, double THigh,
                                 double tol, int max_iter, double *__restrict__ Tout,
                                 int32_t *__restrict__ flag) {
    const int nsp = m.nsp;
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n;
         c += (int64_t)gridDim.x * blockDim.x) {
        double Tnew = T0[c];
        const double Ttol = T0[c] * tol;
        int it = 0, f = 1;
        while (true) {
            const double Test = Tnew;
            double hm = 0.0, cpm = 0.0;
            for (int i = 0; i < nsp; ++i) {
                double cp, h;
                species_cp_h(m, i, Test, cp, h);
                const double yi = Y[(int64_t)i * n + c];
                hm += h * yi;
                cpm += cp * yi;
            }
            const double v = Test - (hm - ha[c]) / cpm;
            if (v < TLow) {
                f = 0;
                Tnew = TLow;
            } else if (v > THigh) {
                f = 2;
                Tnew = THigh;
            } else {
                f = 1;
                Tnew = v;
            }
            if (it++ > max_iter) break;
            if (!(fabs(Tnew - Test) > Ttol)) break;
        }
        Tout[c] = Tnew;
        if (flag) flag[c] = f;
    }
}

// thermoList::TEa_rho (thermoList.inl:343-348 through thermoList.cpp:501-533):
// the same Newton iteration on the mixture's internal energy at fixed
// density, e(T) = sum_i Y_i h_i(T) - p / rho with p = rho Rm T, and
// de/dT = sum_i Y_i cp_i(T) - Rm (thermoList.inl:145-162, 302-306)
__global__ void t_from_ea_kernel(const __grid_constant__ DevMech m, int64_t n,
                                 const double *__restrict__ ea, const double *__restrict__ Y,
                                 const double *__restrict__ rho, const double *__restrict__ T0,
                                 double TLow, double THigh, double tol, int max_iter,
                                 double *__restrict__ Tout, int32_t *__restrict__ flag) {
    const int nsp = m.nsp;
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n;
         c += (int64_t)gridDim.x * blockDim.x) {
        double w = 0.0;
        for (int i = 0; i < nsp; ++i) w += Y[(int64_t)i * n + c] / ldg(&m.W[i]);
        const double Rm = kRu / (1.0 / hmax(w, kVeryTiny));
        const double r = rho[c];
        double Tnew = T0[c];
        const double Ttol = T0[c] * tol;
        int it = 0, f = 1;
        while (true) {
            const double Test = Tnew;
            double hm = 0.0, cpm = 0.0;
            for (int i = 0; i < nsp; ++i) {
                double cp, h;
                species_cp_h(m, i, Test, cp, h);
                const double yi = Y[(int64_t)i * n + c];
                hm += h * yi;
                cpm += cp * yi;
            }
            const double em = hm - (r * Rm * Test) / r;
            const double cvm = cpm - Rm;
            const double v = Test - (em - ea[c]) / cvm;
            if (v < TLow) {
                f = 0;
                Tnew = TLow;
            } else if (v > THigh) {
                f = 2;
                Tnew = THigh;
            } else {
                f = 1;
                Tnew = v;
            }
            if (it++ > max_iter) break;
            if (!(fabs(Tnew - Test) > Ttol)) break;
        }
        Tout[c] = Tnew;
        if (flag) flag[c] = f;
    }
}

int launch_t_from_ea(const DevMech &m, int64_t n, const double *ea, const double *Y,
                     const double *rho, const double *T0, double TLow, double THigh, double *T,
                     int32_t *flag, cudaStream_t st, std::string &err) {
    if (n <= 0) return HC_OK;
    const int64_t blocks = (n + 127) / 128;
    t_from_ea_kernel<<<(unsigned)(blocks < 148 * 64 ? blocks : 148 * 64), 128, 0, st>>>(
        m, n, ea, Y, rho, T0, TLow, THigh, 1.0e-4, 100, T, flag);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        err = std::string("t_from_ea_kernel: ") + cudaGetErrorString(e);
        return HC_E_CUDA;
    }
    return HC_OK;
}

int launch_t_from_ha(const DevMech &m, int64_t n, const double *ha, const double *Y,
                     const double *T0, double TLow, double THigh, double *T, int32_t *flag,
                     cudaStream_t st, std::string &err) {
    if (n <= 0) return HC_OK;
    const int64_t blocks = (n + 127) / 128;
    t_from_ha_kernel<<<(unsigned)(blocks < 148 * 64 ? blocks : 148 * 64), 128, 0, st>>>(
        m, n, ha, Y, T0, TLow, THigh, 1.0e-4, 100, T, flag);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        err = std::string("t_from_ha_kernel: ") + cudaGetErrorString(e);
        return HC_E_CUDA;
    }
    return HC_OK;
}

}  // namespace hc
