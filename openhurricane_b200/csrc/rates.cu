// Explicit and point-implicit chemistry source terms, L lanes per cell.
//
//   omega_i W_i            chemistrySource::calculateSourceTerms (chemistrySource.cpp:1370-1406)
//   Ri, diag_j             ::calculateSourceTermsImp with withoutLastSpec = true (:1412-1450, 422-480)
//   q, Kc, DqDci, DqDT     reactionTypes.cpp:178-445, 843-876
//
// What bounds it: the FP64 pipe and the latency of the rate laws' exp and log. Lanes
// share a cell's species and reactions, each reaction's tables come as one 16-byte
// and one 32-byte load from shared memory, a lane sums its reactions' contributions
// in its own column of shared memory and the columns are added last. Measured
// (B200) against a 32- or 64-lane group per cell with list walks: 1,048,576 cells of
// 9 species 3777 -> 219 us, 65,536 of 53 species 3471 -> 397 us, implicit terms
// of 262,144 cells of 9 species (which formed the whole Jacobian) 3292 -> 152 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "../../include/hurchem_b200.h"
#include "launch.cuh"
#include "rates.cuh"

namespace hc {

namespace {

constexpr int kThreads = 128;

// doubles of shared memory: per cell {c, g} (, d) and per lane f (, diag, dq/dT), and the mixture sums
__host__ __device__ constexpr int cell_doubles(int nsp, int L, bool imp) {
    return (nsp + 1) * (imp ? 3 + 3 * L : 2 + L) + (imp ? 2 * L : 0);
}
__host__ __device__ constexpr size_t table_bytes(int nrc) { return (size_t)nrc * (sizeof(int4) + sizeof(double4)); }

// L: lanes per cell (compile time: the cells of a block, the species' stride, are a shift)
template <bool IMP, int L>
__global__ void __launch_bounds__(kThreads, IMP ? 4 : 7)
rates_kernel(const __grid_constant__ RMech m, const __grid_constant__ DevMech dm, int64_t n,
             const double *__restrict__ T_, const double *__restrict__ rho_, const double *__restrict__ Y,
             double *__restrict__ Ri, double *__restrict__ diag) {
    extern __shared__ __align__(16) double smem_r[];
    const int nsp = m.nsp, nrc = m.nrc, S = nsp + 1;
    double4 *rate = reinterpret_cast<double4 *>(smem_r);
    int4 *code = reinterpret_cast<int4 *>(rate + nrc);
    for (int r = threadIdx.x; r < nrc; r += kThreads) {
        rate[r] = m.rate[r];
        code[r] = m.code[r];
    }
    constexpr int B = kThreads / L;               // cells of the block
    const int cl = threadIdx.x % B, l = threadIdx.x / B;
    double2 *cg = reinterpret_cast<double2 *>(code + nrc) + cl;
    double *d = reinterpret_cast<double *>(code + nrc) + 2 * S * B + cl;
    double *f0 = d + (IMP ? S * B : 0);           // [L][S]
    double *f = f0 + l * S * B;
    double *dg = f + L * S * B, *jt = dg + L * S * B;   // IMP only
    double *part = f0 + 3 * L * S * B;            // IMP only: sum Y cp, sum Y / W per lane
    const int64_t cell0 = (int64_t)blockIdx.x * B + cl;
    const bool live = cell0 < n;
    const int64_t cell = live ? cell0 : n - 1;
    const double T = T_[cell], rho = rho_[cell];
    const double invT = frcp(hmax(T, kTiny)), logT = fast_log(T), lT = (T > kTiny) ? logT : -34.538776394910684;
    double ycp = 0.0, yw = 0.0;
    for (int i = l; i < nsp; i += L) {
        const double *t = m.th + kRTh * i;
        const double *a = species_range(t, T);
        const double Yi = Y[(int64_t)i * n + cell];
        cg[i * B] = make_double2(hmax(rho * Yi * ldg(&t[4]), 0.0), species_gibbs(t, a, T, lT));
        if (IMP) {
            // (dG0/dT - G0/T) / Ru: -h/T inside the fitted range; outside, where
            // the reference clamps cp but not s and g, the difference of the two cp
            double hc, cp;
            species_hcp(t, T, hc, cp);
            const double a0 = ldg(&a[0]), a1 = ldg(&a[1]), a2 = ldg(&a[2]), a3 = ldg(&a[3]), a4 = ldg(&a[4]);
            const double h = T * (a0 + T * (a1 * 0.5 + T * (a2 * (1.0 / 3.0) + T * (a3 * 0.25 + T * (a4 * 0.2))))) + ldg(&a[5]);
            d[i * B] = (cp - (a0 + T * (a1 + T * (a2 + T * (a3 + T * a4))))) - h * invT;
            ycp += Yi * cp * ldg(&t[4]);
            yw += Yi * ldg(&t[4]);
        }
    }
    if (l == 0) {
        cg[nsp * B] = make_double2(1.0, 0.0);
        if (IMP) d[nsp * B] = 0.0;
    }
    if (IMP) {
        part[(2 * l) * B] = ycp;
        part[(2 * l + 1) * B] = yw;
    }
    for (int i = 0; i < S; ++i) {
        f[i * B] = 0.0;
        if (IMP) dg[i * B] = jt[i * B] = 0.0;
    }
    __syncthreads();
    const double iWL = IMP ? ldg(&m.th[kRTh * (nsp - 1) + 4]) : 0.0;
    double ctot = 0.0;
    for (int i = 0; i < nsp; ++i) ctot += cg[i * B].x;
    for (int r = l; r < nrc; r += L) {
        const double4 k4 = rate[r];
        const int4 w = code[r];
        const RxnVals v = rxn_eval<IMP, true>(m, w, k4, [cg](int i) { return cg[i * B]; },
                                              [cg](int i) { return cg[i * B].x; }, [d](int i) { return d[i * B]; }, T,
                                              invT, logT, ctot);
        const int i0 = w.x & 255, i1 = (w.x >> 8) & 255, i2 = (w.x >> 16) & 255;
        const int j0 = w.y & 255, j1 = (w.y >> 8) & 255, j2 = (w.y >> 16) & 255;
        double xf = 1.0, xb = 1.0;                // multiplicities of the first factors, rarely not 1
        if ((w.z & (15 << kRmf)) != (1 << kRmf | 1 << kRmb)) {
            xf = (double)((w.z >> kRmf) & 3);
            xb = (double)((w.z >> kRmb) & 3);
        }
        f[i0 * B] -= xf * v.q;
        if (w.z & 2) f[i1 * B] -= v.q;
        if (w.z & 4) f[i2 * B] -= v.q;
        f[j0 * B] += xb * v.q;
        if (w.z & 16) f[j1 * B] += v.q;
        if (w.z & 32) f[j2 * B] += v.q;
        if (!IMP) continue;
        // d q / d c_L of the last species, whose concentration follows from the others
        const bool eff = (w.x >> 24) != kArrhenius;
        const int last = (w.z >> kRlast) & 7;
        double dL = eff ? ldg(&dm.eff[(int64_t)r * nsp + nsp - 1]) * v.g : 0.0;
#pragma unroll
        for (int k = 0; k < 6; ++k)
            if (k == last) dL += v.d[k];
        auto add = [&](int i, double nu, double dc) {
            const double ei = (eff && i < nsp) ? ldg(&dm.eff[(int64_t)r * nsp + i]) * v.g : 0.0;
            const double wr = ldg(&dm.W[i < nsp ? i : 0]) * iWL;
            dg[i * B] += nu * ((dc + ei) - wr * dL);
            jt[i * B] += nu * v.dq;
        };
        add(i0, -xf, v.d[0]);
        if (w.z & 2) add(i1, -1.0, v.d[1]);
        if (w.z & 4) add(i2, -1.0, v.d[2]);
        add(j0, xb, v.d[3]);
        if (w.z & 16) add(j1, 1.0, v.d[4]);
        if (w.z & 32) add(j2, 1.0, v.d[5]);
    }
    __syncthreads();
    if (!live) return;
    double cv = 0.0, eL = 0.0, rcv = 0.0;
    if (IMP) {
        double a = 0.0, b = 0.0;
        for (int k = 0; k < L; ++k) {
            a += part[(2 * k) * B];
            b += part[(2 * k + 1) * B];
        }
        cv = kRu * (a - b);
        double cp, h;
        species_hcp(m.th + kRTh * (nsp - 1), T, h, cp);
        eL = kRu * iWL * (h - T);
        rcv = 1.0 / (rho * cv);
    }
    for (int i = l; i < nsp; i += L) {
        double v = 0.0, dd = 0.0, jj = 0.0;
        for (int k = 0; k < L; ++k) {
            v += f0[(k * S + i) * B];
            if (IMP) {
                dd += f0[((L + k) * S + i) * B];
                jj += f0[((2 * L + k) * S + i) * B];
            }
        }
        const double W = ldg(&dm.W[i]);
        Ri[(int64_t)i * n + cell] = v * W;
        if (IMP && i < nsp - 1) {
            double cp, h;
            species_hcp(m.th + kRTh * i, T, h, cp);
            diag[(int64_t)i * n + cell] = dd + jj * W * (eL - kRu * ldg(&m.th[kRTh * i + 4]) * (h - T)) * rcv;
        }
    }
}

}  // namespace

static size_t rates_smem(int nsp, int nrc, int L, bool imp) {
    return table_bytes(nrc) + sizeof(double) * (size_t)cell_doubles(nsp, L, imp) * (kThreads / L);
}

bool rates_fit(int nsp, int nrc, bool implicit) { return rates_smem(nsp, nrc, 32, implicit) <= kMaxSmem; }

// Lanes per cell. Many cells: as few lanes as shared memory lets 256 threads of
// an SM have (each lane brings its own accumulators), and twice as many where that
// puts a third more threads on the SM (explicit terms, 9 species: one lane, 53:
// four; implicit, 9 species: two). Few cells: more lanes, each with fewer reactions
// in its chain, while all threads run at once. Measured in us, lanes 1 2 4 8 16 32:
//   9 species, explicit,  262,144 cells:  62.0  66.0  74.2  96.9 144   238
//                          65,536 cells:  23.1  21.1  23.0  29.2  40.8  64.1
//                           8,192 cells:  16.9  12.7  10.4   9.7   9.3  12.7
//   9 species, implicit,  262,144 cells:   159   146   168   220   357   672
//                          65,536 cells:  64.3  43.2  49.8  60.2  93.6   171
//                          16,384 cells:  29.5  21.2  17.0  21.1  29.4  47.9
//   53 species, explicit,  65,536 cells:   720   626   380   414   487   489
//                           8,192 cells:   185  99.4  59.0  64.1  74.1  68.6
//                           2,048 cells:   183  99.0  53.8  31.3  23.0  29.2
static int choose_lanes(int nsp, int nrc, int64_t n, int num_sms, bool imp) {
    auto places = [&](int L) {
        const size_t sm = rates_smem(nsp, nrc, L, imp);
        if (sm > kMaxSmem) return 0;
        return kThreads * std::min((int)(228 * 1024 / (sm + 1024)), imp ? 4 : 7);   // registers: 4 and 7 blocks
    };
    int L = 1;
    while (L < 32 && places(L) < 256) L *= 2;
    if (places(L) < 256)
        for (L = 1; L < 32 && places(L) == 0;) L *= 2;
    while (L < 32 && 3 * places(2 * L) >= 4 * places(L)) L *= 2;
    while (L < 32 && 2 * L <= nrc && n * 2 * L <= (int64_t)num_sms * places(2 * L)) L *= 2;
    return L;
}

template <int L>
static int launch_lanes(const RMech &m, const DevMech &dm, int num_sms, int64_t n, const double *T, const double *rho,
                        const double *Y, double *Ri, double *diag, cudaStream_t st, std::string &err) {
    const bool imp = diag != nullptr;
    constexpr int B = kThreads / L;
    const unsigned grid = (unsigned)((n + B - 1) / B);
    const size_t sm = rates_smem(m.nsp, m.nrc, L, imp);
    // a block alone on its SM and within the default limit goes without: 257 cells of 9
    // species, a call bound by its host side, 8.4 -> 8.1 us (it varies by 3 %)
    if (sm > 48 * 1024 || grid > (unsigned)num_sms) {
        const int rc = imp ? allow_smem<rates_kernel<true, L>>(err) : allow_smem<rates_kernel<false, L>>(err);
        if (rc != HC_OK) return rc;
    }
    if (imp) rates_kernel<true, L><<<grid, kThreads, sm, st>>>(m, dm, n, T, rho, Y, Ri, diag);
    else rates_kernel<false, L><<<grid, kThreads, sm, st>>>(m, dm, n, T, rho, Y, Ri, nullptr);
    HC_LCUDA(cudaGetLastError());
    return HC_OK;
}

int launch_rates(const RMech &m, const DevMech &dm, int num_sms, int64_t n, const double *T, const double *rho,
                 const double *Y, double *Ri, double *diag, cudaStream_t st, std::string &err) {
    switch (choose_lanes(m.nsp, m.nrc, n, num_sms, diag != nullptr)) {
    case 1: return launch_lanes<1>(m, dm, num_sms, n, T, rho, Y, Ri, diag, st, err);
    case 2: return launch_lanes<2>(m, dm, num_sms, n, T, rho, Y, Ri, diag, st, err);
    case 4: return launch_lanes<4>(m, dm, num_sms, n, T, rho, Y, Ri, diag, st, err);
    case 8: return launch_lanes<8>(m, dm, num_sms, n, T, rho, Y, Ri, diag, st, err);
    case 16: return launch_lanes<16>(m, dm, num_sms, n, T, rho, Y, Ri, diag, st, err);
    default: return launch_lanes<32>(m, dm, num_sms, n, T, rho, Y, Ri, diag, st, err);
    }
}

}  // namespace hc
