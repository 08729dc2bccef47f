// Block-per-cell integrator and Jacobian (bcell.cuh): instantiations by the
// number of unknowns and their launch.
#include <algorithm>
#include <string>

#include "../../include/hurchem_b200.h"
#include "bcell.cuh"
#include "launch.cuh"
#include "variants.h"

namespace hc {

// columns per warp and rows per lane: N + 1 <= 8 CPW columns, N <= 32 SL rows
#define HC_B_DISPATCH(N, FN, ...)                       \
    ((N) <= 32 ? FN<5, 1>(__VA_ARGS__) : (N) <= 55 ? FN<7, 2>(__VA_ARGS__) : FN<9, 2>(__VA_ARGS__))

template <int CPW, int SL>
static size_t b_smem(const RMech &m, const BMech &b) {
    return sizeof(double) * BLayout<CPW, SL>::doubles(m, b);
}

bool launch_b_fits(const RMech &m, const BMech &b) {
    const int N = m.nsp + 1;
    return N <= 64 && HC_B_DISPATCH(N, b_smem, m, b) <= kMaxSmem;
}

template <auto Kernel>
static int b_grid(size_t sm, int num_sms, int64_t n, int64_t &grid, std::string &err) {
    int per_sm = 0;
    if (int rc = allow_smem<Kernel>(err)) return rc;
    HC_LCUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, Kernel, kBThreads, sm));
    if (per_sm < 1) {
        err = "block-per-cell kernel does not fit on an SM";
        return HC_E_UNSUPPORTED;
    }
    grid = std::min<int64_t>(n, (int64_t)per_sm * num_sms);
    return HC_OK;
}

template <int CPW, int SL>
static int launch_bi(const RMech &m, const BMech &b, int num_sms, const IntegratorParams &P, const CellIO &io,
                     cudaStream_t st, std::string &err) {
    const size_t sm = b_smem<CPW, SL>(m, b);
    int64_t grid = 0;
    const int rc = b_grid<integrate_b_kernel<CPW, SL>>(sm, num_sms, io.nqueue, grid, err);
    if (rc != HC_OK || grid <= 0) return rc;
    integrate_b_kernel<CPW, SL><<<(unsigned)grid, kBThreads, sm, st>>>(m, b, P, io);
    HC_LCUDA(cudaGetLastError());
    return HC_OK;
}

int launch_integrate_b(const RMech &m, const BMech &b, int num_sms, const IntegratorParams &P, const CellIO &io,
                       cudaStream_t st, std::string &err) {
    return HC_B_DISPATCH(m.nsp + 1, launch_bi, m, b, num_sms, P, io, st, err);
}

template <int CPW, int SL>
static int launch_bj(const RMech &m, const BMech &b, int num_sms, int64_t n, const double *c, const double *T,
                     double *dydt, double *J, cudaStream_t st, std::string &err) {
    const size_t sm = b_smem<CPW, SL>(m, b);
    int64_t grid = 0;
    const int rc = b_grid<jacobian_b_kernel<CPW, SL>>(sm, num_sms, n, grid, err);
    if (rc != HC_OK || grid <= 0) return rc;
    IntegratorParams P{};
    jacobian_b_kernel<CPW, SL><<<(unsigned)grid, kBThreads, sm, st>>>(m, b, P, n, c, T, dydt, J);
    HC_LCUDA(cudaGetLastError());
    return HC_OK;
}

int launch_jacobian_b(const RMech &m, const BMech &b, int num_sms, int64_t n, const double *c, const double *T,
                      double *dydt, double *J, cudaStream_t st, std::string &err) {
    return HC_B_DISPATCH(m.nsp + 1, launch_bj, m, b, num_sms, n, c, T, dydt, J, st, err);
}

}  // namespace hc
