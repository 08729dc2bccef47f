// Warp-per-cell (wcell.cuh) and segment-per-cell (scell.cuh) integrators:
// instantiations for N <= 10 and 16 unknowns and their launch.
#include <algorithm>
#include <string>

#include "../../include/hurchem_b200.h"
#include "launch.cuh"
#include "scell.cuh"
#include "wcell.cuh"

namespace hc {

// most warps per block whose shared memory fits (0: not even one)
template <int N>
static int w_warps(const WMech &m, const IntegratorParams &P) {
    int w = kWWarps;
    while (w > 0 && w6_smem_bytes<N>(m, w, P.auto_update_jacobian != 0) > kMaxSmem) w /= 2;
    return w;
}

bool launch_w_fits(const WMech &m, const IntegratorParams &P) {
    return (m.nsp + 1 <= 10 ? w_warps<10>(m, P) : w_warps<16>(m, P)) > 0;
}

template <int N, int BLOCKS, bool AUTO>
static int launch_w(const WMech &m, int num_sms, const IntegratorParams &P, const CellIO &io,
                    cudaStream_t st, std::string &err) {
    auto kern = integrate_w_kernel<N, BLOCKS, AUTO>;
    const int warps = w_warps<N>(m, P);
    const size_t sm = w6_smem_bytes<N>(m, warps, P.auto_update_jacobian != 0);
    int per_sm = 0;
    if (warps > 0) {
        if (int rc = allow_smem<integrate_w_kernel<N, BLOCKS, AUTO>>(err)) return rc;
        HC_LCUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * warps, sm));
    }
    if (per_sm < 1) {
        err = "warp-per-cell kernel does not fit on an SM";
        return HC_E_UNSUPPORTED;
    }
    // fewer cells than warps: one block per cell until every SM has its blocks,
    // so that few cells do not share an SM's issue slots
    const int64_t grid = std::min<int64_t>(io.nqueue, (int64_t)per_sm * num_sms);
    if (grid <= 0) return HC_OK;
    kern<<<(unsigned)grid, 32 * warps, sm, st>>>(m, P, io);
    HC_LCUDA(cudaGetLastError());
    return HC_OK;
}

// One block of eight warps per SM and no spills, or two with 128 registers a thread.
// A flow step ends with its stiffest cells, whose iterations the first build does in
// 4.5 us against 6.5 us; only when the cells go round many times does the second's
// larger number in flight pay. First / second build in ms, Dirichlet cells at 1e-7 s, mixed
// cells at 1e-6 s and at 1e-5 s: 12,288 cells 116 / 158, 79 / 100 and 320 / 421; 18,944
// 175 / 180, 121 / 114 and 493 / 513; 37,888 348 / 309, 243 / 211 and 980 / 859. So the
// line lies at 8 cells for each of the second's warps. Where shared memory holds one block
// only (mechanisms with many reactions) the second build would be the first with spills:
// 15 species / 45 reactions, first / second: 20,000 cells 266 / 320 ms, 40,000 486 / 577.
template <int N>
static int launch_w(const WMech &m, int num_sms, const IntegratorParams &P, const CellIO &io,
                    cudaStream_t st, std::string &err) {
    const int warps = w_warps<N>(m, P);
    const size_t sm = w6_smem_bytes<N>(m, warps, P.auto_update_jacobian != 0);
    const bool two = 2 * (sm + 1024) <= 228 * 1024;       // blocks an SM by shared memory
    const bool few = !two || io.nqueue < (int64_t)8 * 2 * warps * num_sms;
    if (P.auto_update_jacobian)
        return few ? launch_w<N, 1, true>(m, num_sms, P, io, st, err) : launch_w<N, 2, true>(m, num_sms, P, io, st, err);
    return few ? launch_w<N, 1, false>(m, num_sms, P, io, st, err) : launch_w<N, 2, false>(m, num_sms, P, io, st, err);
}

int launch_integrate_w(const WMech &m, int num_sms, const IntegratorParams &P, const CellIO &io,
                       cudaStream_t st, std::string &err) {
    const int N = m.nsp + 1;
    if (N <= 10) return launch_w<10>(m, num_sms, P, io, st, err);
    if (N <= 16) return launch_w<16>(m, num_sms, P, io, st, err);
    err = "warp-per-cell kernel takes nsp + 1 <= 16";
    return HC_E_UNSUPPORTED;
}

template <int N>
static int launch_s(const WMech &m, int num_sms, const IntegratorParams &P, const CellIO &io,
                    cudaStream_t st, std::string &err) {
    auto kern = integrate_s_kernel<N>;
    constexpr int G = SLayout<N>::G;
    const size_t sm = w_tables_bytes(m.nsp, m.nrc, m.nrc32, m.nent, m.ntb, m.njob32) +
                      sizeof(double) * SLayout<N>::doubles(m.nrc, m.njob) * G * kSWarps;
    int per_sm = 0;
    if (sm <= kMaxSmem) {
        if (int rc = allow_smem<integrate_s_kernel<N>>(err)) return rc;
            HC_LCUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * kSWarps, sm));
    }
    if (per_sm < 1) {
        err = "segment-per-cell kernel does not fit on an SM";
        return HC_E_UNSUPPORTED;
    }
    const int64_t blocks_needed = (io.nqueue + G * kSWarps - 1) / (G * kSWarps);
    const int64_t grid = std::min<int64_t>(blocks_needed, (int64_t)per_sm * num_sms);
    if (grid <= 0) return HC_OK;
    kern<<<(unsigned)grid, 32 * kSWarps, sm, st>>>(m, P, io);
    HC_LCUDA(cudaGetLastError());
    return HC_OK;
}

int launch_integrate_s(const WMech &m, int num_sms, const IntegratorParams &P, const CellIO &io,
                       cudaStream_t st, std::string &err) {
    const int N = m.nsp + 1;
    if (N <= 10) return launch_s<10>(m, num_sms, P, io, st, err);
    if (N <= 16) return launch_s<16>(m, num_sms, P, io, st, err);
    err = "segment-per-cell kernel takes nsp + 1 <= 16";
    return HC_E_UNSUPPORTED;
}

}  // namespace hc
