// Block-per-cell implicit-Euler integrator and Jacobian evaluation for
// mechanisms of 17 .. 64 unknowns whose reactions have the direct form
// (rates.cuh), FP64, both reactors.
//
// Eight warps (256 threads) work on one cell. What bounds it: one Newton
// iteration of one cell, a chain of N dependent pivot steps between the
// evaluations; the flow step lasts as long as its stiffest cell. So:
//
//  * reactions: warps take tasks of 32 reactions from a list that the host
//    balanced by rate form (fall-off costs several times a plain one). Each lane
//    writes a record (q, dq/dT, the efficiencies' factor g, dq/dc of each
//    factor, g times each listed efficiency) to shared memory;
//  * J, f and the column of T: every nonzero is a signed sum of record values (a
//    coefficient of 2 is two terms), read from a flat term list: items sorted by
//    length, 32 of them in lock step per warp, two 16-bit terms a word. The third
//    bodies' dense columns are rank one: where most efficiencies are 1 their sum
//    over the reactions is one number per row, added when the row is used, and
//    only the listed differences are terms;
//  * temperature row: two threads per column sum h_i J_ij;
//  * Gaussian elimination with partial pivoting on [I - dt J | rhs] in registers: a warp
//    owns a block of columns of ALL rows (rows on lanes), so the pivot search is a
//    warp reduction. The warp that owns the current columns runs ahead and
//    publishes each step's multipliers and pivot; the warps to its right apply
//    them to their columns behind a named barrier at which it only arrives. The
//    rows of U stay in their lanes, each column of U goes to shared memory as its
//    owner passes it, and the warp with the right-hand side substitutes back.
//    (Gauss-Jordan needs no substitution but is not backward stable, see wcell.cuh.)
//
// Measured (B200, 53 species / 325 reactions): one Newton iteration of one cell takes
// 20.5 us with two cells on an SM (before: 143 us in the cell group of 64 lanes; with
// four warps a cell 28.5 us), a pivot step 450 cycles and a step of the substitution
// about 60; 768 cells, flow step of 1e-7 s: 945 -> 244 ms; 8191 Jacobians and
// right-hand sides: 1487 -> 283 us.
#pragma once

#include "rates.cuh"
#include "stepctl.cuh"

namespace hc {

constexpr int kBWarps = 8, kBThreads = 32 * kBWarps;
constexpr int kBBlocks = 2;          // blocks an SM: 128 registers a thread

// Tables beside RMech (pack_b, capi.cu). Records: kBd + F + R values per
// reaction (F, R: most factors a side), then the listed efficiencies' values; `zero` is a
// place past them and past the pivot steps' multipliers, which nothing writes.
constexpr int kBSteps = 10 * 64;
// place of column k of U (k rows in pivot order) behind them
__host__ __device__ constexpr int b_ucol(int k) { return kBSteps + k * (k - 1) / 2; }
struct BMech {
    int32_t nf, stride;      // forward factors of a record, doubles per record
    int32_t ndv;             // listed efficiencies
    int32_t zero;            // the zero that padding terms read
    int32_t ld;              // row stride of J: nsp species, T, f, odd
    const int32_t *task;     // [tasks][32] reaction of the lane, -1: none
    const int32_t *tptr;     // [kBWarps + 1] tasks of each warp
    // item groups in pairs of equal length, read from the block's shared memory
    const int32_t *gptr;     // [kBWarps + 1] pairs of each warp
    int32_t npair, nword;    // pairs; words of a lane over all pairs
    const int32_t *pair;     // [npair] first word | words of a lane << 16; a word holds the pair's two groups
    const uint32_t *dst;     // [npair][32] the two places: J region, or kBRow | row for a third-body sum
    const uint2 *term;       // [nword][32] per group two terms: record place | sign << 15
};
constexpr uint32_t kBRow = 0x8000u;
enum BRec : int { kBq = 0, kBdq = 1, kBg = 2, kBd = 3 };

template <int CPW, int SL>
struct BLayout {
    static constexpr int kS = 66;                       // species slots (nsp <= 63, the absent factor's slot)
    static constexpr int kC = 0, kD = 2 * kS, kH = 3 * kS, kCP = 4 * kS, kCM = 5 * kS;
    static constexpr int kX = 6 * kS;                   // solution, rows' third-body sums
    static constexpr int kRow = 7 * kS;
    static constexpr int kT = 8 * kS;                   // column sums of h J (66), then the scalars
    static constexpr int kSc = 9 * kS;                  // [8]
    static constexpr int kPV = kSc + 8;                 // pivots: 1 / pivot [64], rows (int) [64]
    static constexpr int kTab = kPV + 96;               // the term lists
    // the pivot steps' multipliers (CPW steps of 64) lie over the records, dead by then
    static_assert(CPW * 64 <= kBSteps && CPW < 15, "room and barriers of the pivot steps");
    __host__ __device__ static int tables(const BMech &b) { return 32 * b.nword + 16 * b.npair + ((b.npair + 3) / 4) * 2; }
    __host__ __device__ static int records(const RMech &r, const BMech &b) {
        return (b.zero + 2) & ~1;
    }
    __host__ __device__ static size_t doubles(const RMech &r, const BMech &b) {
        return (size_t)kTab + tables(b) + records(r, b) + (size_t)r.nsp * b.ld + 2;
    }
};

__device__ __forceinline__ void b_sync() { asm volatile("bar.sync 0;" ::: "memory"); }

template <int CPW, int SL>
struct BCell {
    using L = BLayout<CPW, SL>;
    static constexpr int E = SL;         // rows lane and lane + 32; every warp carries all elements
    static constexpr unsigned full = 0xffffffffu;
    const RMech &m;
    const BMech &bm;
    const IntegratorParams &P;
    double *s;
    int lane, warp, nsp, N;
    double cvRu;
    double *rec, *J;
    const uint2 *term;
    const uint32_t *dst;
    const int32_t *pair;
    double a[SL][CPW];
    double f[SL];

    __device__ BCell(const RMech &mm, const BMech &b, const IntegratorParams &pp, double *sm)
        : m(mm), bm(b), P(pp), s(sm), lane(threadIdx.x & 31), warp(threadIdx.x >> 5), nsp(mm.nsp), N(mm.nsp + 1) {
        cvRu = (pp.reactor == 1) ? kRu : 0.0;
        term = reinterpret_cast<const uint2 *>(s + L::kTab);
        dst = reinterpret_cast<const uint32_t *>(s + L::kTab + 32 * bm.nword);
        pair = reinterpret_cast<const int32_t *>(dst + 32 * bm.npair);
        rec = s + L::kTab + L::tables(bm);
        J = rec + L::records(m, bm);
    }

    __device__ __forceinline__ bool has(int e) const { return lane + 32 * e < N; }
    __device__ __forceinline__ int elem(int e) const { return lane + 32 * e; }
    __device__ __forceinline__ bool f_here() const { return true; }
    __device__ __forceinline__ double T_of(const double (&y)[E]) const {
        return __shfl_sync(full, (SL == 2 && nsp >= 32) ? y[SL - 1] : y[0], nsp & 31);
    }
    __device__ __forceinline__ double sum(double v) const {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(full, v, o);
        return v;
    }
    __device__ __forceinline__ double max_nonneg(double v) const {
        const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
        const unsigned mh = __reduce_max_sync(full, hi);
        const unsigned ml = __reduce_max_sync(full, hi == mh ? lo : 0u);
        return __hiloint2double((int)mh, (int)ml);
    }
    __device__ __forceinline__ int first_bad(const double (&x)[E]) const {
        int first = 1 << 30;
#pragma unroll
        for (int e = E - 1; e >= 0; --e) {
            const unsigned bad = __ballot_sync(full, has(e) && !finite(x[e]));
            if (bad) first = 32 * e + __ffs(bad) - 1;
        }
        return first;
    }
    static constexpr bool kAuto = false;   // autoUpdateJacobian takes the cell group

    // once per block: the places nothing writes later, the term lists
    __device__ void init() {
        const int n = (int)L::doubles(m, bm);
        for (int i = threadIdx.x; i < n; i += kBThreads) s[i] = 0.0;
        b_sync();
        for (int i = threadIdx.x; i < 32 * bm.nword; i += kBThreads) const_cast<uint2 *>(term)[i] = __ldg(&bm.term[i]);
        for (int i = threadIdx.x; i < 32 * bm.npair; i += kBThreads) const_cast<uint32_t *>(dst)[i] = __ldg(&bm.dst[i]);
        for (int i = threadIdx.x; i < bm.npair; i += kBThreads) const_cast<int32_t *>(pair)[i] = __ldg(&bm.pair[i]);
        if (threadIdx.x == 0) s[L::kC + 2 * nsp] = 1.0;
        b_sync();
    }

    // f and J at y: J region [i][j] (T, then f after the species) without the rows'
    // third-body sums (kRow), the temperature row in kT. Ends with the block synchronised.
    __device__ __forceinline__ void evaluate_j(const double (&y)[E], bool rhs_only) {
        const double T = T_of(y);
        const double invT = fast_rcp(hmax(T, kTiny));
        const double logT = fast_log(T), lT = (T > kTiny) ? logT : -34.538776394910684;
        const bool raw = rhs_only && cvRu != 0.0;      // third bodies take c as given
        double2 *cg = reinterpret_cast<double2 *>(s + L::kC);
        double *d = s + L::kD, *h = s + L::kH, *cp = s + L::kCP, *cM = s + L::kCM;
        double ct = 0.0;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int i = lane + 32 * e;
            if (i < nsp) ct += raw ? y[e] : hmax(y[e], 0.0);
        }
        const double ctot = sum(ct);
        // ---- species: eight of each warp
        {
            const int i = warp * 8 + (lane & 7);
            const double yi = __shfl_sync(full, y[0], i & 31), yj = __shfl_sync(full, y[SL - 1], i & 31);
            if (lane < 8 && i < nsp) {
                const double yv = (i >= 32) ? yj : yi;
                const double *t = m.th + kRTh * i;
                const double tl = ldg(&t[0]), th = ldg(&t[2]);
                const double *q = species_range(t, T);
                const double a0 = ldg(&q[0]), a1 = ldg(&q[1]), a2 = ldg(&q[2]), a3 = ldg(&q[3]), a4 = ldg(&q[4]);
                const double a5 = ldg(&q[5]);
                double hR = T * (a0 + T * (a1 * 0.5 + T * (a2 * (1.0 / 3.0) + T * (a3 * 0.25 + T * (a4 * 0.2))))) + a5;
                double cpR = a0 + T * (a1 + T * (a2 + T * (a3 + T * a4)));
                const double dcp = a1 + T * (2.0 * a2 + T * (3.0 * a3 + T * (4.0 * a4)));
                cg[i] = make_double2(hmax(yv, 0.0), species_gibbs(t, q, T, lT));
                cM[i] = raw ? yv : hmax(yv, 0.0);
                double dv = -hR * invT;
                if (T < tl || T > th) {
                    // cp clamped, h extrapolated from the range's end (JANAF.cpp:142-199)
                    const double Tc = hmin(hmax(T, tl), th);
                    const double cc = a0 + Tc * (a1 + Tc * (a2 + Tc * (a3 + Tc * a4)));
                    dv += cc - cpR;
                    cpR = cc;
                    hR = Tc * (a0 + Tc * (a1 * 0.5 + Tc * (a2 * (1.0 / 3.0) + Tc * (a3 * 0.25 + Tc * (a4 * 0.2))))) + a5 +
                         cc * (T - Tc);
                }
                d[i] = dv;
                h[i] = hR * kRu - cvRu * T;
                cp[i] = cpR * kRu - cvRu;
                s[L::kX + i] = dcp * kRu;
            }
        }
        b_sync();
        // ---- reactions
        const int g0 = ldg(&bm.gptr[warp]), g1 = ldg(&bm.gptr[warp + 1]);
        for (int t = ldg(&bm.tptr[warp]); t < ldg(&bm.tptr[warp + 1]); ++t) {
            const int r = ldg(&bm.task[32 * t + lane]);
            if (r < 0) continue;
            const int4 w = __ldg(&m.code[r]);
            const double2 *k2 = reinterpret_cast<const double2 *>(m.rate + r);
            const double2 ka = __ldg(k2), kb = __ldg(k2 + 1);
            const RxnVals v = rxn_eval<true, false>(m, w, make_double4(ka.x, ka.y, kb.x, kb.y),
                                                    [cg](int i) { return cg[i]; }, [cM](int i) { return cM[i]; },
                                                    [d](int i) { return d[i]; }, T, invT, logT, ctot);
            double *R = rec + r * bm.stride;
            R[kBq] = v.q;
            R[kBdq] = v.dq;
            R[kBg] = v.g;
            R[kBd] = v.d[0];
            R[kBd + 1] = v.d[1];
            if (bm.nf == 3) R[kBd + 2] = v.d[2];
            double *Q = R + kBd + bm.nf;
            Q[0] = v.d[3];
            Q[1] = v.d[4];
            if (bm.stride - kBd - bm.nf == 3) Q[2] = v.d[5];
            if ((w.x >> 24) != kArrhenius) {
                const int e0 = w.w & 0xffff, ne = (w.z >> kRneff) & 255;
                for (int e = e0; e < e0 + ne; ++e) rec[m.nrc * bm.stride + e] = ldg(&m.eval[e]) * v.g;
            }
        }
        b_sync();
        // ---- nonzeros of J, f, the column of T, the rows' third-body sums
        auto flip = [](double v, uint32_t sign) {
            return __hiloint2double(__double2hiint(v) ^ (int)(sign & 0x80000000u), __double2loint(v));
        };
        for (int q = g0; q < g1; ++q) {
            const int pi = pair[q];
            const uint2 *t = term + 32 * (pi & 0xffff) + lane;
            const uint32_t to = dst[32 * q + lane];
            double u0 = 0.0, u1 = 0.0, v0 = 0.0, v1 = 0.0;
#pragma unroll 4
            for (int k = pi >> 16; k > 0; --k, t += 32) {
                const uint2 w = *t;
                u0 += flip(rec[w.x & 0x7fffu], w.x << 16);
                u1 += flip(rec[(w.x >> 16) & 0x7fffu], w.x);
                v0 += flip(rec[w.y & 0x7fffu], w.y << 16);
                v1 += flip(rec[(w.y >> 16) & 0x7fffu], w.y);
            }
            auto put = [&](uint32_t at, double v) {
                double *p = (at & kBRow) ? s + L::kRow + (at & 0x7fffu) : J + at;
                *p = v;
            };
            put(to & 0xffffu, u0 + u1);
            put(to >> 16, v0 + v1);
        }
        b_sync();
        // ---- temperature equation: column sums (chemistrySource.cpp:863-906, 975-1055)
        {
            const int part = threadIdx.x & 3;
            for (int jb = 0; jb <= N; jb += kBThreads / 4) {
                const int j = jb + (threadIdx.x >> 2);
                double u = 0.0, v = 0.0;
                if (j <= N) {
                    const double *col = J + j;
                    int i = part;
                    for (; i + 4 < nsp; i += 8) {
                        u += h[i] * col[i * bm.ld];
                        v += h[i + 4] * col[(i + 4) * bm.ld];
                    }
                    if (i < nsp) u += h[i] * col[i * bm.ld];
                }
                u += v;
                u += __shfl_xor_sync(full, u, 1);
                u += __shfl_xor_sync(full, u, 2);
                if (part == 0 && j <= N) s[L::kT + j] = u;
            }
            // scalars: one of the first four warps each
            double z = 0.0;
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const int i = lane + 32 * e;
                if (i >= nsp) continue;
                z += (warp == 0) ? y[e] * cp[i] : (warp == 1) ? y[e] * s[L::kX + i]
                     : (warp == 2) ? h[i] * s[L::kRow + i] : cp[i] * J[i * bm.ld + N];
            }
            z = sum(z);
            if (lane == 0 && warp < 4) s[L::kSc + warp] = z;
        }
        b_sync();
        // the temperature row, one column a thread: scalars C, sum y dcp/dT, sum h kRow, sum cp f
        const double *sc = s + L::kSc;
        const double icCp = frcp(sc[0]), DT = s[L::kT + N] * icCp;
        double v = 0.0;
        const int j = threadIdx.x;
        if (j <= N) {
            const double cpj = (j < nsp) ? cp[j] : (j == nsp) ? sc[1] : 0.0;
            const double S = s[L::kT + j] + ((j < nsp) ? sc[2] : (j == nsp) ? sc[3] : 0.0);
            v = (cpj * DT - S) * icCp;
        }
        b_sync();
        if (j <= N) s[L::kT + j] = v;
        b_sync();
    }

    __device__ __forceinline__ void evaluate(const double (&y)[E], const double (&y0)[E], double dt, bool rhs_only) {
        evaluate_j(y, rhs_only);
        const double *row[E];
        double sr[E];
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int i = lane + 32 * e;
            row[e] = (i < nsp) ? J + i * bm.ld : s + L::kT;
            sr[e] = (i < nsp) ? s[L::kRow + i] : 0.0;
            f[e] = (i <= nsp) ? row[e][N] : 0.0;
        }
        if (rhs_only) {
            b_sync();   // the next evaluation overwrites what is read here
            return;
        }
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int i = lane + 32 * e, diag = i - warp * CPW;
#pragma unroll
            for (int k = 0; k < CPW; ++k) {
                const int j = warp * CPW + k;
                double v = 0.0;
                if (j < nsp) v = row[e][j] + sr[e];
                else if (j == nsp) v = row[e][j];
                v = ((diag == k) ? 1.0 : 0.0) - dt * v;
                if (j == N) v = (-y[e] + y0[e]) + dt * f[e];
                a[e][k] = v;
            }
        }
        b_sync();       // the records' room becomes the pivot steps'
    }

    // key of a pivot candidate: the upper bits of its magnitude and its row
    __device__ __forceinline__ unsigned pivot_key(const double (&v)[SL], const int (&at)[SL]) const {
        unsigned key = 0u;
#pragma unroll
        for (int e = 0; e < SL; ++e) {
            const unsigned hi = (unsigned)__double2hiint(v[e]) & 0x7fffffffu;
            const unsigned ke = (at[e] < 64) ? 0u : ((hi & ~63u) | (unsigned)(63 - (lane + 32 * e)));
            key = ke > key ? ke : key;
        }
        return key;
    }

    // column q of the pivot row (row p, in its lane's registers) to every lane
    __device__ __forceinline__ double row_of(int p, int q) const {
        return __shfl_sync(full, (SL == 2 && p >= 32) ? a[SL - 1][q] : a[0][q], p & 31);
    }

    __device__ __forceinline__ void solve(double (&x)[E], bool) {
        // the pivot step that row lane + 32 e was chosen in (N and more: not yet, none)
        int at[SL];
#pragma unroll
        for (int e = 0; e < SL; ++e) at[e] = has(e) ? 1 << 20 : -1;
        auto mark = [&](int p, int k) {
#pragma unroll
            for (int e = 0; e < SL; ++e) at[e] = (lane + 32 * e == p) ? k : at[e];
        };
        const int *prow = reinterpret_cast<const int *>(s + L::kPV + 64);
        const int last = N / CPW;       // the warp that holds the right-hand side
        // the columns to the left: follow their owners
        for (int w = 0; w < warp && w <= last; ++w) {
            const int n = (N - w * CPW < CPW) ? N - w * CPW : CPW;
#pragma unroll 1
            for (int k = 0; k < n; ++k) {
                asm volatile("bar.sync %0, %1;" ::"r"(1 + k), "r"(32 * (kBWarps - w)) : "memory");
                const int p = prow[w * CPW + k];
                double l[SL];
#pragma unroll
                for (int e = 0; e < SL; ++e) l[e] = rec[64 * k + lane + 32 * e];
                mark(p, w * CPW + k);
#pragma unroll
                for (int q = 0; q < CPW; ++q) {
                    const double u = row_of(p, q);
#pragma unroll
                    for (int e = 0; e < SL; ++e) a[e][q] -= l[e] * u;
                }
            }
            // every warp that follows has read panel w before warp w + 1 publishes over it
            asm volatile("bar.sync 15, %0;" ::"r"(32 * (kBWarps - w)) : "memory");
        }
        // This warp's own columns, always column 0: they move one place to the left as
        // they are updated, so that one copy of the step serves all of them (unrolled
        // steps ran at the speed of the instruction fetch). The next pivot column comes
        // first and by shuffles; its search and reciprocals run under the other columns.
        const int n = N - warp * CPW < CPW ? N - warp * CPW : CPW;
        double v[SL], own[SL];
#pragma unroll
        for (int e = 0; e < SL; ++e) {
            v[e] = a[e][0];
            own[e] = fast_rcp(v[e]);
        }
        unsigned top = __reduce_max_sync(full, pivot_key(v, at));
#pragma unroll 1
        for (int K = 0; K < n; ++K) {
            const int p = 63 - (int)(top & 63u), k = warp * CPW + K;
            const bool high = SL == 2 && p >= 32;
            const double inv = __shfl_sync(full, high ? own[SL - 1] : own[0], p & 31);
            const double u1 = row_of(p, 1);
            // rows chosen before keep their entry, a column of U; the others are eliminated
            double l[SL], uv[SL];
#pragma unroll
            for (int e = 0; e < SL; ++e) {
                uv[e] = v[e];
                l[e] = (at[e] < k || lane + 32 * e == p) ? 0.0 : v[e] * inv;
            }
#pragma unroll
            for (int e = 0; e < SL; ++e) v[e] = a[e][1] - l[e] * u1;
            mark(p, k);
            top = __reduce_max_sync(full, pivot_key(v, at));
#pragma unroll
            for (int e = 0; e < SL; ++e) rec[64 * K + lane + 32 * e] = l[e];
            if (lane == 0) {
                s[L::kPV + k] = inv;
                reinterpret_cast<int *>(s + L::kPV + 64)[k] = p;
            }
            __syncwarp();
            if (warp < kBWarps - 1)
                asm volatile("bar.arrive %0, %1;" ::"r"(1 + K), "r"(32 * (kBWarps - warp)) : "memory");
            double u[CPW];
#pragma unroll
            for (int q = 2; q < CPW; ++q) u[q] = row_of(p, q);
#pragma unroll
            for (int e = 0; e < SL; ++e)
                if ((unsigned)at[e] < (unsigned)k) rec[b_ucol(k) + at[e]] = uv[e];
#pragma unroll
            for (int e = 0; e < SL; ++e) {
                own[e] = fast_rcp(v[e]);
                a[e][0] = v[e];
#pragma unroll
                for (int q = 1; q + 1 < CPW; ++q) a[e][q] = a[e][q + 1] - l[e] * u[q + 1];
            }
        }
        if (warp < kBWarps - 1 && warp <= last)
            asm volatile("bar.arrive 15, %0;" ::"r"(32 * (kBWarps - warp)) : "memory");
        if (warp == last) {
            // back substitution in pivot order (lane k has unknowns k and k + 32); the
            // right-hand side has moved to column 0
#pragma unroll
            for (int e = 0; e < SL; ++e) s[L::kX + lane + 32 * e] = a[e][0];
            __syncwarp();
            double b[SL], pinv[SL];
#pragma unroll
            for (int e = 0; e < SL; ++e) {
                const int k = lane + 32 * e;
                pinv[e] = (k < N) ? s[L::kPV + k] : 0.0;
                b[e] = (k < N) ? s[L::kX + prow[k]] * pinv[e] : 0.0;
            }
            // rows scaled by their pivot: x_k is b_k, a shuffle and an FMA a step in the chain
            for (int e0 = SL - 1; e0 >= 0; --e0) {
                const int lo = 32 * e0, hi = (N < lo + 32) ? N : lo + 32;
#pragma unroll 8
                for (int k = hi - 1; k >= lo; --k) {
                    double u[SL];
#pragma unroll
                    for (int e = 0; e < SL; ++e) u[e] = (lane + 32 * e < k) ? rec[b_ucol(k) + lane + 32 * e] * pinv[e] : 0.0;
                    const double xk = __shfl_sync(full, e0 ? b[SL - 1] : b[0], k & 31);
#pragma unroll
                    for (int e = 0; e < SL; ++e) b[e] -= u[e] * xk;
                }
            }
            __syncwarp();
#pragma unroll
            for (int e = 0; e < SL; ++e) s[L::kX + lane + 32 * e] = b[e];
        }
        b_sync();
#pragma unroll
        for (int e = 0; e < SL; ++e) x[e] = has(e) ? s[L::kX + lane + 32 * e] : 0.0;
        b_sync();
    }
};

template <int CPW, int SL>
__global__ void __launch_bounds__(kBThreads, kBBlocks)
integrate_b_kernel(const __grid_constant__ RMech m, const __grid_constant__ BMech bm,
                   const __grid_constant__ IntegratorParams P, const __grid_constant__ CellIO io) {
    using L = BLayout<CPW, SL>;
    extern __shared__ __align__(16) double smem_b[];
    StepControl<BCell<CPW, SL>> ci(m, bm, P, smem_b);
    ci.init();
    const int nsp = m.nsp, lane = ci.lane;
    double W[SL];
#pragma unroll
    for (int e = 0; e < SL; ++e) W[e] = (lane + 32 * e < nsp) ? ldg(&m.th[kRTh * (lane + 32 * e) + 3]) : 1.0;
    // the first cells go round the blocks, the rest by the queue
    for (long long k = blockIdx.x; k < io.nqueue;) {
        const int64_t cell = io.order ? (int64_t)io.order[k] : (int64_t)k;
        ci.start();
        const double Ti = io.T[cell];
        const double tstep = io.dt[cell] * io.dt_factor;
        const double rho0 = io.rho[cell];
        double y[SL], c0[SL];
#pragma unroll
        for (int e = 0; e < SL; ++e) {
            const int i = lane + 32 * e;
            c0[e] = (i < nsp) ? rho0 * io.Y[(int64_t)i * io.ncells + cell] / W[e] : 0.0;
            y[e] = (i == nsp) ? Ti : c0[e];
        }
        if (Ti < P.T_threshold) {
            if (ci.warp == 0) {
                if (lane == 0) {
                    io.subdt[cell] = tstep;
                    if (io.status) io.status[cell] = 1;  // HC_CELL_SKIPPED
                    if (io.cost) io.cost[cell] = 0;
                }
                if (io.Ri)
                    for (int i = lane; i < nsp; i += 32) io.Ri[(int64_t)i * io.ncells + cell] = 0.0;
            }
        } else {
            double sub = hmin(tstep, hmin(io.subdt[cell], P.dt_max));
            ci.cell(tstep, sub, y);
            // ciToYi (chemistrySource.cpp:1225-1246) and rho = p / (Rm T)
            const double Tn = ci.T_of(y);
            double yi[SL], t = 0.0;
#pragma unroll
            for (int e = 0; e < SL; ++e) {
                yi[e] = (lane + 32 * e < nsp) ? hmax(0.0, y[e]) : 0.0;
                t += yi[e] * W[e];
            }
            const double rr = ci.sum(t);
            t = 0.0;
#pragma unroll
            for (int e = 0; e < SL; ++e) {
                yi[e] = yi[e] * W[e] / hmax(rr, kTiny);
                t += yi[e];
            }
            const double ys = ci.sum(t);
            t = 0.0;
#pragma unroll
            for (int e = 0; e < SL; ++e) {
                if (ys != 1.0) yi[e] /= ys;
                t += yi[e] / W[e];
            }
            const double wsum = ci.sum(t);
            const double Rm = kRu * hmax(wsum, kVeryTiny);
            if (ci.warp == 0) {
#pragma unroll
                for (int e = 0; e < SL; ++e) {
                    const int i = lane + 32 * e;
                    if (i >= nsp) continue;
                    io.Y[(int64_t)i * io.ncells + cell] = yi[e];
                    if (io.Ri) io.Ri[(int64_t)i * io.ncells + cell] = (y[e] - c0[e]) / tstep * W[e];
                }
                if (lane == 0) {
                    ci.store(io, cell, Tn, sub);
                    // constant volume keeps the density (chemistrySource.cpp:1317-1323)
                    if (P.reactor != 1) io.rho[cell] = io.p[cell] / (Rm * Tn);
                }
            }
        }
        // the next cell: one thread asks, the block reads it
        b_sync();
        if (threadIdx.x == 0)
            reinterpret_cast<long long *>(smem_b + L::kSc)[7] = (long long)gridDim.x + (long long)atomicAdd(io.queue_head, 1ULL);
        b_sync();
        k = reinterpret_cast<long long *>(smem_b + L::kSc)[7];
        b_sync();
    }
}

// f and the analytic Jacobian at given states (chemistrySource::DyDt, ::jacobian)
template <int CPW, int SL>
__global__ void __launch_bounds__(kBThreads, kBBlocks)
jacobian_b_kernel(const __grid_constant__ RMech m, const __grid_constant__ BMech bm,
                  const __grid_constant__ IntegratorParams P, int64_t n, const double *__restrict__ c,
                  const double *__restrict__ T, double *__restrict__ dydt, double *__restrict__ Jo) {
    using L = BLayout<CPW, SL>;
    extern __shared__ __align__(16) double smem_b[];
    BCell<CPW, SL> ci(m, bm, P, smem_b);
    ci.init();
    const int nsp = m.nsp, N = nsp + 1, lane = ci.lane;
    for (int64_t k = blockIdx.x; k < n; k += gridDim.x) {
        double y[SL];
#pragma unroll
        for (int e = 0; e < SL; ++e) {
            const int i = lane + 32 * e;
            y[e] = (i < nsp) ? c[(int64_t)i * n + k] : (i == nsp) ? T[k] : 0.0;
        }
        ci.evaluate_j(y, Jo == nullptr);
        if (dydt)
            for (int i = threadIdx.x; i < N; i += kBThreads)
                dydt[k * N + i] = (i < nsp) ? ci.J[i * bm.ld + N] : smem_b[L::kT + N];
        if (Jo) {
            // a warp per row: 8-byte stores of consecutive columns
            for (int i = ci.warp; i < N; i += kBWarps) {
                const double sr = (i < nsp) ? smem_b[L::kRow + i] : 0.0;
                const double *row = (i < nsp) ? ci.J + i * bm.ld : smem_b + L::kT;
                for (int j = lane; j < N; j += 32) Jo[(k * N + i) * N + j] = row[j] + (j < nsp ? sr : 0.0);
            }
        }
        b_sync();
    }
}

}  // namespace hc
