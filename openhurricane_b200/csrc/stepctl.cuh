// The reference's step control (ImplicitEuler::solve / adaptiveSolve /
// NewtonIteration, ODEsSolver::maxError) around a cell that several lanes of
// a warp, or several warps, integrate together. Every warp of the cell runs
// it with the same values, so that the control flow is uniform.
//
// Cell provides: E elements per lane, kAuto (autoUpdateJacobian is on), has(e) (the lane
// carries element e), T_of(y), evaluate(y, y0, dt, rhs_only) with f[e] where f_here(),
// solve(x, reuse) with the last factors where reuse, first_bad(bad) and max_nonneg(v).
#pragma once

#include "integrator.cuh"

namespace hc {

template <class Cell>
struct StepControl : Cell {
    static constexpr int E = Cell::E;
    static constexpr unsigned full = 0xffffffffu;
    using Cell::P;
    int countStep;
    double lts0, lts1;           // lastTimeStep_[0], [1]
    double yk0[E], yk1[E];       // yklast_[0], [1] (this lane's elements)
    int n_jac, n_rhs, n_newton, n_steps, n_attempts;   // every new Jacobian is factored: n_lu = n_jac
    int status;

    template <class... A>
    __device__ StepControl(A &&...a) : Cell(a...) {}

    __device__ void start() {
        countStep = 0;
        lts0 = lts1 = 0.0;
#pragma unroll
        for (int e = 0; e < E; ++e) yk0[e] = yk1[e] = 0.0;
        n_jac = n_rhs = n_newton = n_steps = n_attempts = 0;
        status = 0;
    }

    // ODEsSolver::maxError (ODEsSolver.cpp:37-46) over the lanes where `on`;
    // NaN terms do not raise the max
    __device__ double norm(bool on, double atol, double rtol, const double (&y0)[E], const double (&y)[E],
                           const double (&d)[E]) const {
        double m = 0.0;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const double v = fabs(d[e]) * frcp(atol + rtol * hmax(fabs(y0[e]), fabs(y[e])));
            if (on && this->has(e) && v > m) m = v;
        }
        return this->max_nonneg(m);
    }

    // ImplicitEuler::solve(t0, y0, dydt0, dt, y) with ::NewtonIteration and
    // ::maxIncrement (ImplicitEuler.cpp:40-52, 101-251)
    __device__ double step(const double (&y0)[E], double dt, double (&yk)[E], int &rc) {
        ++n_attempts;
#pragma unroll
        for (int e = 0; e < E; ++e) yk[e] = y0[e];
        int count = 0;
        double lastErr = 0.0, d[E];
        bool on = true, error_pass = false;
        constexpr bool autoJ = Cell::kAuto;
        const int stepJ = P.step_to_update_jac;
        while (true) {
            const bool keepJ = autoJ && !error_pass && count != 0 && count % stepJ != 0;
            if (error_pass || keepJ) ++n_rhs; else ++n_jac;
            this->evaluate(yk, y0, dt, error_pass || keepJ);
            if (error_pass) {
                // the first step's error estimate
#pragma unroll
                for (int e = 0; e < E; ++e) d[e] = yk[e] - y0[e] - dt * this->f[e];
                on = this->f_here();
                break;
            }
            double x[E];
            this->solve(x, keepJ);
            ++n_newton;
            const int bad = this->first_bad(x);
#pragma unroll
            for (int e = 0; e < E; ++e)
                if (this->has(e) && this->elem(e) < bad) yk[e] += x[e];
            if (bad < (1 << 30)) return 1000.0;
            const double maxErr = norm(true, P.atol, P.rtol, yk, yk, x);
            if (count > 0) {
                const double diver = maxErr * frcp(hmax(lastErr, kTiny));
                const int lim = autoJ ? ((30 * stepJ > 50) ? 30 * stepJ : 50) : 5;
                if (diver > 2 && count > lim) return 1000.0;
            }
            lastErr = maxErr;
            count++;
            if (count > 1000) return maxErr;
            if (P.max_newton_total > 0 && n_newton >= P.max_newton_total) {
                rc = kRcIterLimit;
                return 1000.0;
            }
            if (maxErr > 1.0) continue;
            if (countStep == 0) {
                error_pass = true;
                continue;
            }
            const double dtn = lts0, dtn1 = lts1;
            const double f1 = 2.0 * frcp(dtn * (dtn + dtn1));
            const double f2 = 2.0 * frcp(dtn1 * (dtn + dtn1));
#pragma unroll
            for (int e = 0; e < E; ++e) d[e] = (f1 * (yk[e] - y0[e]) - f2 * (y0[e] - yk1[e])) * ((dtn * dtn) * 0.5);
            break;
        }
        bool nan = false;
#pragma unroll
        for (int e = 0; e < E; ++e) nan = nan || (this->has(e) && isnan(yk[e]));
        if (__any_sync(full, nan)) return 1.5;
        return norm(on, P.atol_inc, P.rtol_inc, y0, yk, d);
    }

    // ImplicitEuler::adaptiveSolve (ImplicitEuler.cpp:253-292) with checkNewY
    // (chemistrySource.cpp:1152-1164)
    __device__ int adaptive(double &t, double &dt0, double (&y)[E]) {
        double dt = dt0;
        double error = 0.0, scale = 0.0;
        double yTemp[E];
        lts1 = lts0;
        int count = 0;
        const double Told = this->T_of(y);
        do {
            lts0 = dt;
            int rc = kRcOk;
            error = step(y, dt, yTemp, rc);
            if (rc != kRcOk) return rc;
            const double Tnew = this->T_of(yTemp);
            if ((Tnew - Told) > P.T_alpha * Told) {
                dt *= P.T_beta;
                if (count < 100) {
                    error = 2;
                    count++;
                    if (dt <= kVeryTiny) return kRcUnderflow;
                    continue;
                }
            }
            // the factor of a rejected step, and of the next one after an accepted step
            scale = hmax(P.safescale * fpow_pos(error, -P.alphainc), P.minscale);
            if (error > 1.0) {
                dt *= scale;
                if (dt <= kVeryTiny) return kRcUnderflow;
            }
        } while (error > 1.0);
        t += dt;
#pragma unroll
        for (int e = 0; e < E; ++e) y[e] = yTemp[e];
        ++n_steps;
        if (error > P.err_accept_limit) dt0 = hmin(scale, P.maxscale) * dt;
        else dt0 = hmax(P.safescale * P.maxscale * dt, dt);
        return kRcOk;
    }

    // ImplicitEuler::solve(t0, tn, dt0, y) (ImplicitEuler.cpp:294-342), t0 = 0
    __device__ int interval(double &tn, double &dt0, double (&y)[E]) {
        double t = 0.0;
        double dt = 0.2 * dt0;
        double dtReached = 0.0;
        bool last = false;
        for (int n = 0; n < P.maxstep; ++n) {
            countStep = n;
#pragma unroll
            for (int e = 0; e < E; ++e) {
                yk1[e] = (n == 0) ? yk1[e] : yk0[e];
                yk0[e] = y[e];
            }
            const double dtTry0 = dt;
            if ((t + dt - tn) * (t + dt - 0.0) > 0) {
                dt = tn - t;
                last = true;
            } else if (t + dt == tn) {
                last = true;
            }
            const int rc = adaptive(t, dt, y);
            if (rc != kRcOk) return rc;
            dtReached = t;
            if ((t - tn) * (tn - 0.0) >= 0) {
                if (n > 0 && last) dt0 = hmin(dtTry0, tn);
                return kRcOk;
            }
        }
        status |= 2;  // HC_CELL_MAXSTEP
        tn = dtReached;
        return kRcOk;
    }

    // chemistrySource::solve of one cell over tstep (chemistrySource.cpp:1511-1555);
    // sub: the warm-start sub-step, updated
    __device__ void cell(double tstep, double &sub, double (&y)[E]) {
        double leftTime = tstep;
        int rc = kRcOk;
        while (leftTime > 0.0) {
            double d = leftTime;
            rc = interval(d, sub, y);
            if (rc != kRcOk) break;
            leftTime -= d;
        }
        if (rc == kRcUnderflow) status |= 4;
        if (rc == kRcIterLimit) status |= 8;
    }

    // one lane writes the cell's scalars
    __device__ void store(const CellIO &io, int64_t cell, double Tn, double sub) const {
        io.T[cell] = Tn;
        io.subdt[cell] = sub;
        if (io.status) io.status[cell] = status;
        if (io.cost) io.cost[cell] = n_newton;
        if (io.counters) {
            atomicAdd(&io.counters[0], (unsigned long long)n_jac);
            atomicAdd(&io.counters[1], (unsigned long long)n_rhs);
            atomicAdd(&io.counters[2], (unsigned long long)n_jac);
            atomicAdd(&io.counters[3], (unsigned long long)n_newton);
            atomicAdd(&io.counters[4], (unsigned long long)n_steps);
            atomicAdd(&io.counters[5], (unsigned long long)n_attempts);
        }
    }
};

}  // namespace hc
