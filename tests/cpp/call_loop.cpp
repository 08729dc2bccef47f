// One entry point called again and again from the calling thread (ctypes has released the
// interpreter lock), for the tests of calls from several host threads. Stops at the first
// result other than 0 and returns it.
#include <cstdint>

typedef int (*props_fn)(void *, int64_t, const double *, const double *, const double *, double *, double *,
                        double *, double *, double *, void *);
typedef int (*jac_fn)(void *, int64_t, const double *, const double *, const double *, double *, double *, void *);

extern "C" {

int loop_properties(props_fn f, int reps, void *m, int64_t n, const double *T, const double *p, const double *Y,
                    double *ha, double *cp, double *mu, double *kappa, double *D, void *stream) {
    for (int k = 0; k < reps; ++k)
        if (int rc = f(m, n, T, p, Y, ha, cp, mu, kappa, D, stream)) return rc;
    return 0;
}

int loop_jacobian(jac_fn f, int reps, void *m, int64_t n, const double *c, const double *T, const double *p,
                  double *dydt, double *J, void *stream) {
    for (int k = 0; k < reps; ++k)
        if (int rc = f(m, n, c, T, p, dydt, J, stream)) return rc;
    return 0;
}
}
