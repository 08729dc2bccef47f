// Host build of the kernels' elementary functions (openhurricane_b200/csrc/fastmath.cuh).
// Reads from stdin, printing 17 significant digits:
//   "E x" -> fast_exp, "X x" -> lean_exp, "L x" -> fast_log
//   "F troe alpha T*** T* T** four T ratio M dlr" -> fall_off: w, gM, wT
#include <cmath>
#include <cstdio>

using std::exp;
using std::fabs;
using std::fma;
using std::frexp;
using std::isinf;
using std::isnan;
using std::ldexp;
using std::log;

#include "../../openhurricane_b200/csrc/fastmath.cuh"

int main() {
    char kind[2];
    while (std::scanf("%1s", kind) == 1) {
        double v[10];
        if (kind[0] == 'F') {
            for (int k = 0; k < 10; ++k)
                if (std::scanf("%lf", &v[k]) != 1) return 1;
            const double T = v[6], e1 = exp(-T / v[2]), e2 = exp(-T / v[3]), e3 = v[5] != 0 ? exp(-v[4] / T) : 0.0;
            const hc::FallOff f = hc::fall_off<true>(v[0] != 0, v[1], 1.0 / v[2], 1.0 / v[3], v[4], e1, e2, e3, v[7], v[8],
                                                     v[9], 1.0 / T);
            std::printf("%.17g %.17g %.17g\n", f.w, f.gM, f.wT);
        } else {
            if (std::scanf("%lf", &v[0]) != 1) return 1;
            std::printf("%.17g\n", kind[0] == 'E' ? hc::fast_exp(v[0]) : kind[0] == 'X' ? hc::lean_exp(v[0]) : hc::fast_log(v[0]));
        }
    }
    return 0;
}
