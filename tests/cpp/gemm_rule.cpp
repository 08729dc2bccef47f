// Host build of the GEMM's pipeline-depth rule: "tiles_m tiles_n K sms" lines -> stages
#include <cstdio>

#include "../../openhurricane_b200/csrc/gemm_rule.h"

int main() {
    int m, n, k, sms;
    while (std::scanf("%d %d %d %d", &m, &n, &k, &sms) == 4) std::printf("%d\n", hc::gemm_stages(m, n, k, sms));
    return 0;
}
