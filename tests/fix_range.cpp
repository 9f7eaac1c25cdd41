// The range check of the fixed-point FP64 sweep (pn_fix.cuh) on the CPU: stdin has lines
// "m0 m v2 sx sy sz eL inv_c2", stdout 1 for a star inside the range and 0 outside.
#include <cstdio>

#include "../pn_gb300/csrc/pn_fix.cuh"

int main() {
    double m0, m, v2, s[3], ic2;
    int eL;
    while (scanf("%lf %lf %lf %lf %lf %lf %d %lf", &m0, &m, &v2, &s[0], &s[1], &s[2], &eL, &ic2) == 8)
        printf("%d\n", (int)pn::fix::in_range(s, v2, m, m0, eL, pn::fix::velocity_limit(ic2)));
    return 0;
}
