// Host build of csrc/normal64.cuh: unit complex normals of n word pairs.
#include "../cl_var_dt_gb300/csrc/normal64.cuh"

extern "C" void normals(long n, const uint32_t *x, const uint32_t *y, double *re, double *im) {
    for (long i = 0; i < n; ++i) clv::normal64(x[i], y[i], re[i], im[i]);
}

#ifdef NORMAL64_MAIN
// All pairs of the words given as arguments (for a build that checks for undefined behaviour).
#include <cstdio>
#include <cstdlib>
int main(int argc, char **argv) {
    double sum = 0;
    for (int i = 1; i < argc; ++i)
        for (int j = 1; j < argc; ++j) {
            const uint32_t x = (uint32_t)strtoul(argv[i], nullptr, 0), y = (uint32_t)strtoul(argv[j], nullptr, 0);
            double re, im;
            normals(1, &x, &y, &re, &im);
            sum += re + im;
        }
    printf("%g\n", sum);
}
#endif
