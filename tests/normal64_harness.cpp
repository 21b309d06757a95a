// Host build of csrc/normal64.cuh: unit complex normals of n word pairs.
#include "../cl_var_dt_gb300/csrc/normal64.cuh"

extern "C" void normals(long n, const uint32_t *x, const uint32_t *y, double *re, double *im) {
    for (long i = 0; i < n; ++i) clv::normal64(x[i], y[i], re[i], im[i]);
}
