// Host build of csrc/drift_math.cuh: the reference model's drift at one site.
#include "host_cuda.h"
#include "../cl_var_dt_gb300/csrc/drift_math.cuh"

using namespace clv;

// f: psi(tau-1), psi(tau), psi(tau+1), psibar(tau), psibar(tau+1), kin(tau-1), kinbar(tau+1), four
// components each; k: K then Kbar
template <class R>
static void drift(const double *par, const double *f, double *k) {
    using C2 = typename Cx<R>::T;
    ChainDev ch{};
    ch.eps = par[0]; ch.a_x = par[1]; ch.mu = par[2]; ch.P = par[3]; ch.Q = par[4]; ch.G = par[5];
    C2 v[7][4], K[4], Kc[4];
    for (int i = 0; i < 28; ++i) v[i / 4][i % 4] = mk<C2>((R)f[2 * i], (R)f[2 * i + 1]);
    const DriftConsts<R> dk(ch);
    // whole, and by field and component halves: the same bits
    drift_ref4_vals<R>(dk, v[0], v[1], v[2], v[3], v[4], v[5], v[6], K, Kc);
    for (int a = 0; a < 4; ++a) {
        k[2 * a] = K[a].x; k[2 * a + 1] = K[a].y;
        k[8 + 2 * a] = Kc[a].x; k[9 + 2 * a] = Kc[a].y;
    }
    for (int half = 0; half < 2; ++half) {
        C2 H[4], Hc[4];
        const int mask = half ? 0xC : 0x3;
        drift_ref4_vals<R>(dk, v[0], v[1], v[2], v[3], v[4], v[5], v[6], H, Hc, 1, mask);
        drift_ref4_vals<R>(dk, v[0], v[1], v[2], v[3], v[4], v[5], v[6], H, Hc, 2, mask);
        for (int a = 2 * half; a < 2 * half + 2; ++a)
            if (std::memcmp(&H[a], &K[a], sizeof(C2)) || std::memcmp(&Hc[a], &Kc[a], sizeof(C2))) k[0] = NAN;
    }
}
extern "C" void drift_ref4(int fp64, long n, const double *par, const double *f, double *k) {
    for (long i = 0; i < n; ++i) {
        if (fp64) drift<double>(par, f + 56 * i, k + 16 * i);
        else drift<float>(par, f + 56 * i, k + 16 * i);
    }
}
