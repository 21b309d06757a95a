// drift_math.cuh -- per-site drift of both models on register values.
//
// Inputs at one spatial site: psi(tau-1) pm, psi(tau) pc, psi(tau+1) pp,
// psibar(tau) cc, psibar(tau+1) cp, kinetic terms km = kin(tau-1) and
// kp = kinbar(tau+1).  Outputs K (psi drift) and Kc (psibar drift).
#pragma once

#include "clv_internal.cuh"

namespace clv {

// Complex arithmetic with every rounding written out, so that all kernels that compute a
// drift (fused, tiled, step loop; whole or split by field and component) get the same
// bits from the same inputs whatever the compiler does around them.
template <class R, class C2> __device__ __forceinline__ C2 xadd(C2 a, C2 b) {
    C2 r; r.x = add_rn<R>(a.x, b.x); r.y = add_rn<R>(a.y, b.y); return r;
}
template <class R, class C2> __device__ __forceinline__ C2 xsub(C2 a, C2 b) {
    C2 r; r.x = add_rn<R>(a.x, -b.x); r.y = add_rn<R>(a.y, -b.y); return r;
}
template <class R, class C2> __device__ __forceinline__ C2 xscale(R s, C2 a) {
    C2 r; r.x = mul_rn<R>(s, a.x); r.y = mul_rn<R>(s, a.y); return r;
}
// a b
template <class R, class C2> __device__ __forceinline__ C2 xmul(C2 a, C2 b) {
    C2 r;
    r.x = fma_rn<R>(a.x, b.x, -mul_rn<R>(a.y, b.y));
    r.y = fma_rn<R>(a.x, b.y, mul_rn<R>(a.y, b.x));
    return r;
}
// s + a b and s - a b: four fused multiply-adds
template <class R, class C2> __device__ __forceinline__ C2 xmadd(C2 s, C2 a, C2 b) {
    C2 r;
    r.x = fma_rn<R>(-a.y, b.y, fma_rn<R>(a.x, b.x, s.x));
    r.y = fma_rn<R>(a.y, b.x, fma_rn<R>(a.x, b.y, s.y));
    return r;
}
template <class R, class C2> __device__ __forceinline__ C2 xmsub(C2 s, C2 a, C2 b) {
    C2 r;
    r.x = fma_rn<R>(a.y, b.y, fma_rn<R>(-a.x, b.x, s.x));
    r.y = fma_rn<R>(-a.y, b.x, fma_rn<R>(-a.x, b.y, s.y));
    return r;
}

// Per-chain constants of the drift in the working precision, loaded once per CTA.
template <class R>
struct DriftConsts {
    R eps, pre, g2, ec0, ec1;
    R mu[4];
    bool scaled;  // a_x is not 1 (a product with 1 is left out)
    __device__ __forceinline__ explicit DriftConsts(const ChainDev &ch) {
        eps = (R)ch.eps;
        pre = (R)ch.a_x;
        g2 = (R)(2 * ch.G);
        scaled = pre != (R)1;
        ec0 = (R)(ch.eps * ch.c0);  // spin-1: eps c0 and eps c1 (the drift's prefactors)
        ec1 = (R)(ch.eps * ch.c1);
        mu[0] = (R)(ch.mu + ch.P + ch.Q);
        mu[1] = (R)ch.mu;
        mu[2] = (R)ch.mu;
        mu[3] = (R)(ch.mu - ch.P + ch.Q);
    }
};

// Reference 4-component model: calculate_drift_without_noise
// (Propagator_without_cutoff.cu:24-128) with factor = 1.  which: 1 = K only, 2 =
// Kbar only, 3 = both (a CTA-uniform choice of the kernels that split the fields);
// cmask: the components a whose K[a], Kc[a] are computed (bit a; CTA-uniform).
//
// The contact term of component a with the multiplied field k and the other field b (three
// densities and an exchange product in the reference) is, with n_01 = k_0 b_0 + k_1 b_1, n_23 the
// same of 2 and 3, X = k_0 b_2 + k_1 b_3 and Y = k_2 b_0 + k_3 b_1,
//   t_0 = n_01 k_0 + X k_2,  t_1 = n_01 k_1 + X k_3,  t_2 = n_23 k_2 + Y k_0,  t_3 = n_23 k_3 + Y k_1.
// For the other field's drift k and b change places, that is, X and Y do, so one set serves both
// fields' drifts of a (psi(tau), psibar(tau+1)) pair: the streaming kernel computes it once and
// carries it.  94 FP64 operations per field (102 when a_x is not 1; 20 fewer when carried) instead
// of 144 in the component-wise form: the reference model's reduce pass is bound by the FP64
// pipe (2 operations per clock and SM).  No term is added that cancels again: a form with the
// sum of all four densities, which takes component 3 - a's out of t_a, carries its rounding
// where that component is far above the others.
template <class C2>
struct Ref4Pair {
    C2 n01, n23, X, Y;  // times -2G
};
// which: 1 = what K's components of cmask need, 2 = Kbar's, 3 = both (and all components)
template <class R, class C2>
__device__ __forceinline__ Ref4Pair<C2> ref4_pair(R g2, const C2 *psi, const C2 *bar, int which = 3, int cmask = 0xF) {
    Ref4Pair<C2> p;
    const bool lo = (cmask & 3) != 0, hi = (cmask & 12) != 0;
    auto two = [&](int a, int b, int c, int d) { return xscale<R>(-g2, xmadd<R>(xmul<R>(psi[a], bar[b]), psi[c], bar[d])); };
    if (lo) p.n01 = two(0, 0, 1, 1);
    if (hi) p.n23 = two(2, 2, 3, 3);
    if (which == 3 || (which == 1 ? lo : hi)) p.X = two(0, 2, 1, 3);
    if (which == 3 || (which == 1 ? hi : lo)) p.Y = two(2, 0, 3, 1);
    return p;
}

// p: ref4_pair of (pm, cc).
template <class R, class C2>
__device__ __forceinline__ void drift_ref4_psi(const DriftConsts<R> &k, const Ref4Pair<C2> &p, const C2 *pm, const C2 *pc,
                                               const C2 *km, C2 *K, int cmask = 0xF) {
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        if (!((cmask >> a) & 1)) continue;
        C2 m = a < 2 ? p.n01 : p.n23;
        m.x = add_rn<R>(k.mu[a], m.x);
        C2 in = xmadd<R>(km[a], m, pm[a]);
        in = xmadd<R>(in, a < 2 ? p.X : p.Y, pm[a ^ 2]);
        K[a].x = fma_rn<R>(k.eps, in.x, add_rn<R>(pm[a].x, -pc[a].x));
        K[a].y = fma_rn<R>(k.eps, in.y, add_rn<R>(pm[a].y, -pc[a].y));
        if (k.scaled) K[a] = xscale<R>(k.pre, K[a]);
    }
}

// p: ref4_pair of (pc, cp).
template <class R, class C2>
__device__ __forceinline__ void drift_ref4_bar(const DriftConsts<R> &k, const Ref4Pair<C2> &p, const C2 *pp, const C2 *cc,
                                               const C2 *cp, const C2 *kp, C2 *Kc, int cmask = 0xF) {
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        if (!((cmask >> a) & 1)) continue;
        // the chemical-potential term of the conjugate drift multiplies psi(tau+1)
        // (Propagator_without_cutoff.cu:71,88,105,122)
        C2 in;
        in.x = fma_rn<R>(k.mu[a], pp[a].x, kp[a].x);
        in.y = fma_rn<R>(k.mu[a], pp[a].y, kp[a].y);
        in = xmadd<R>(in, a < 2 ? p.n01 : p.n23, cp[a]);
        in = xmadd<R>(in, a < 2 ? p.Y : p.X, cp[a ^ 2]);
        Kc[a].x = fma_rn<R>(k.eps, in.x, add_rn<R>(cp[a].x, -cc[a].x));
        Kc[a].y = fma_rn<R>(k.eps, in.y, add_rn<R>(cp[a].y, -cc[a].y));
        if (k.scaled) Kc[a] = xscale<R>(k.pre, Kc[a]);
    }
}

template <class R, class C2>
__device__ __forceinline__ void drift_ref4_vals(const DriftConsts<R> &k, const C2 *pm, const C2 *pc,
                                                const C2 *pp, const C2 *cc, const C2 *cp,
                                                const C2 *km, const C2 *kp, C2 *K, C2 *Kc, int which = 3,
                                                int cmask = 0xF) {
    if (which & 1) drift_ref4_psi<R>(k, ref4_pair<R>(k.g2, pm, cc, 1, cmask), pm, pc, km, K, cmask);
    if (which & 2) drift_ref4_bar<R>(k, ref4_pair<R>(k.g2, pc, cp, 2, cmask), pp, cc, cp, kp, Kc, cmask);
}

// Spin-1 model.  Of one (bar, ket) pair the contact potential V = c0/2 n^2 + c1/2 (Fz^2 +
// F+ F-) = c0/2 n^2 + c1/2 Fz^2 + c1 P M has the bilinears n = sum_m bar_m ket_m, F_z =
// bar_0 ket_0 - bar_2 ket_2, P = F+/sqrt2 = bar_0 ket_1 + bar_1 ket_2, M = F-/sqrt2 =
// bar_1 ket_0 + bar_2 ket_1.  The derivatives need them as the coefficients
//   A = eps (c0 n + c1 Fz),  N = eps c0 n,  B = eps (c0 n - c1 Fz),  eps c1 P,  eps c1 M:
//   eps dV/dbar = (A ket_0 + M ket_1, N ket_1 + P ket_0 + M ket_2, B ket_2 + P ket_1),
//   eps dV/dket = (A bar_0 + P bar_1, N bar_1 + M bar_0 + P bar_2, B bar_2 + M bar_1).
// The pair (psibar(tau+1), psi(tau)) enters both the psibar drift at tau and the psi
// drift at tau+1, so the streaming kernels with registers to spare compute it once and
// carry it.
template <class C2>
struct Spin1Link {
    C2 A, N, B, P, M;
};

template <class R, class C2>
__device__ __forceinline__ Spin1Link<C2> spin1_link(const DriftConsts<R> &k, const C2 *bar, const C2 *ket) {
    Spin1Link<C2> l;
    const C2 p0 = xmul<R>(bar[0], ket[0]), p2 = xmul<R>(bar[2], ket[2]);
    l.N = xscale<R>(k.ec0, xmadd<R>(xadd<R>(p0, p2), bar[1], ket[1]));
    const C2 f = xscale<R>(k.ec1, xsub<R>(p0, p2));
    l.A = xadd<R>(l.N, f);
    l.B = xsub<R>(l.N, f);
    l.P = xscale<R>(k.ec1, xmadd<R>(xmul<R>(bar[0], ket[1]), bar[1], ket[2]));
    l.M = xscale<R>(k.ec1, xmadd<R>(xmul<R>(bar[1], ket[0]), bar[2], ket[1]));
    return l;
}

// K_m = kin_m(tau-1) - psi_m(tau) - eps dV/dbar_m with l the pair (psibar(tau), psi(tau-1) = pm).
template <class R, class C2>
__device__ __forceinline__ void spin1_drift_psi(const Spin1Link<C2> &l, const C2 *pm, const C2 *pc, const C2 *km, C2 *K) {
    K[0] = xmsub<R>(xmsub<R>(xsub<R>(km[0], pc[0]), l.A, pm[0]), l.M, pm[1]);
    K[1] = xmsub<R>(xmsub<R>(xmsub<R>(xsub<R>(km[1], pc[1]), l.N, pm[1]), l.P, pm[0]), l.M, pm[2]);
    K[2] = xmsub<R>(xmsub<R>(xsub<R>(km[2], pc[2]), l.B, pm[2]), l.P, pm[1]);
}

// Kbar_m = kinbar_m(tau+1) - psibar_m(tau) - eps dV/dket_m with l the pair (psibar(tau+1) = cp, psi(tau)).
template <class R, class C2>
__device__ __forceinline__ void spin1_drift_bar(const Spin1Link<C2> &l, const C2 *cp, const C2 *cc, const C2 *kp, C2 *Kc) {
    Kc[0] = xmsub<R>(xmsub<R>(xsub<R>(kp[0], cc[0]), l.A, cp[0]), l.P, cp[1]);
    Kc[1] = xmsub<R>(xmsub<R>(xmsub<R>(xsub<R>(kp[1], cc[1]), l.N, cp[1]), l.M, cp[0]), l.P, cp[2]);
    Kc[2] = xmsub<R>(xmsub<R>(xsub<R>(kp[2], cc[2]), l.B, cp[2]), l.M, cp[1]);
}

// which: 1 = K only, 2 = Kbar only, 3 = both.
template <class R, class C2>
__device__ __forceinline__ void drift_spin1_vals(const DriftConsts<R> &k, const C2 *pm, const C2 *pc,
                                                 const C2 *cc, const C2 *cp, const C2 *km,
                                                 const C2 *kp, C2 *K, C2 *Kc, int which = 3) {
    if (which & 1) spin1_drift_psi<R>(spin1_link<R>(k, cc, pm), pm, pc, km, K);
    if (which & 2) spin1_drift_bar<R>(spin1_link<R>(k, cp, pc), cp, cc, kp, Kc);
}

// |z|^2 of a drift value for the K/max rule's reduction, rounded the same way in
// every kernel that reduces it (x x + (y y), one fused multiply-add), so that the
// kernels' step sizes agree bit for bit.
template <class R, class C2>
__device__ __forceinline__ R abs2(C2 z) {
    return fma_rn<R>(z.x, z.x, mul_rn<R>(z.y, z.y));
}

// psi + dt K + z (multiply_by_timestep, add_noise, summation); conj = 1 adds conj(z).  dt K + z
// is rounded once (fused multiply-add).
template <class R, class C2>
__device__ __forceinline__ C2 langevin_update(C2 p, C2 K, R dt, C2 z, bool conj) {
    C2 o;
    o.x = add_rn<R>(p.x, fma_rn<R>(K.x, dt, z.x));
    o.y = add_rn<R>(p.y, fma_rn<R>(K.y, dt, conj ? -z.y : z.y));
    return o;
}

// Maximum of values that are not negative or NaN, NaN when either argument is, so that a
// reduction of |drift| carries a non-finite drift to the chain's finish by itself.  FP64
// compares the bit patterns as integers (ordered alike, NaN above infinity): no operation
// on the FP64 pipe.
__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ double max_nan(double a, double b) {
    const unsigned long long x = (unsigned long long)__double_as_longlong(a), y = (unsigned long long)__double_as_longlong(b);
    return __longlong_as_double((long long)(x > y ? x : y));
}

// |z| of a drift value for the reference's rule.  FP64: the library's hypot takes about 60
// operations of the FP64 pipe, as many as a third of the drift; between 2^-511 and 2^497
// the sum of squares neither overflows nor underflows, and its root takes five (a single-
// precision reciprocal root of the mantissa, its bits moved by integer operations, and two
// Newton steps on the root with the residual formed by a fused multiply-add): within 1.1
// units in the last place.
__device__ __forceinline__ float abs_drift(float2 z) { return hypotf(z.x, z.y); }
__device__ __forceinline__ double abs_drift(double2 z) {
    const unsigned hx = (unsigned)__double2hiint(z.x) & 0x7fffffffu, hy = (unsigned)__double2hiint(z.y) & 0x7fffffffu;
    if ((hx > hy ? hx : hy) - 0x20000000u >= 0x3f000000u) return hypot(z.x, z.y);
    const double s = __fma_rn(z.x, z.x, __dmul_rn(z.y, z.y));
    // s = m 4^k, 1 <= m < 4
    const int hs = __double2hiint(s), k = ((hs >> 20) - 1023) >> 1, hm = hs - (k << 21), lo = __double2loint(s);
    const double m = __hiloint2double(hm, lo);
    const float y = rsqrtf(__int_as_float(((hm - 0x38000000) << 3) | (int)((unsigned)lo >> 29)));
    const int yb = __float_as_int(y), yh = (yb >> 3) + 0x38000000, yl = (int)((unsigned)yb << 29);
    const double y0 = __hiloint2double(yh, yl), h = __hiloint2double(yh - 0x00100000, yl);  // y, y / 2
    double g = __dmul_rn(m, y0);
    g = __fma_rn(__fma_rn(-g, g, m), h, g);
    g = __fma_rn(__fma_rn(-g, g, m), h, g);
    return __hiloint2double(__double2hiint(g) + (k << 20), __double2loint(g));
}
__device__ __forceinline__ bool not_finite(float a) { return !isfinite(a); }
__device__ __forceinline__ bool not_finite(double a) { return ((unsigned)__double2hiint(a) & 0x7ff00000u) == 0x7ff00000u; }

// Block-wide (max, sum) with warp shuffles; result valid in thread 0.
__device__ __forceinline__ void block_max_sum(double &mx, double &sm) {
    __shared__ double smx[32], ssm[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        sm += __shfl_xor_sync(0xffffffffu, sm, o);
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) { smx[warp] = mx; ssm[warp] = sm; }
    __syncthreads();
    if (warp == 0) {
        const int nw = (blockDim.x + 31) >> 5;
        mx = lane < nw ? smx[lane] : 0.0;
        sm = lane < nw ? ssm[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            sm += __shfl_xor_sync(0xffffffffu, sm, o);
        }
    }
    __syncthreads();
}

// New step of one chain from its reduction (run by one thread).  REF rule:
// compute_new_dt of Propagator_without_cutoff.cu:372-404; K/max rule:
// dt = min(dt_max, K / max|drift|) with the reduction taken over |K|^2.
__device__ __forceinline__ double step_rule(const ChainDev &ch, ChainState &st, int dt_rule,
                                            double &mx, double sm, double &mean) {
    double dt;
    mean = 0.0;
    if (dt_rule == CLV_DT_REF_MEANMAX) {
        // (a power of two divides exactly: one product instead of a quotient's chain)
        const long long n = (long long)ch.ncomp * ch.V * ch.nt;
        mean = (n & (n - 1)) == 0 ? sm * __hiloint2double((1023 - (63 - __clzll(n))) << 20, 0) : sm / (double)n;
        if (mx <= 0.0) dt = ch.DT;
        else dt = __dmul_rn(mean / mx, ch.DT);
        if (dt < ch.dt_min) { dt = ch.dt_min; st.clamp_low++; st.flags |= CLV_FLAG_DT_CLAMPED_LOW; }
        if (dt > ch.dt_max_clamp) { dt = ch.dt_max_clamp; st.clamp_high++; st.flags |= CLV_FLAG_DT_CLAMPED_HIGH; }
        dt = __dadd_rn(__dmul_rn(1.0 - ch.alpha, ch.DT), __dmul_rn(ch.alpha, dt));
    } else {
        mx = sqrt(mx);
        dt = ch.dt_max;
        if (mx > 0.0) {
            const double t = ch.K / mx;
            if (t < dt) dt = t;
        }
    }
    return dt;
}

}  // namespace clv
