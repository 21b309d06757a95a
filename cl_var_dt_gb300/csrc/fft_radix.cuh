// fft_radix.cuh -- in-register DFT butterflies of radix 2, 3, 4, 5, 6, 8, 9, 10, 12, 15, 16 used by
// the shared-memory Stockham FFTs (line filter and fused step).
//
// Radix<C2, R>::run<S>(a) replaces a[0..R) by y_q = sum_r a_r exp(S 2 pi i r q / R)
// with the direction S = -1 (forward) or +1 (inverse) fixed at compile time, so
// the multiplications by +-i fold into the additions; run(a, S) dispatches a
// runtime direction.
#pragma once

#include <type_traits>

#include "clv_internal.cuh"
#include "fft_int.cuh"

namespace clv {

// A butterfly's real constant in the arithmetic type: itself, or with 62 fraction bits (lo: what
// the double c leaves of it).
template <class R> __host__ __device__ constexpr R kconst(double c, double lo = 0.0) { return (R)c; }
template <> __host__ __device__ constexpr long long kconst<long long>(double c, double lo) {
    return (long long)(c * 4611686018427387904.0) + (long long)(lo * 4611686018427387904.0 + (lo < 0 ? -0.5 : 0.5));
}

// S * i * z for a compile-time direction S
template <int S, class C2>
__device__ __forceinline__ C2 times_si(C2 z) {
    C2 r;
    if (S > 0) { r.x = -z.y; r.y = z.x; }
    else { r.x = z.y; r.y = -z.x; }
    return r;
}

// Arithmetic of the butterflies.  FP64 writes every rounding out, so that all plans that
// run the same butterflies give the same bits wherever they are inlined, with the fused
// multiply-adds placed by hand (FP64 operations are the bound).  FP32 uses the packed two-lane FP32
// instructions of sm_100+ (add/sub .rn.f32x2: two IEEE single additions, the
// same results as the scalar pair), so one instruction moves a complex sum.
template <class C2> __device__ __forceinline__ C2 vadd(C2 a, C2 b) { return cadd(a, b); }
template <class C2> __device__ __forceinline__ C2 vsub(C2 a, C2 b) { return csub(a, b); }
__device__ __forceinline__ unsigned long long f2_pack(float2 a) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
    return r;
}
__device__ __forceinline__ float2 f2_unpack(unsigned long long r) {
    float2 a;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a.x), "=f"(a.y) : "l"(r));
    return a;
}
template <> __device__ __forceinline__ float2 vadd<float2>(float2 a, float2 b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_pack(a)), "l"(f2_pack(b)));
    return f2_unpack(r);
}
template <> __device__ __forceinline__ float2 vsub<float2>(float2 a, float2 b) {
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_pack(a)), "l"(f2_pack(b)));
    return f2_unpack(r);
}

template <> __device__ __forceinline__ double2 vadd<double2>(double2 a, double2 b) {
    return make_double2(__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y));
}
template <> __device__ __forceinline__ double2 vsub<double2>(double2 a, double2 b) {
    return make_double2(__dadd_rn(a.x, -b.x), __dadd_rn(a.y, -b.y));
}
// s z for a real s; z w (twiddle)
__device__ __forceinline__ float2 vscale(float s, float2 z) { return make_float2(s * z.x, s * z.y); }
__device__ __forceinline__ double2 vscale(double s, double2 z) { return make_double2(__dmul_rn(s, z.x), __dmul_rn(s, z.y)); }
__device__ __forceinline__ float2 vmul(float2 z, float2 w) { return cmul(z, w); }
__device__ __forceinline__ double2 vmul(double2 z, double2 w) {
    return make_double2(__fma_rn(z.x, w.x, -__dmul_rn(z.y, w.y)), __fma_rn(z.x, w.y, __dmul_rn(z.y, w.x)));
}
// z conj(w)
template <class C2> __device__ __forceinline__ C2 vmulc(C2 z, C2 w) {
    w.y = -w.y;
    return vmul(z, w);
}
// p = e + s z and m = e - s z for a real constant s
__device__ __forceinline__ void vaxpy2(float2 e, float s, float2 z, float2 &p, float2 &m) {
    const float2 w = vscale(s, z);
    p = vadd(e, w);
    m = vsub(e, w);
}
__device__ __forceinline__ void vaxpy2(double2 e, double s, double2 z, double2 &p, double2 &m) {
    p = make_double2(__fma_rn(s, z.x, e.x), __fma_rn(s, z.y, e.y));
    m = make_double2(__fma_rn(-s, z.x, e.x), __fma_rn(-s, z.y, e.y));
}

// p = f a + g b and m = f a - g b for real f, g: at FP64 two products and four fused
// multiply-adds instead of four products and four sums
__device__ __forceinline__ void vpair(float f, float2 a, float g, float2 b, float2 &p, float2 &m) {
    const float2 x = vscale(f, a), y = vscale(g, b);
    p = vadd(x, y);
    m = vsub(x, y);
}
__device__ __forceinline__ void vpair(double f, double2 a, double g, double2 b, double2 &p, double2 &m) {
    vaxpy2(vscale(f, a), g, b, p, m);
}

// Radix<C2, R>::run<S> is the butterfly, run_scaled<S>(a, f) the butterfly of f[r] a[r]
// (the first inverse pass after the filter).
template <class C2, int R>
struct Radix;

template <class C2>
struct Radix<C2, 2> {
    template <int S>
    static __device__ __forceinline__ void run(C2 *a) {
        C2 t = a[0];
        a[0] = vadd(t, a[1]);
        a[1] = vsub(t, a[1]);
    }
    static __device__ __forceinline__ void run(C2 *a, int) { run<1>(a); }
};

template <class C2>
struct Radix<C2, 4> {
    template <int S>
    static __device__ __forceinline__ void run(C2 *a) {
        finish<S>(a, vadd(a[0], a[2]), vsub(a[0], a[2]), vadd(a[1], a[3]), vsub(a[1], a[3]));
    }
    template <int S>
    static __device__ __forceinline__ void finish(C2 *a, C2 s02, C2 d02, C2 s13, C2 d13) {
        d13 = times_si<S>(d13);
        a[0] = vadd(s02, s13);
        a[2] = vsub(s02, s13);
        a[1] = vadd(d02, d13);
        a[3] = vsub(d02, d13);
    }
    template <int S, class RR>
    static __device__ __forceinline__ void run_scaled(C2 *a, RR f0, RR f1, RR f2, RR f3) {
        C2 s02, d02, s13, d13;
        vpair(f0, a[0], f2, a[2], s02, d02);
        vpair(f1, a[1], f3, a[3], s13, d13);
        finish<S>(a, s02, d02, s13, d13);
    }
    static __device__ __forceinline__ void run(C2 *a, int S) {
        if (S < 0) run<-1>(a); else run<1>(a);
    }
};

template <class C2>
struct Radix<C2, 8> {
    template <int S>
    static __device__ __forceinline__ void run(C2 *a) {
        C2 e[4] = {a[0], a[2], a[4], a[6]};
        C2 o[4] = {a[1], a[3], a[5], a[7]};
        Radix<C2, 4>::template run<S>(e);
        Radix<C2, 4>::template run<S>(o);
        finish<S>(a, e, o);
    }
    template <int S, class RR>
    static __device__ __forceinline__ void run_scaled(C2 *a, const RR *f) {
        C2 e[4] = {a[0], a[2], a[4], a[6]};
        C2 o[4] = {a[1], a[3], a[5], a[7]};
        Radix<C2, 4>::template run_scaled<S>(e, f[0], f[2], f[4], f[6]);
        Radix<C2, 4>::template run_scaled<S>(o, f[1], f[3], f[5], f[7]);
        finish<S>(a, e, o);
    }
    template <int S>
    static __device__ __forceinline__ void finish(C2 *a, const C2 *e, const C2 *o) {
        using R = decltype(a[0].x);
        const R h = kconst<R>(0.70710678118654752440, -4.833646656726457e-17);
        // twiddles exp(S 2 pi i q/8), q = 1, 2, 3: h t1, S i, h t3
        C2 t1, t3;
        if (S < 0) {
            t1.x = add_rn<R>(o[1].x, o[1].y); t1.y = add_rn<R>(o[1].y, -o[1].x);
            t3.x = add_rn<R>(o[3].y, -o[3].x); t3.y = -add_rn<R>(o[3].x, o[3].y);
        } else {
            t1.x = add_rn<R>(o[1].x, -o[1].y); t1.y = add_rn<R>(o[1].y, o[1].x);
            t3.x = -add_rn<R>(o[3].x, o[3].y); t3.y = add_rn<R>(o[3].x, -o[3].y);
        }
        const C2 w2 = times_si<S>(o[2]);
        a[0] = vadd(e[0], o[0]); a[4] = vsub(e[0], o[0]);
        vaxpy2(e[1], h, t1, a[1], a[5]);
        a[2] = vadd(e[2], w2);   a[6] = vsub(e[2], w2);
        vaxpy2(e[3], h, t3, a[3], a[7]);
    }
    static __device__ __forceinline__ void run(C2 *a, int S) {
        if (S < 0) run<-1>(a); else run<1>(a);
    }
};

// z * w for a constant w = (wr, wi)
__device__ __forceinline__ I2 cmulc(I2 z, long long wr, long long wi) { return vmul(z, WCplx{wsplit(wr), wsplit(wi)}); }
template <class C2, class R>
__device__ __forceinline__ C2 cmulc(C2 z, R wr, R wi) {
    C2 w;
    w.x = wr;
    w.y = wi;
    return vmul(z, w);
}

// 16 = 4 x 4: x[4 n1 + n2] -> radix 4 over n1 (index k1), twiddle W16^(n2 k1),
// radix 4 over n2 (index k2) -> X[k1 + 4 k2], W16 = exp(S 2 pi i / 16).
template <class C2>
struct Radix<C2, 16> {
    template <int S>
    static __device__ __forceinline__ void run(C2 *a) {
        using R = decltype(a[0].x);
        const R c = kconst<R>(0.92387953251128675613), s = kconst<R>(0.38268343236508977173);
        const R h = kconst<R>(0.70710678118654752440);
        const R sg = (R)S;
        C2 y[4][4];
#pragma unroll
        for (int n2 = 0; n2 < 4; ++n2) {
            C2 t[4] = {a[n2], a[4 + n2], a[8 + n2], a[12 + n2]};
            Radix<C2, 4>::template run<S>(t);
#pragma unroll
            for (int k1 = 0; k1 < 4; ++k1) y[n2][k1] = t[k1];
        }
        // W16^m = (cos(2 pi m/16), S sin(2 pi m/16))
        y[1][1] = cmulc(y[1][1], c, sg * s);   // m = 1
        y[1][2] = cmulc(y[1][2], h, sg * h);   // m = 2
        y[1][3] = cmulc(y[1][3], s, sg * c);   // m = 3
        y[2][1] = cmulc(y[2][1], h, sg * h);   // m = 2
        y[2][2] = times_si<S>(y[2][2]);        // m = 4
        y[2][3] = cmulc(y[2][3], -h, sg * h);  // m = 6
        y[3][1] = cmulc(y[3][1], s, sg * c);   // m = 3
        y[3][2] = cmulc(y[3][2], -h, sg * h);  // m = 6
        y[3][3] = cmulc(y[3][3], -c, -sg * s); // m = 9
#pragma unroll
        for (int k1 = 0; k1 < 4; ++k1) {
            C2 t[4] = {y[0][k1], y[1][k1], y[2][k1], y[3][k1]};
            Radix<C2, 4>::template run<S>(t);
#pragma unroll
            for (int k2 = 0; k2 < 4; ++k2) a[k1 + 4 * k2] = t[k2];
        }
    }
    static __device__ __forceinline__ void run(C2 *a, int S) {
        if (S < 0) run<-1>(a); else run<1>(a);
    }
};

template <class C2>
struct Radix<C2, 3> {
    template <int S>
    static __device__ __forceinline__ void run(C2 *a) {
        using R = decltype(a[0].x);
        const R half = kconst<R>(0.5), s3 = kconst<R>(0.86602540378443864676, 5.017542110903451e-17);
        const C2 t1 = vadd(a[1], a[2]), t2 = vsub(a[1], a[2]);
        C2 m;
        if constexpr (std::is_same_v<R, long long>) {
            m = vsub(a[0], ihalf(t1));
        } else {
            m.x = fma_rn<R>(-half, t1.x, a[0].x);
            m.y = fma_rn<R>(-half, t1.y, a[0].y);
        }
        a[0] = vadd(a[0], t1);
        if constexpr (sizeof(R) == 8) {
            vaxpy2(m, s3, times_si<S>(t2), a[1], a[2]);
        } else {
            const C2 r = times_si<S>(vscale(s3, t2));
            a[1] = vadd(m, r);
            a[2] = vsub(m, r);
        }
    }
    static __device__ __forceinline__ void run(C2 *a, int S) {
        if (S < 0) run<-1>(a); else run<1>(a);
    }
};

// 12 = 4 x 3, coprime factors (Good-Thomas, no twiddles): x[(3 n1 + 4 n2) mod 12] ->
// radix 4 over n1 (index k1) for each n2, radix 3 over n2 (index k2) ->
// X[(9 k1 + 4 k2) mod 12], since (3 n1 + 4 n2)(9 k1 + 4 k2) = 3 n1 k1 + 4 n2 k2 mod 12.
template <class C2>
struct Radix<C2, 12> {
    template <int S>
    static __device__ __forceinline__ void run(C2 *a) {
        C2 y[3][4];
#pragma unroll
        for (int n2 = 0; n2 < 3; ++n2) {
            C2 t[4] = {a[(4 * n2) % 12], a[(3 + 4 * n2) % 12], a[(6 + 4 * n2) % 12], a[(9 + 4 * n2) % 12]};
            Radix<C2, 4>::template run<S>(t);
#pragma unroll
            for (int k1 = 0; k1 < 4; ++k1) y[n2][k1] = t[k1];
        }
#pragma unroll
        for (int k1 = 0; k1 < 4; ++k1) {
            C2 t[3] = {y[0][k1], y[1][k1], y[2][k1]};
            Radix<C2, 3>::template run<S>(t);
#pragma unroll
            for (int k2 = 0; k2 < 3; ++k2) a[(9 * k1 + 4 * k2) % 12] = t[k2];
        }
    }
    static __device__ __forceinline__ void run(C2 *a, int S) {
        if (S < 0) run<-1>(a); else run<1>(a);
    }
};

template <class C2>
struct Radix<C2, 5> {
    template <int S>
    static __device__ __forceinline__ void run(C2 *a) {
        using R = decltype(a[0].x);
        const R c1 = kconst<R>(0.30901699437494742410, -2.716057601841253e-17), c2 = kconst<R>(-0.80901699437494742410, 2.716057601841253e-17);
        const R s1 = kconst<R>(0.95105651629515357212, 4.09345009000873e-17), s2 = kconst<R>(0.58778525229247312917, -7.93475083819002e-18);
        const C2 t1 = vadd(a[1], a[4]), t2 = vadd(a[2], a[3]);
        const C2 t3 = vsub(a[1], a[4]), t4 = vsub(a[2], a[3]);
        C2 b1, b2, q1, q2;
        b1.x = fma_rn<R>(c2, t2.x, fma_rn<R>(c1, t1.x, a[0].x)); b1.y = fma_rn<R>(c2, t2.y, fma_rn<R>(c1, t1.y, a[0].y));
        b2.x = fma_rn<R>(c1, t2.x, fma_rn<R>(c2, t1.x, a[0].x)); b2.y = fma_rn<R>(c1, t2.y, fma_rn<R>(c2, t1.y, a[0].y));
        q1.x = fma_rn<R>(s1, t3.x, mul_rn<R>(s2, t4.x)); q1.y = fma_rn<R>(s1, t3.y, mul_rn<R>(s2, t4.y));
        q2.x = fma_rn<R>(s2, t3.x, -mul_rn<R>(s1, t4.x)); q2.y = fma_rn<R>(s2, t3.y, -mul_rn<R>(s1, t4.y));
        q1 = times_si<S>(q1);
        q2 = times_si<S>(q2);
        a[0] = vadd(a[0], vadd(t1, t2));
        a[1] = vadd(b1, q1);
        a[4] = vsub(b1, q1);
        a[2] = vadd(b2, q2);
        a[3] = vsub(b2, q2);
    }
    static __device__ __forceinline__ void run(C2 *a, int S) {
        if (S < 0) run<-1>(a); else run<1>(a);
    }
};

// Coprime factors N = N1 N2 without twiddles (Good-Thomas): x[(N2 n1 + N1 n2) mod N] ->
// radix N1 over n1 (index k1) for each n2, radix N2 over n2 (index k2) ->
// X[(E1 k1 + E2 k2) mod N] with E1 = 1 mod N1, 0 mod N2 and E2 = 0 mod N1, 1 mod N2.
template <class C2, int N1, int N2>
struct GoodThomas {
    static constexpr int N = N1 * N2;
    static constexpr int unit(int m, int other) {  // the multiple of `other` that is 1 mod m
        int e = other;
        while (e % m != 1) e += other;
        return e;
    }
    static constexpr int E1 = unit(N1, N2), E2 = unit(N2, N1);
    template <int S>
    static __device__ __forceinline__ void run(C2 *a) {
        C2 y[N2][N1];
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2) {
            C2 t[N1];
#pragma unroll
            for (int n1 = 0; n1 < N1; ++n1) t[n1] = a[(N2 * n1 + N1 * n2) % N];
            Radix<C2, N1>::template run<S>(t);
#pragma unroll
            for (int k1 = 0; k1 < N1; ++k1) y[n2][k1] = t[k1];
        }
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) {
            C2 t[N2];
#pragma unroll
            for (int n2 = 0; n2 < N2; ++n2) t[n2] = y[n2][k1];
            Radix<C2, N2>::template run<S>(t);
#pragma unroll
            for (int k2 = 0; k2 < N2; ++k2) a[(E1 * k1 + E2 * k2) % N] = t[k2];
        }
    }
};
template <class C2> struct Radix<C2, 6> : GoodThomas<C2, 2, 3> {};
template <class C2> struct Radix<C2, 10> : GoodThomas<C2, 2, 5> {};
template <class C2> struct Radix<C2, 15> : GoodThomas<C2, 3, 5> {};

// 9 = 3 x 3: x[3 n1 + n2] -> radix 3 over n1 (index k1), twiddle W9^(n2 k1), radix 3 over
// n2 (index k2) -> X[k1 + 3 k2].
template <class C2>
struct Radix<C2, 9> {
    template <int S>
    static __device__ __forceinline__ void run(C2 *a) {
        using R = decltype(a[0].x);
        // W9^m = (cos(2 pi m / 9), S sin(2 pi m / 9)), m = 1, 2, 4
        const R c[3] = {kconst<R>(0.76604444311897803520, 2.1750711742081045e-17), kconst<R>(0.17364817766693034885, -1.0090493350843633e-17), kconst<R>(-0.93969262078590838405, 4.385093284002042e-17)};
        const R s[3] = {kconst<R>(S * 0.64278760968653932632, S * -3.659607900790949e-17), kconst<R>(S * 0.98480775301220805937, S * 3.905108875799298e-17), kconst<R>(S * 0.34202014332566873304, S * 2.0136016534644645e-17)};
        C2 y[3][3];
#pragma unroll
        for (int n2 = 0; n2 < 3; ++n2) {
            C2 t[3] = {a[n2], a[3 + n2], a[6 + n2]};
            Radix<C2, 3>::template run<S>(t);
#pragma unroll
            for (int k1 = 0; k1 < 3; ++k1) y[n2][k1] = t[k1];
        }
        y[1][1] = cmulc(y[1][1], c[0], s[0]);
        y[1][2] = cmulc(y[1][2], c[1], s[1]);
        y[2][1] = cmulc(y[2][1], c[1], s[1]);
        y[2][2] = cmulc(y[2][2], c[2], s[2]);
#pragma unroll
        for (int k1 = 0; k1 < 3; ++k1) {
            C2 t[3] = {y[0][k1], y[1][k1], y[2][k1]};
            Radix<C2, 3>::template run<S>(t);
#pragma unroll
            for (int k2 = 0; k2 < 3; ++k2) a[k1 + 3 * k2] = t[k2];
        }
    }
};

// cos(2 pi m / 64) for m = 0 .. 16, and both parts of W64^m for any m by symmetry.
__host__ __device__ constexpr double cos64_quarter(int m) {
    switch (m) {
        case 0: return 1.0;
        case 1: return 0.995184726672196886245;
        case 2: return 0.980785280403230449126;
        case 3: return 0.956940335732208864936;
        case 4: return 0.923879532511286756128;
        case 5: return 0.881921264348355029713;
        case 6: return 0.831469612302545237079;
        case 7: return 0.773010453362736960811;
        case 8: return 0.707106781186547524401;
        case 9: return 0.634393284163645498215;
        case 10: return 0.555570233019602224743;
        case 11: return 0.471396736825997648556;
        case 12: return 0.382683432365089771728;
        case 13: return 0.290284677254462367636;
        case 14: return 0.195090322016128267848;
        case 15: return 0.0980171403295606019942;
        default: return 0.0;
    }
}
__host__ __device__ constexpr double cos64(int m) {
    m &= 63;
    return m <= 16 ? cos64_quarter(m) : (m <= 32 ? -cos64_quarter(32 - m) : (m <= 48 ? -cos64_quarter(m - 32) : cos64_quarter(64 - m)));
}
__host__ __device__ constexpr double sin64(int m) { return cos64((m + 48) & 63); }  // cos(2 pi (m - 16) / 64)

// 32 = 4 x 8: x[8 n1 + n2] -> radix 4 over n1 (index k1), twiddle W32^(n2 k1), radix 8 over
// n2 (index k2) -> X[k1 + 4 k2].
template <class C2>
struct Radix<C2, 32> {
    template <int S>
    static __device__ __forceinline__ void run(C2 *a) {
        using R = decltype(a[0].x);
        C2 y[4][8];
#pragma unroll
        for (int n2 = 0; n2 < 8; ++n2) {
            C2 t[4] = {a[n2], a[8 + n2], a[16 + n2], a[24 + n2]};
            Radix<C2, 4>::template run<S>(t);
#pragma unroll
            for (int k1 = 0; k1 < 4; ++k1) {
                const int m = 2 * n2 * k1;
                if (m == 0) y[k1][n2] = t[k1];
                else if (m == 16) y[k1][n2] = times_si<S>(t[k1]);
                else y[k1][n2] = cmulc(t[k1], kconst<R>(cos64(m)), kconst<R>(S * sin64(m)));
            }
        }
#pragma unroll
        for (int k1 = 0; k1 < 4; ++k1) {
            Radix<C2, 8>::template run<S>(y[k1]);
#pragma unroll
            for (int k2 = 0; k2 < 8; ++k2) a[k1 + 4 * k2] = y[k1][k2];
        }
    }
};

// 64 = 8 x 8: x[8 n1 + n2] -> radix 8 over n1 (index k1), twiddle W64^(n2 k1), radix 8
// over n2 (index k2) -> X[k1 + 8 k2], W64 = exp(S 2 pi i / 64); the twiddles are
// compile-time constants.  For a thread that holds a whole 64-site line in registers.
template <class C2>
struct Radix<C2, 64> {
    template <int S>
    static __device__ __forceinline__ void run(C2 *a) {
        using R = decltype(a[0].x);
        C2 y[8][8];
#pragma unroll
        for (int n2 = 0; n2 < 8; ++n2) {
            C2 t[8];
#pragma unroll
            for (int n1 = 0; n1 < 8; ++n1) t[n1] = a[8 * n1 + n2];
            Radix<C2, 8>::template run<S>(t);
#pragma unroll
            for (int k1 = 0; k1 < 8; ++k1) {
                const int m = n2 * k1;
                if (m == 0) y[n2][k1] = t[k1];
                else if (m == 16) y[n2][k1] = times_si<S>(t[k1]);
                else y[n2][k1] = cmulc(t[k1], kconst<R>(cos64(m)), kconst<R>(S * sin64(m)));
            }
        }
#pragma unroll
        for (int k1 = 0; k1 < 8; ++k1) {
            C2 t[8];
#pragma unroll
            for (int n2 = 0; n2 < 8; ++n2) t[n2] = y[n2][k1];
            Radix<C2, 8>::template run<S>(t);
#pragma unroll
            for (int k2 = 0; k2 < 8; ++k2) a[k1 + 8 * k2] = t[k2];
        }
    }
};

template <class C2, int R, int S, class RR>
__device__ __forceinline__ void radix_scaled(C2 *a, const RR *f) {
    if constexpr (R == 4) {
        Radix<C2, 4>::template run_scaled<S>(a, f[0], f[1], f[2], f[3]);
    } else if constexpr (R == 8) {
        Radix<C2, 8>::template run_scaled<S>(a, f);
    } else {
#pragma unroll
        for (int q = 0; q < R; ++q) a[q] = vscale(f[q], a[q]);
        Radix<C2, R>::template run<S>(a);
    }
}

}  // namespace clv
