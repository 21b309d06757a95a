// fft_int.cuh -- complex arithmetic of the FP64 line filters in 64-bit fixed point.
//
// GB300 retires two FP64 operations per clock and SM, but a 64-bit integer addition takes
// two of its 64 integer lanes and a 64 x 64 product three 32 x 32 -> 64 multiply-adds: a
// butterfly's additions cost a twentieth and its products a third of the FP64 pipe's.  A
// line filter is linear, so its FP64 lines are transformed as block fixed point: every
// line (or slice) is scaled by a power of two of its own, runs forward transform, filter and
// inverse in integers, and is converted back.
//
// * Block floating point: a pass of radix R first shifts its line by the bits that keep R
//   times the largest component, which the pass before it has found, below 2^62.25; the first
//   pass' input is scaled to that.  The shifts add up per line.  The middle pass shifts its
//   product with the filter by ceil(log2 R), for the inverse butterfly whose inputs it has
//   only in registers.
// * Twiddles carry 62 fraction bits (fixed_twiddles), filters 60 relative to the power of two
//   at or above their largest value.  Products are rounded (their low halves' product, at most a
//   unit of the last kept bit and a third of it on average, is dropped); the tile filter's shifts
//   and the radix-3 butterfly's halves are rounded without a bias.
// Values below 2^-1022 count as zero; a line with an infinity or NaN is NaN.  Against
// long-double transforms, over all lines of 8 to 2048 sites: a condensate with fluctuations, and
// one site a thousand times the others, under the exponential filter 0.4 to 1.6 10^-16 in the
// 2-norm, where FP64 butterflies of 8, 4, 2, 3 and 5 give 1.2 to 3.5 10^-16; under k^2 0.4 to
// 4.1 10^-16 against 1.2 to 9.2 10^-16.  No length or filter is further off than they are, in
// the 2-norm or at the worst site.
#pragma once

#include "clv_internal.cuh"

namespace clv {

struct __align__(16) I2 {
    long long x, y;
};
// A factor split for 32-bit products, value h 2^32 + l with l signed.
struct WReal {
    int l, h;
};
struct __align__(16) WCplx {
    WReal x, y;
};
__host__ __device__ __forceinline__ constexpr WReal wsplit(long long w) {
    return WReal{(int)(unsigned)(unsigned long long)w,
                 (int)((w - (long long)(int)(unsigned)(unsigned long long)w) >> 32)};
}
struct ISplit {
    int l, h;
};
__device__ __forceinline__ ISplit isplit(long long z) {
    ISplit s;
    s.l = (int)(unsigned)(unsigned long long)z;
    s.h = (int)(z >> 32) + (int)((unsigned)s.l >> 31);
    return s;
}
// (z w) >> Q: high product and the two cross products; the product of the low halves, at most
// 2^62 in either direction, is dropped (2^62 is a unit of the result at Q = 62).
template <int Q>
__device__ __forceinline__ long long imulq(long long z, WReal w) {
    const ISplit s = isplit(z);
    const long long cross = (long long)s.h * w.l + ((long long)s.l * w.h + (1ll << (Q - 33)));
    return ((long long)s.h * w.h << (64 - Q)) + (cross >> (Q - 32));
}
constexpr int kTwQ = 62, kFiltQ = 60, kTop = 62;

__device__ __forceinline__ I2 vadd(I2 a, I2 b) { return I2{a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ I2 vsub(I2 a, I2 b) { return I2{a.x - b.x, a.y - b.y}; }
// z w and z conj(w)
template <bool CONJ>
__device__ __forceinline__ I2 imul(I2 z, WCplx w) {
    const ISplit a = isplit(z.x), b = isplit(z.y);
    const long long half = 1ll << (kTwQ - 33);
    const long long cx = CONJ ? (long long)a.h * w.x.l + (long long)a.l * w.x.h + (long long)b.h * w.y.l + (long long)b.l * w.y.h + half
                              : (long long)a.h * w.x.l + (long long)a.l * w.x.h - (long long)b.h * w.y.l - (long long)b.l * w.y.h + half;
    const long long cy = CONJ ? (long long)b.h * w.x.l + (long long)b.l * w.x.h - (long long)a.h * w.y.l - (long long)a.l * w.y.h + half
                              : (long long)b.h * w.x.l + (long long)b.l * w.x.h + (long long)a.h * w.y.l + (long long)a.l * w.y.h + half;
    const long long hx = CONJ ? (long long)a.h * w.x.h + (long long)b.h * w.y.h : (long long)a.h * w.x.h - (long long)b.h * w.y.h;
    const long long hy = CONJ ? (long long)b.h * w.x.h - (long long)a.h * w.y.h : (long long)b.h * w.x.h + (long long)a.h * w.y.h;
    return I2{(hx << (64 - kTwQ)) + (cx >> (kTwQ - 32)), (hy << (64 - kTwQ)) + (cy >> (kTwQ - 32))};
}
__device__ __forceinline__ I2 vmul(I2 z, WCplx w) { return imul<false>(z, w); }
__device__ __forceinline__ I2 vmulc(I2 z, WCplx w) { return imul<true>(z, w); }
// products with the butterflies' real constants (62 fraction bits)
__device__ __forceinline__ I2 vscale(long long s, I2 z) {
    const WReal w = wsplit(s);
    return I2{imulq<kTwQ>(z.x, w), imulq<kTwQ>(z.y, w)};
}
__device__ __forceinline__ void vaxpy2(I2 e, long long s, I2 z, I2 &p, I2 &m) {
    const I2 w = vscale(s, z);
    p = vadd(e, w);
    m = vsub(e, w);
}
template <> __device__ __forceinline__ long long add_rn<long long>(long long a, long long b) { return a + b; }
template <> __device__ __forceinline__ long long mul_rn<long long>(long long c, long long z) { return imulq<kTwQ>(z, wsplit(c)); }
template <> __device__ __forceinline__ long long fma_rn<long long>(long long c, long long z, long long s) {
    return s + imulq<kTwQ>(z, wsplit(c));
}
// z 2^-s and z / 2, rounded: a value half way between two goes up or down by the other part's
// last bit.  A truncating shift, or halves that always go up, would be off in one direction at
// every element of a pass, which the passes that follow add up at a few sites of the line
// (lines of 900 sites: 3 to 4 times the error of the others there).
__device__ __forceinline__ I2 ishift(I2 z, int s) {
    const long long half = (1ll << s) >> 1;
    const int any = s > 0;
    return I2{(z.x + (half - ((int)z.y & any))) >> s, (z.y + (half - ((int)z.x & any))) >> s};
}
__device__ __forceinline__ I2 ihalf(I2 z) { return I2{(z.x + ((int)z.y & 1)) >> 1, (z.y + ((int)z.x & 1)) >> 1}; }
// z 2^-s rounded down, for the radix-4 passes of lines of up to 256 sites: their errors are 0.1 to
// 0.3 of the FP64 butterflies' either way (at the worst site 0.6), and the step of 256 chains of
// 256 x 128 takes 4.07 ms instead of 4.26.
__device__ __forceinline__ I2 ishift_down(I2 z, int s) { return I2{z.x >> s, z.y >> s}; }
// High word of the magnitude of a line's largest component.
__device__ __forceinline__ unsigned imag_bits(I2 z) {
    const int a = (int)(z.x >> 32), b = (int)(z.y >> 32);
    const unsigned u = (unsigned)(a ^ (a >> 31)), v = (unsigned)(b ^ (b >> 31));
    return u > v ? u : v;
}
// Shifts before a butterfly of R inputs: the least that keeps R times a component below
// 2^62.25, so that the outputs, of up to sqrt(2) times that, keep within 63 bits and their
// products with twiddles too (imul's cross products: 2^30.75 2^31.5 + 2^31.5 2^30 < 2^63).
// Counting R as the next power of two, and the component too, would leave up to two bits of the
// 62 unused in every pass: a condensate fills them all at one frequency, and what it leaves to the
// others is their precision (lines of 729 and 900 sites: 1.3 times the FP64 butterflies' error, now 0.7).
// ishift_for: of a component with the high word mag; ifirst_for: of a double with the high
// word raw, which to_fixed puts in [2^61, 2^62).
__device__ __forceinline__ int ishift_for(unsigned mag, int r) {
    const unsigned long long t = (unsigned long long)(mag + 1u) * (unsigned)r;  // units of 2^32
    const int s = 33 - __clzll((long long)t);                                   // t >> s in [2^30, 2^31)
    return s < 0 ? 0 : s + ((t >> s) > 1276901416ull);                          // 2^30.25
}
__device__ __forceinline__ int ifirst_for(unsigned raw, int r) {
    const unsigned t = ((raw & 0xfffffu) + 0x100001u) * (unsigned)r;  // units of 2^41
    const int s = 10 - __clz((int)t);                                 // t >> s in [2^21, 2^22)
    return s + ((t >> s) > 2493948u);                                 // 2^21.25
}
// product with a filter value (kFiltQ fraction bits), shifted by another S <= 4 bits
template <int S>
__device__ __forceinline__ I2 ifilter(long long f, I2 z) {
    static_assert(kFiltQ + S <= 64, "shift of the high product");
    const WReal w = wsplit(f);
    return I2{imulq<kFiltQ + S>(z.x, w), imulq<kFiltQ + S>(z.y, w)};
}

// Conversions, by moving bits (a product and a conversion each way on the FP64 pipe measured
// 3 to 6 % slower).  emax: biased exponent of the line's largest component, which goes to
// [2^(kTop - 1), 2^kTop) >> s.  Values below 2^-1022 count as zero.
__device__ __forceinline__ long long to_fixed(double x, int emax, int s) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const int ex = (int)((hi >> 20) & 0x7ffu), r = (ex ? emax : 8192) - ex + (64 - kTop) + s;
    const unsigned long long m = ((unsigned long long)(0x80000000u | (hi << 11) | (lo >> 21)) << 32) | (lo << 11);
    const unsigned long long v = r > 63 ? 0ull : m >> r;
    return (hi >> 31) ? -(long long)v : (long long)v;
}
// The double nearest v 2^e times the unit of to_fixed at s = 0; NaN for a line with an
// infinity or NaN.  (Zero below, infinity above the normal range.)
__device__ __forceinline__ double from_fixed(long long v, int emax, int e) {
    if (emax == 0x7ff) return __longlong_as_double(0x7ff8000000000000ll);
    const unsigned long long a = v < 0 ? 0 - (unsigned long long)v : (unsigned long long)v;
    if (a == 0) return 0.0;
    const int l = __clzll((long long)a);
    const unsigned long long m = a << l;
    const int be = emax + e - l + (64 - kTop);  // biased exponent
    unsigned long long b = ((unsigned long long)(be - 1) << 52) + (m >> 11) + ((m >> 10) & 1);
    if (be < 1 || be > 2046) b = be < 1 ? 0 : 0x7ff0000000000000ull;
    return __longlong_as_double((long long)(v < 0 ? b | 0x8000000000000000ull : b));
}
// 2^e as a double, -1022 <= e <= 1023
__device__ __forceinline__ double pow2(int e) { return __hiloint2double((e + 1023) << 20, 0); }
// least e with x <= 2^e, x > 0 finite and normal
__device__ __forceinline__ int exp_above(double x) {
    const int hi = __double2hiint(x), e = ((hi >> 20) & 0x7ff) - 1023;
    return e + (((hi & 0xfffff) | __double2loint(x)) != 0);
}
// Table entry: a filter value relative to 2^e.
__device__ __forceinline__ long long filter_fixed(double f, int e) { return __double2ll_rn(f * pow2(kFiltQ - e)); }

// Exponent word of the largest component, for a line's maximum.
__device__ __forceinline__ unsigned mag_bits(double2 z) {
    const unsigned a = (unsigned)__double2hiint(z.x) & 0x7fffffffu, b = (unsigned)__double2hiint(z.y) & 0x7fffffffu;
    return a > b ? a : b;
}

}  // namespace clv
