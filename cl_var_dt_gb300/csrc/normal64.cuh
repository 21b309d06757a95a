// normal64.cuh -- unit complex normals at FP64 accuracy on the integer pipes.
//
// Box-Muller of two 32-bit words, u1 = (x + 1/2) 2^-32, u2 = y 2^-32:
//   r = sqrt(-2 ln u1),  z = r (cos 2 pi u2 + i sin 2 pi u2).
// GB300 retires two FP64 operations per clock and SM, and log, sincospi and sqrt of a
// double take about 75 of them: 40 clocks of the SM's FP64 pipe for one complex normal,
// which made the noise the largest part of every FP64 step.  The inputs are integers, so
// the whole transform runs in 64-bit fixed point instead (a 64 x 64 -> high 64 product
// costs a sixth of a clock per SM, an addition a fortieth), and only the two finished
// doubles are assembled, also by integer operations.  Measured: the stored-drift update of
// the reference model on 128 x 128 x 128 imaginary times (four normals a site) 2.52 -> 0.40
// ms, 0.84 of the copy bandwidth; the FP64 step of 32 chains of 256 x 128 2.26 -> 1.56 ms.
//
// * ln u1, table-driven after Tang (ACM TOMS 16, 1990): u1 = a 2^-33 with the odd integer
//   a = 2x + 1 = m 2^e, 1 <= m < 2; c = c_i / 512 near 1 / m by the top 7 fraction bits
//   of m, so that r = m c - 1 is an exact integer with |r| <= 2^-7, and
//   -2 ln u1 = 2 (32 - e) ln 2 + 2 ln(2 c) - 2 ln(1 + r), the last by its Taylor series
//   to r^9.  The table's ends are exact (c = 1 and 1/2), so nothing cancels near u1 = 1.
// * sqrt: a single-precision reciprocal square root refined by one third-order step on
//   the residual 1 - y^2 v, which is formed exactly.
// * cos, sin: the nearest multiple of pi/4 is split off the integer angle exactly; the
//   remainder, |a| <= pi/8, by Taylor series to the 16th (sine 15th) power.
// Error below 0.65 units in the last place of each returned part (mean 0.25, as correct
// rounding has), against 128-bit arithmetic over 3 million words and all special ones.
#pragma once

#include <stdint.h>

#if defined(__CUDACC__)
#define CLV_HD __device__ __forceinline__
#else
#include <cmath>
#include <cstring>
#define CLV_HD inline
#endif

namespace clv {

// {2 ln(2 c_i) 2^62, c_i}: c_i = 512 / (interval midpoint) rounded, exact at both ends
struct LogEntry {
    uint64_t t;
    uint64_t c;
};
#if defined(__CUDACC__)
static __device__ const LogEntry kLogTable[128] = {
#else
static const LogEntry kLogTable[128] = {
#endif
    {0x58B90BFBE8E7BCD6ull, 512}, {0x5736C771B05D9234ull, 506}, {0x5632B6D735E624C2ull, 502}, {0x552C919E66525EA4ull, 498},
    {0x54669302E8D1199Bull, 495}, {0x535CB4E8E7F4011Dull, 491}, {0x5250AA0E8BF01DEDull, 487}, {0x51862F08717B09F4ull, 484},
    {0x50763FA119CAB992ull, 480}, {0x4FA8CE4DACBD6E0Full, 477}, {0x4E94DCF9FAF7E632ull, 473}, {0x4DC45ED51D1ED717ull, 470},
    {0x4CAC4CE44875C4C8ull, 466}, {0x4BD8AA65425518B6ull, 463}, {0x4B03A7B5123A2EE6ull, 460}, {0x4A2D4037D81E0ABCull, 457},
    {0x49556F3A63DF2CF0ull, 454}, {0x483373464AADB64Dull, 450}, {0x475843F99DC00C21ull, 447}, {0x467B9AD19F25BB31ull, 444},
    {0x459D72AEAE98380Eull, 441}, {0x44BDC6564FBEF14Cull, 438}, {0x43DC90726D25F53Bull, 435}, {0x43458F32E75ADF82ull, 433},
    {0x4261BD3D5CD482E4ull, 430}, {0x417C52F49916702Aull, 427}, {0x40954A969743FB1Aull, 424}, {0x3FAC9E41EC2AE395ull, 421},
    {0x3F10946DFD3D8459ull, 419}, {0x3E251EBF5E0DD967ull, 416}, {0x3D37F4CB30C3EAC9ull, 413}, {0x3C98E350D0EE085Aull, 411},
    {0x3BA8D4098389417Eull, 408}, {0x3B07CE4B145E7CA1ull, 406}, {0x3A14C75CE43CC84Bull, 403}, {0x3971C0E89AF593FBull, 401},
    {0x387BAF4F9B5A9AE7ull, 398}, {0x37D69B3B4E36F7EFull, 396}, {0x3730B12D2621F6B3ull, 394}, {0x36363C1D7BF8B6D2ull, 391},
    {0x358E3184B161C818ull, 389}, {0x34E5492CD7B3D42Dull, 387}, {0x33E647D97F3097E5ull, 384}, {0x333B2B022FC11597ull, 382},
    {0x328F2838422DF575ull, 380}, {0x31E23D0E6CC58EFCull, 378}, {0x3134670D8284B56Bull, 376}, {0x302DE83B41A92B6Bull, 373},
    {0x2F7DBC146F5F7F3Cull, 371}, {0x2ECC9C2473B79D82ull, 369}, {0x2E1A85C4F1246BABull, 367}, {0x2D6776446B287B13ull, 365},
    {0x2CB36AE607C3E504ull, 363}, {0x2BFE60E14F27A791ull, 361}, {0x2B485561E99FC339ull, 359}, {0x2A9145875BA4C5A0ull, 357},
    {0x29D92E64C004D35Full, 355}, {0x29200D008013A198ull, 353}, {0x2865DE5409D0276Bull, 351}, {0x2808610D0D4FC77Aull, 350},
    {0x274C98AAD28BD38Eull, 348}, {0x268FBB3530FAA9ADull, 346}, {0x25D1C575C23A6138ull, 344}, {0x2512B427BD0D46BDull, 342},
    {0x245283F79EF2CB45ull, 340}, {0x23F1FF3C9145E51Bull, 339}, {0x23301A5BA846DECFull, 337}, {0x226D0E05275160BEull, 335},
    {0x220B17F35C95AA31ull, 334}, {0x214649C4E721C6BFull, 332}, {0x20804B2969A081B6ull, 330}, {0x201CD88B5AA0398Dull, 329},
    {0x1F550A564B7B3707ull, 327}, {0x1E8C0252AA5A5FE9ull, 325}, {0x1E27076E2AF2E5EAull, 324}, {0x1D5C216B4FBB915Cull, 322},
    {0x1C8FF7C79A9A21ACull, 320}, {0x1C2968558C18C0A3ull, 319}, {0x1B5B519E8FB5A46Full, 317}, {0x1AF3C94E80BFF2D9ull, 316},
    {0x1A23BC1FE2B56319ull, 314}, {0x19BB362E7DFB8356ull, 313}, {0x18E928DE886D40AAull, 311}, {0x187FA06520C91090ull, 310},
    {0x17AB890210D9091Cull, 308}, {0x1740F8F54037A4CAull, 307}, {0x16D60FE719D21C8Dull, 306}, {0x15FF3070A793D3C8ull, 304},
    {0x159338D9982085D3ull, 303}, {0x14BA36F39A55E55Aull, 301}, {0x144D2B6CCB7D1E68ull, 300}, {0x13DFC2B0ECC629CBull, 299},
    {0x1303D718E47FD2FFull, 297}, {0x129552F81FF5234Cull, 296}, {0x12266F190A5ACB7Dull, 295}, {0x114785846742AC69ull, 293},
    {0x10D77E7CD08E5967ull, 292}, {0x10671512CA596E2Aull, 291}, {0x0F85186008B15331ull, 289}, {0x0F1383B7157972F5ull, 288},
    {0x0EA189EB3659AEAFull, 287}, {0x0E2F2A47ADE3A18Bull, 286}, {0x0D49369D256AB1B3ull, 284}, {0x0CD5A1231019D66Eull, 283},
    {0x0C61A2EB18CD907Bull, 282}, {0x0BED3B36BD896642ull, 281}, {0x0B032C549BA861D9ull, 279}, {0x0A8D839F830C1FB5ull, 278},
    {0x0A176E5F5323781Eull, 277}, {0x09A0EBCB0DE8E849ull, 276}, {0x0929FB17850A0B7Cull, 275}, {0x08B29B7751BD7074ull, 274},
    {0x07C28C300458A998ull, 272}, {0x0749DAE2B6C2D484ull, 271}, {0x06D0B75C465C6FB1ull, 270}, {0x065720C3B238FADFull, 269},
    {0x05DD163D8CB73F12ull, 268}, {0x056296EBF2393523ull, 267}, {0x04E7A1EE7FAF57EAull, 266}, {0x046C366248F65FF1ull, 265},
    {0x03F05361CF06600Aull, 264}, {0x0373F804F5F232FFull, 263}, {0x02F72360FAB62355ull, 262}, {0x0279D48868D4AE9Eull, 261},
    {0x01FC0A8B0FC03E3Dull, 260}, {0x017DC475F810A76Eull, 259}, {0x00FF015358833C48ull, 258}, {0x0000000000000000ull, 256},
};

#if defined(__CUDACC__)
CLV_HD uint64_t umulhi64(uint64_t a, uint64_t b) { return __umul64hi(a, b); }
CLV_HD int64_t smulhi64(int64_t a, int64_t b) { return __mul64hi(a, b); }
CLV_HD uint32_t umulhi32(uint32_t a, uint32_t b) { return __umulhi(a, b); }
CLV_HD int32_t smulhi32(int32_t a, int32_t b) { return __mulhi(a, b); }
CLV_HD int lead64(uint64_t a) { return __clzll((long long)a); }
CLV_HD int lead32(uint32_t a) { return __clz((int)a); }
CLV_HD float rsqrt_seed(float v) { return rsqrtf(v); }
CLV_HD double bits_double(uint64_t b) { return __longlong_as_double((long long)b); }
CLV_HD LogEntry log_entry(int i) {
    const ulonglong2 e = __ldg(reinterpret_cast<const ulonglong2 *>(kLogTable) + i);
    LogEntry r;
    r.t = e.x; r.c = e.y;
    return r;
}
#else
CLV_HD uint64_t umulhi64(uint64_t a, uint64_t b) { return (uint64_t)(((unsigned __int128)a * b) >> 64); }
CLV_HD int64_t smulhi64(int64_t a, int64_t b) { return (int64_t)(((__int128)a * b) >> 64); }
CLV_HD uint32_t umulhi32(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
CLV_HD int32_t smulhi32(int32_t a, int32_t b) { return (int32_t)(((int64_t)a * b) >> 32); }
CLV_HD int lead64(uint64_t a) { return a ? __builtin_clzll(a) : 64; }
CLV_HD int lead32(uint32_t a) { return a ? __builtin_clz(a) : 32; }
CLV_HD float rsqrt_seed(float v) { return 1.0f / sqrtf(v); }
CLV_HD double bits_double(uint64_t b) { double d; memcpy(&d, &b, 8); return d; }
CLV_HD LogEntry log_entry(int i) { return kLogTable[i]; }
#endif
// (a b) >> 32 of a 64-bit and a 32-bit factor
CLV_HD uint64_t mul64x32hi(uint64_t a, uint32_t b) {
    return (uint64_t)(uint32_t)(a >> 32) * b + (((uint64_t)(uint32_t)a * b) >> 32);
}

// -2 ln u1 of the word x as v 2^ex, 2^63 <= v < 2^64.
CLV_HD uint64_t neg2log_fixed(uint32_t x, int &ex) {
    const uint64_t a = 2 * (uint64_t)x + 1;
    const int lz = lead64(a), e = 63 - lz;                  // a = m 2^e, 0 <= e <= 32
    const LogEntry t = log_entry((int)((a << lz) >> 56) & 127);
    // r = a c 2^-(e+9) - 1 in units of 2^-63 (exact: 43 significant bits), |r| <= 2^-7
    const int64_t r = (int64_t)((a * t.c - (512ull << e)) << (54 - e));
    const int64_t rs = (int64_t)((uint64_t)r << 6);         // 64 r
    const int32_t r32 = (int32_t)(rs >> 32);
    // ln(1 + r) / r = 1 - r/2 + r^2/3 - ... + r^8/9: Horner, 32 bits for the powers r^4 ...
    int32_t q = 0x10000000 - (smulhi32(r32, 0x0E38E38E) >> 5);            // 1/8 - r/9, units 2^-31
    q = 0x12492492 - (smulhi32(r32, q) >> 5);
    q = 0x15555555 - (smulhi32(r32, q) >> 5);
    q = 0x1999999A - (smulhi32(r32, q) >> 5);                             // 1/5 - r (1/6 - ...)
    int64_t p = 0x2000000000000000ll - (smulhi64(rs, (int64_t)((uint64_t)(uint32_t)q << 32)) >> 5);  // 1/4 - ..., units 2^-63
    p = 0x2AAAAAAAAAAAAAABll - (smulhi64(rs, p) >> 5);
    p = 0x4000000000000000ll - (smulhi64(rs, p) >> 5);
    const uint64_t P = 0x8000000000000000ull - (uint64_t)(smulhi64(rs, p) >> 5);  // in (0.99, 1.01) 2^63
    // |ln(1 + r)| = w 2^-(62 + s) with |r| normalised first, so that a tiny r keeps its bits
    const bool neg = r < 0;
    const uint64_t ra = neg ? 0 - (uint64_t)r : (uint64_t)r;
    // (its least magnitude but 0 is 2^22; the bit set here bounds the shift below at r = 0, whose w is 0)
    const int s = lead64(ra | 256);                         // 7 .. 55
    const uint64_t w = umulhi64(ra << s, P);
    // sum in units of 2^-62 for e = 32 (a sum below 1.39), of 2^-58 else (below 46)
    const int sh = e == 32 ? 0 : 4;
    const uint64_t k = (uint64_t)(32 - e) * 0x058B90BFBE8E7BCDull + (t.t >> sh);
    const uint64_t d = w >> (s - 1 + sh);
    uint64_t v = neg ? k + d : k - d;
    ex = sh - 62;
    if (k == 0) { v = w; ex = -61 - s; }                    // u1 within 2^-8 of 1 (r < 0 there)
    const int l = lead64(v);
    ex -= l;
    return v << l;
}

// sqrt(v 2^ex) as s 2^es, 2^63 <= s < 2^64.
CLV_HD uint64_t sqrt_fixed(uint64_t v, int ex, int &es) {
    const int odd = ex & 1;
    v >>= odd;                                              // X = v 2^-62 in [1, 4)
    ex += odd;
    const float y0 = rsqrt_seed((float)(uint32_t)(v >> 32) * 9.31322574615478515625e-10f);  // 2^-30
    float yf = y0 * 2147483648.0f;
    const uint32_t y = (uint32_t)(yf < 2147483648.0f ? yf : 2147483648.0f);  // units 2^-31
    const uint64_t s0 = mul64x32hi(v, y);                   // X y, units 2^-61
    // residual 1 - y s0, units 2^-64 (the product's integer part wraps away)
    const int64_t r = (int64_t)(0 - (((uint64_t)(uint32_t)(s0 >> 32) * y << 4) + (((uint64_t)(uint32_t)s0 * y) >> 28)));
    const int64_t h = r >> 13;
    const int64_t corr = (r >> 1) + ((3 * ((h * h) >> 38)) >> 3);  // (1 - r)^(-1/2) - 1 = r/2 + 3 r^2/8
    const uint64_t s = s0 + (uint64_t)smulhi64((int64_t)s0, corr);
    es = (ex + 62) / 2 - 63;                                // ex + 62 is even
    // s in [1, 2) 2^61 up to its last units: keep the top bit in place at both ends
    const uint64_t one = 1ull << 61;
    return (s < one ? one : s >= 2 * one ? 2 * one - 1 : s) << 2;
}

// The double nearest (-1)^neg m 2^e.
CLV_HD double assemble64(uint64_t m, int e, bool neg) {
    if (m == 0) return 0.0;
    const int l = lead64(m);
    m <<= l;
    const uint64_t f = (m >> 11) + ((m >> 10) & 1);         // 53 bits, rounded
    const uint64_t b = ((uint64_t)(e - l + 63 + 1022) << 52) + f;
    return bits_double(neg ? b | 0x8000000000000000ull : b);
}

// Real and imaginary parts of the unit complex normal of the words (x, y).
CLV_HD void normal64(uint32_t x, uint32_t y, double &re, double &im) {
    int ex, es;
    const uint64_t v = neg2log_fixed(x, ex);
    const uint64_t s = sqrt_fixed(v, ex, es);
    // angle 2 pi y 2^-32 = o pi/4 + sign(a) |a| 2 pi 2^-32, |a| <= 2^28
    const uint32_t o = ((y + 0x10000000u) >> 29) & 7u;
    const int32_t ai = (int32_t)(y - (o << 29));
    const bool an = ai < 0;
    const uint32_t a = an ? 0u - (uint32_t)ai : (uint32_t)ai;
    const uint64_t u = (uint64_t)a * a << 7;                // (a 2^-28)^2, units 2^-63
    const uint32_t u32 = (uint32_t)(u >> 32);               // units 2^-31
    // sin = (a 2^-28) (pi/8) sum_k (-1)^k ((pi/8)^2 u)^k / (2k + 1)!: units 2^-64; the powers
    // u^4 ... in 32 bits (units 2^-62)
    uint32_t q = 0x00000F48u - (umulhi32(u32, 3u) << 1);
    q = 0x003C60EAu - (umulhi32(u32, q) << 1);
    q = 0xA83C1A44u - (umulhi32(u32, q) << 1);
    uint64_t g = 0x000004CB4B3398AFull - (umulhi64(u, (uint64_t)q << 2) << 1);
    g = 0x000519AF19DD6AB8ull - (umulhi64(u, g) << 1);
    g = 0x0295779CC4B7CA58ull - (umulhi64(u, g) << 1);
    g = 0x6487ED5110B4611Aull - (umulhi64(u, g) << 1);
    // cos = 1 - ..., units 2^-63; the powers u^4 ... in 32 bits (units 2^-58)
    uint32_t c32 = 0x00001F9Du - (umulhi32(u32, 7u) << 1);
    c32 = 0x0069B47Du - (umulhi32(u32, c32) << 1);
    c32 = 0xF0FA8345u - (umulhi32(u32, c32) << 1);
    uint64_t c = 0x00002ABA78FC7980ull - (umulhi64(u, (uint64_t)c32 << 5) << 1);
    c = 0x0020783E1036B587ull - (umulhi64(u, c) << 1);
    c = 0x09DE9E64DF22EF2Dull - (umulhi64(u, c) << 1);
    c = 0x8000000000000000ull - (umulhi64(u, c) << 1);
    // |sin| = t 2^-(60 + la) with the integer angle normalised first
    const int la = lead32(a | 1u);                          // >= 3
    const uint64_t t = mul64x32hi(g, a << la);
    uint64_t A = c, B = t;
    int ea = -63, eb = -60 - la;
    bool nb = an;
    if (o & 1u) {                                           // cos, sin of pi/4 + the remainder
        const uint64_t sn = t >> (la - 3);                  // units 2^-63
        const uint64_t lo = c - sn, hi = c + sn;
        A = umulhi64(an ? hi : lo, 0xB504F333F9DE6484ull);
        B = umulhi64(an ? lo : hi, 0xB504F333F9DE6484ull);
        eb = -63;
        nb = false;
    }
    // quadrant o / 2: (A, B), (-B, A), (-A, -B), (B, -A)
    const bool swap = (o & 2u) != 0;
    const bool half = (o & 4u) != 0;                        // quadrants 2 and 3
    const uint64_t ma = umulhi64(s, swap ? B : A), mb = umulhi64(s, swap ? A : B);
    const int e1 = es + 64 + (swap ? eb : ea), e2 = es + 64 + (swap ? ea : eb);
    const bool n1 = swap ? nb == half : half, n2 = swap ? half : nb != half;
    re = assemble64(ma, e1, n1);
    im = assemble64(mb, e2, n2);
}

}  // namespace clv
