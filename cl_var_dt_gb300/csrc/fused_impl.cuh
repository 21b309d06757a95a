// fused_impl.cuh -- the whole Langevin step of 1D chains of 64, 128 or 256 sites, their
// slices in shared memory, in one kernel that streams through imaginary time.
//
// A CTA owns imaginary times [tau0, tau1) of one chain.  Field slices
// (all components of one tau, contiguous in the [c][tau][x][y][z] layout) arrive
// in shared memory by TMA bulk copies (cp.async.bulk + mbarrier), prefetched
// two slices ahead.  For every tau the CTA
//   1. applies the kinetic filter to psi(tau) and psibar(tau+1) in shared
//      memory (FFT of the line, real filter, inverse FFT; FP64 in integers, IntLine);
//   2. computes the drift K(tau), Kbar(tau) of every site from the resident
//      slices psi(tau-1), psi(tau), psi(tau+1), psibar(tau), psibar(tau+1) and the
//      kinetic terms kin(tau-1), kinbar(tau+1);
//   3. adds dt K + sqrt(dt) xi (in-register Philox noise or an injected buffer)
//      and stores psi(tau), psibar(tau) of the new state into the other buffer
//      of the ping-pong pair.
// So each field is read once and written once per step (plus one halo slice per
// CTA), the kinetic term never reaches HBM, and no drift array exists.
//
// The step size depends on max|drift| over the whole chain.  Modes:
//   SPEC    : update with dt = dt_max (the K/max rule's cap) while reducing
//             |K|; the chain's last CTA computes the true dt and marks the step
//             accepted when it equals dt_max.  Otherwise an APPLY pass redoes
//             the chain from the untouched input buffer.  Results are identical
//             to the two-pass order.
//   MAXONLY : reduce only (no stores); the last CTA computes dt.
//   APPLY   : update with the dt of the chain's state (after MAXONLY, or for
//             rejected chains after SPEC).
#pragma once

#include "clv_internal.cuh"
#include "clv_launch.h"
#include "drift_math.cuh"
#include "fft_radix.cuh"

#include <type_traits>

namespace clv {

// ------------------------------------------------------------ TMA / mbarrier
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}"
                 ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load_1d(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Bounded wait: gives up after 0.5 s or 2^22 polls, whichever comes first (far
// beyond any copy's latency), so a copy that never lands cannot hang the GPU.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = globaltimer_ns();
    for (int i = 0; i < (1 << 22); ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 255) == 255 && globaltimer_ns() - t0 > 500000000ull) return false;
    }
    return false;
}

// ---------------------------------------------------------- contiguous lines
// Intermediate layouts are padded with one
// spare element after every 16, which removes the shared-memory bank conflicts
// of the strided Stockham stores.
__device__ __forceinline__ int padi(int i) { return i + (i >> 4); }

// ------------------------------------ compile-time plans for power-of-two lines
// Stockham pass with every size known at compile time (NS a power of two).
// Multiplying by the k = 0 twiddle (exactly 1) leaves values unchanged, so the
// twiddle is applied unconditionally.  PT: tw is this pass's own table
// (tw_*_off), else the length-N table exp(-2 pi i m/N).
// Addresses are a per-lane base plus compile-time offsets: padi(a + b) =
// padi(a) + padi(b) whenever (a mod 16) + (b mod 16) < 16, which holds for the
// loads j + r nR (nR a multiple of 16, or j + r nR < 16 per 16-block) and the
// stores o + q NS (o mod 16 + q NS mod 16 < 16 for power-of-two NS and R).
template <class C2, int N, int R, int NS, int S, bool PS, bool PD, bool PT>
__device__ __forceinline__ void ct_pass(const C2 *s, C2 *d, const C2 *tw, int lane) {
    constexpr int nR = N / R, tstep = N / (NS * R);
#pragma unroll 1
    for (int jj = 0; jj < (nR + 31) / 32; ++jj) {
        const int j = lane + 32 * jj;
        if (nR % 32 != 0 && j >= nR) break;
        const int k = j & (NS - 1);
        const C2 *sl = s + (PS ? padi(j) : j);
        const C2 *twl = PT ? tw + k : tw;
        C2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            C2 x = sl[PS ? padi(r * nR) : r * nR];
            if (NS > 1 && r > 0) {
                C2 t;
                if constexpr (PT) {
                    t = twl[(r - 1) * NS];
                } else {
                    t = tw[k * r * tstep];
                    if (S > 0) t.y = -t.y;
                }
                x = vmul(x, t);
            }
            v[r] = x;
        }
        Radix<C2, R>::template run<S>(v);
        const int o = (j / NS) * NS * R + k;
        C2 *dl = d + (PD ? padi(o) : o);
#pragma unroll
        for (int q = 0; q < R; ++q) dl[PD ? padi(q * NS) : q * NS] = v[q];
    }
}

template <class C2, class RR, int N, int R, bool PS, bool PD, bool PT>
__device__ __forceinline__ void ct_mid(const C2 *s, C2 *d, const C2 *tw, const RR *f, RR cst,
                                       int lane) {
    constexpr int nR = N / R;
#pragma unroll 1
    for (int jj = 0; jj < (nR + 31) / 32; ++jj) {
        const int j = lane + 32 * jj;
        if (nR % 32 != 0 && j >= nR) break;
        const C2 *sl = s + (PS ? padi(j) : j);
        C2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            C2 x = sl[PS ? padi(r * nR) : r * nR];
            if (nR > 1 && r > 0) x = vmul(x, PT ? tw[(r - 1) * nR + j] : tw[j * r]);
            v[r] = x;
        }
        Radix<C2, R>::template run<-1>(v);
        RR g[R];
#pragma unroll
        for (int q = 0; q < R; ++q) g[q] = f[j + q * nR] * cst;
        radix_scaled<C2, R, 1>(v, g);
        C2 *dl = d + (PD ? padi(j * R) : j * R);
#pragma unroll
        for (int q = 0; q < R; ++q) dl[q] = v[q];
    }
}

template <class C2, int N, int P, int NS, bool PT>
__device__ __forceinline__ void ct_fwd(const C2 *&cur, C2 *&nxt, C2 *&oth, const C2 *tw, int lane) {
    constexpr int NF = p2_nfac(N);
    if constexpr (P < NF - 1) {
        constexpr int R = p2_fac(N, P);
        const C2 *twp = PT ? tw + tw_fwd_off(N, P) : tw;
        if constexpr (P == 0) ct_pass<C2, N, R, NS, -1, false, true, PT>(cur, nxt, twp, lane);
        else ct_pass<C2, N, R, NS, -1, true, true, PT>(cur, nxt, twp, lane);
        __syncwarp();
        cur = nxt;
        C2 *t = nxt; nxt = oth; oth = t;
        ct_fwd<C2, N, P + 1, NS * R, PT>(cur, nxt, oth, tw, lane);
    }
}

template <class C2, int N, int P, int NS, bool PT>
__device__ __forceinline__ void ct_inv(const C2 *&cur, C2 *&nxt, C2 *&oth, const C2 *tw, int lane) {
    if constexpr (P >= 0) {
        constexpr int R = p2_fac(N, P);
        const C2 *twp = PT ? tw + tw_inv_off(N, P) : tw;
        if constexpr (P == 0) ct_pass<C2, N, R, NS, 1, true, false, PT>(cur, nxt, twp, lane);
        else ct_pass<C2, N, R, NS, 1, true, true, PT>(cur, nxt, twp, lane);
        __syncwarp();
        cur = nxt;
        C2 *t = nxt; nxt = oth; oth = t;
        ct_inv<C2, N, P - 1, NS * R, PT>(cur, nxt, oth, tw, lane);
    }
}

// Filter of one contiguous line of a compile-time length N = 2^k: src (dense) -> ... ->
// out (dense).  The 2 NF - 1 passes alternate the padded buffers X and Y and end in X ==
// out: out may alias X and Y may alias src (src is read only by the first pass).  PT: tw
// holds the per-pass tables (tw_*_off), else the length-N table.
template <class C2, class RR, int N, bool PT = false>
__device__ __forceinline__ void warp_line_filter_ct(const C2 *src, C2 *X, C2 *Y, const C2 *tw,
                                                    const RR *f, RR cst, int lane) {
    constexpr int NF = p2_nfac(N);
    constexpr int RL = p2_fac(N, NF - 1);
    const C2 *twm = PT ? tw + tw_mid_off(N) : tw;
    if constexpr (NF == 1) {
        ct_mid<C2, RR, N, RL, false, false, PT>(src, X, twm, f, cst, lane);
        __syncwarp();
    } else {
        const C2 *cur = src;
        C2 *nxt = X, *oth = Y;
        ct_fwd<C2, N, 0, 1, PT>(cur, nxt, oth, tw, lane);
        ct_mid<C2, RR, N, RL, true, true, PT>(cur, nxt, twm, f, cst, lane);
        __syncwarp();
        cur = nxt;
        { C2 *t = nxt; nxt = oth; oth = t; }
        ct_inv<C2, N, NF - 2, RL, PT>(cur, nxt, oth, tw, lane);
    }
}

// 256 = 8 8 4: forward pass 1 (7 x 8), middle (3 x 64), inverse 1 (7 x 4), inverse 0 (7 x 32)
static_assert(tw_mid_off(256) == 56 && tw_inv_off(256, 1) == 248 && tw_inv_off(256, 0) == 276 &&
              tw_entries(256) == 500, "pass tables of 256");
static_assert(tw_entries(128) == 56 + 64 + 14 + 112 && tw_entries(64) == 56 + 56, "pass-table sizes");

// ----------------------------------------------- FP64 lines on the integer pipes
// Filter of one contiguous line of N = 64, 128 or 256 sites in block floating point
// (fft_int.cuh) by NT = 32 threads of a warp or 64 of two: Stockham passes of radix 4 (N = 128:
// the middle pass of radix 2), one reduction of the line's largest component after each.  The
// passes of a direction are one loop: unrolled radix-8 passes, executed once per line, spent
// most of their time fetching instructions (a 256-site line of the step loop 15400 clocks).
// The result does not depend on NT.
template <int NT>
__device__ __forceinline__ void group_sync(int id) {
    if constexpr (NT == 32) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(NT) : "memory");
}

// INPLACE: every pass reads its elements, waits for the group and writes them back, without the
// scratch line.
template <int N, int NT, bool INPLACE = false>
struct IntLine {
    static constexpr int LOG = N == 64 ? 6 : (N == 128 ? 7 : 8);
    static constexpr int K4 = (LOG - 1) / 2, RL = N >> (2 * K4);  // forward radix-4 passes, the middle radix
    static constexpr int NB = N / 4, REP = (NB + NT - 1) / NT;
    static_assert((N == 64 || N == 128 || N == 256) && (RL == 2 || RL == 4), "lines of 64, 128 or 256 sites");

    int t, id;
    unsigned *slots;  // NT = 64: four words of shared memory of the group
    int par;
    unsigned mx;      // high word of the line's largest component
    int e;            // shifts so far

    // largest of the group's values, after everything it wrote to shared memory is visible
    __device__ __forceinline__ unsigned reduce(unsigned m) {
        m = __reduce_max_sync(0xffffffffu, m);
        if constexpr (NT == 32) {
            __syncwarp();
        } else {
            if ((t & 31) == 0) slots[2 * par + (t >> 5)] = m;
            group_sync<NT>(id);
            const unsigned a = slots[2 * par], b = slots[2 * par + 1];
            m = a > b ? a : b;
            par ^= 1;
        }
        return m;
    }
    __device__ __forceinline__ void track(unsigned &m, const I2 &v) {
        const unsigned u = imag_bits(v);
        m = u > m ? u : m;
    }

    // src (doubles, read only) -> X (doubles), scratch Y; tw: length-N table, f: the component's
    // filter relative to 2^eg
    __device__ __forceinline__ void run(const double2 *src, double2 *X, double2 *Y, const WCplx *tw, const long long *f,
                                        int eg) {
        par = 0;
        unsigned m = 0;
        double2 d[REP][4];
#pragma unroll
        for (int i = 0; i < REP; ++i) {
            const int j = t + NT * i;
            if (NB % NT == 0 || j < NB)
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    d[i][r] = src[j + r * NB];
                    const unsigned u = mag_bits(d[i][r]);
                    m = u > m ? u : m;
                }
        }
        const unsigned raw = reduce(m);
        const int em = (int)(raw >> 20);
        e = ifirst_for(raw, 4);
        m = 0;
#pragma unroll
        for (int i = 0; i < REP; ++i) {
            const int j = t + NT * i;
            if (NB % NT == 0 || j < NB) {
                I2 v[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) v[r] = I2{to_fixed(d[i][r].x, em, e), to_fixed(d[i][r].y, em, e)};
                Radix<I2, 4>::template run<-1>(v);
                I2 *o = reinterpret_cast<I2 *>(X);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    track(m, v[q]);
                    o[padi(4 * j + q)] = v[q];
                }
            }
        }
        mx = reduce(m);
        const I2 *cur = reinterpret_cast<const I2 *>(X);
        I2 *nxt = reinterpret_cast<I2 *>(INPLACE ? X : Y), *oth = reinterpret_cast<I2 *>(X);
        auto swap = [&]() {
            cur = nxt;
            I2 *x = nxt;
            nxt = oth;
            oth = x;
        };
#pragma unroll 1
        for (int p = 1; p < K4; ++p) {
            pass<-1, false>(cur, nxt, tw, 2 * p, 0, 0);
            swap();
        }
        middle(cur, nxt, tw, f);
        swap();
#pragma unroll 1
        for (int p = 0; p < K4 - 1; ++p) {
            pass<1, false>(cur, nxt, tw, LOG - 2 * K4 + 2 * p, 0, 0);
            swap();
        }
        pass<1, true>(cur, nxt, tw, LOG - 2, em, eg);
    }

    // Radix-4 pass at stride NS = 2^ls; LAST: writes doubles, dense.
    template <int S, bool LAST>
    __device__ __forceinline__ void pass(const I2 *s, I2 *dst, const WCplx *tw, int ls, int em, int eg) {
        const int sh = ishift_for(mx, 4);
        e += sh;
        unsigned m = 0;
        I2 u[REP][4];
        if constexpr (INPLACE) {
#pragma unroll
            for (int i = 0; i < REP; ++i)
                if (const int j = t + NT * i; NB % NT == 0 || j < NB)
#pragma unroll
                    for (int r = 0; r < 4; ++r) u[i][r] = s[padi(j) + padi(r * NB)];
            group_sync<NT>(id);
        }
#pragma unroll
        for (int i = 0; i < REP; ++i) {
            const int j = t + NT * i;
            if (NB % NT == 0 || j < NB) {
                const int k = j & ((1 << ls) - 1);
                const I2 *sl = s + padi(j);
                I2 v[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    v[r] = ishift_down(INPLACE ? u[i][r] : sl[padi(r * NB)], sh);
                    if (r > 0) {
                        const WCplx w = tw[(k * r) << (LOG - 2 - ls)];
                        v[r] = S < 0 ? vmul(v[r], w) : vmulc(v[r], w);
                    }
                }
                Radix<I2, 4>::template run<S>(v);
                const int o = ((j >> ls) << (ls + 2)) + k;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if constexpr (LAST) {
                        reinterpret_cast<double2 *>(dst)[o + (q << ls)] =
                            make_double2(from_fixed(v[q].x, em, eg + e), from_fixed(v[q].y, em, eg + e));
                    } else {
                        track(m, v[q]);
                        dst[padi(o + (q << ls))] = v[q];
                    }
                }
            }
        }
        if constexpr (LAST) group_sync<NT>(id);
        else mx = reduce(m);
    }

    // Last forward pass, filter, first inverse pass.
    __device__ __forceinline__ void middle(const I2 *s, I2 *dst, const WCplx *tw, const long long *f) {
        constexpr int LR = RL == 4 ? 2 : 1, NM = N / RL, REPM = (NM + NT - 1) / NT;
        const int sh = ishift_for(mx, RL);
        e += sh + LR;
        unsigned m = 0;
        I2 u[REPM][RL];
        if constexpr (INPLACE) {
#pragma unroll
            for (int i = 0; i < REPM; ++i)
                if (const int j = t + NT * i; NM % NT == 0 || j < NM)
#pragma unroll
                    for (int r = 0; r < RL; ++r) u[i][r] = s[padi(j + r * NM)];
            group_sync<NT>(id);
        }
#pragma unroll
        for (int i = 0; i < REPM; ++i) {
            const int j = t + NT * i;
            if (NM % NT == 0 || j < NM) {
                I2 v[RL];
#pragma unroll
                for (int r = 0; r < RL; ++r) {
                    v[r] = ishift_down(INPLACE ? u[i][r] : s[padi(j + r * NM)], sh);
                    if (r > 0) v[r] = vmul(v[r], tw[j * r]);
                }
                Radix<I2, RL>::template run<-1>(v);
#pragma unroll
                for (int q = 0; q < RL; ++q) v[q] = ifilter<LR>(f[j + q * NM], v[q]);
                Radix<I2, RL>::template run<1>(v);
#pragma unroll
                for (int q = 0; q < RL; ++q) {
                    track(m, v[q]);
                    dst[padi(j * RL + q)] = v[q];
                }
            }
        }
        mx = reduce(m);
    }
};

// The line filter of a CTA's warps: tables in shared memory and the call for one line.  N: the
// compile-time length (per-pass twiddles twT), 0: n at run time (64, 128 or 256; length-n
// twiddles twS).
template <class R, int N>
struct LineFilter;
template <int N>
struct LineFilter<float, N> {
    const float2 *twS, *twT;
    const float *fS;
    int n;
    // fills the tables at smem + 64 (layout fused_ptw_offset); ends without a barrier
    __device__ __forceinline__ LineFilter(unsigned char *smem, const ChainDev &ch, int n_, int, int) : n(N ? N : n_) {
        float2 *tw = reinterpret_cast<float2 *>(smem + 64), *pt = reinterpret_cast<float2 *>(smem + fused_ptw_offset(n, 8));
        float *f = reinterpret_cast<float *>(smem + 64 + n * sizeof(float2));
        const AxisDev &ax = ch.axis[0];
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            tw[i] = ax.tw32[i];
            f[i] = ax.filt32[i];
        }
        if constexpr (N > 0)
            for (int i = threadIdx.x; i < tw_entries(N); i += blockDim.x) pt[i] = ax.ptw32[i];
        twS = tw; twT = pt; fS = f;
    }
    // kinetic term of component c's line: src (read only) -> X, scratch Y
    template <int NT = 32, bool INPLACE = false>
    __device__ __forceinline__ void run(const ChainDev &ch, bool wc, int c, const float2 *src, float2 *X, float2 *Y,
                                        int lane, int = 0) const {
        static_assert(NT == 32, "FP32 lines take one warp");
        const float cst = wc ? (float)ch.comp_const[c] : 1.0f;
        if constexpr (N > 0) {
            warp_line_filter_ct<float2, float, N, true>(src, X, Y, twT, fS, cst, lane);
        } else {
            switch (n) {
                case 64: warp_line_filter_ct<float2, float, 64>(src, X, Y, twS, fS, cst, lane); break;
                case 128: warp_line_filter_ct<float2, float, 128>(src, X, Y, twS, fS, cst, lane); break;
                default: warp_line_filter_ct<float2, float, 256>(src, X, Y, twS, fS, cst, lane); break;
            }
        }
    }
};
template <int N>
struct LineFilter<double, N> {
    const WCplx *twS;
    const long long *fS;
    unsigned *slots;  // four words for each of four 64-thread groups
    int n;
    __device__ __forceinline__ LineFilter(unsigned char *smem, const ChainDev &ch, int n_, int ncomp, int kinetic)
        : n(N ? N : n_) {
        WCplx *tw = reinterpret_cast<WCplx *>(smem + 64);
        long long *f = reinterpret_cast<long long *>(smem + 64 + n * sizeof(WCplx));
        const AxisDev &ax = ch.axis[0];
        for (int i = threadIdx.x; i < n; i += blockDim.x) tw[i] = static_cast<const WCplx *>(ax.tw62)[i];
        for (int c = 0; c < ncomp; ++c) {
            const double cst = kinetic == CLV_KIN_EXP ? ch.comp_const[c] : 1.0;
            const int e = exp_above(ax.fmax * cst);
            for (int i = threadIdx.x; i < n; i += blockDim.x) f[c * n + i] = filter_fixed(ax.filt64[i] * cst, e);
        }
        __shared__ unsigned sl[16];
        slots = sl;
        twS = tw; fS = f;
    }
    template <int LEN, int NT, bool INPLACE>
    __device__ __forceinline__ void line(const double2 *src, double2 *X, double2 *Y, const long long *f, int eg, int t,
                                         int g) const {
        IntLine<LEN, NT, INPLACE> l;
        l.t = t;
        l.id = 1 + g;
        l.slots = slots + 4 * g;
        l.run(src, X, Y, twS, f, eg);
    }
    // kinetic term of component c's line by thread t of NT: src (read only) -> X, scratch Y; g: the
    // group's number when NT = 64
    template <int NT = 32, bool INPLACE = false>
    __device__ __forceinline__ void run(const ChainDev &ch, bool wc, int c, const double2 *src, double2 *X, double2 *Y,
                                        int t, int g = 0) const {
        const int eg = exp_above(ch.axis[0].fmax * (wc ? ch.comp_const[c] : 1.0));
        const long long *f = fS + c * n;
        if constexpr (N > 0) {
            line<N, NT, INPLACE>(src, X, Y, f, eg, t, g);
        } else {
            switch (n) {
                case 64: line<64, NT, INPLACE>(src, X, Y, f, eg, t, g); break;
                case 128: line<128, NT, INPLACE>(src, X, Y, f, eg, t, g); break;
                default: line<256, NT, INPLACE>(src, X, Y, f, eg, t, g); break;
            }
        }
    }
};

template <class R>
__device__ __forceinline__ const typename Cx<R>::T *tw_of(const AxisDev &ax);
template <> __device__ __forceinline__ const double2 *tw_of<double>(const AxisDev &ax) { return ax.tw64; }
template <> __device__ __forceinline__ const float2 *tw_of<float>(const AxisDev &ax) { return ax.tw32; }
template <class R>
__device__ __forceinline__ const R *filt_of(const AxisDev &ax);
template <> __device__ __forceinline__ const double *filt_of<double>(const AxisDev &ax) { return ax.filt64; }
template <> __device__ __forceinline__ const float *filt_of<float>(const AxisDev &ax) { return ax.filt32; }

// -------------------------------------------------------------- the kernel
// One lattice site per thread.  LN: the chains' line length at compile time, 0: at run time
// (the autotuner's alternative).  FAST (LN > 0 only): the production variant -- K/max step rule,
// in-register Philox noise, bulk copies, no stored drift, both fields per CTA --
// with those choices fixed at compile time, so the per-tau frame carries no
// branches on them.
// Per-site state carried in registers across imaginary times: psi(tau-1),
// kin(tau-1), psibar(tau).

// TWO: the production variant of the FP64 spin-1 model where there is more than one CTA for an
// SM: lines filtered in place and registers for two CTAs an SM.  One CTA's 8 warps issue on 21 %
// of the clocks, waiting on their own arithmetic; two overlap (32 chains of 256 x 128: 771 -> 480
// us a step).  With an SM to itself a CTA is 3 % faster with all the registers.
template <class R, int MODEL, int LN, bool FAST = false, bool TWO = false>
// FP64 1D lines off the production variant (the reference's step rule on few CTAs):
// registers capped at two CTAs' worth, so that the programmatic update's CTAs (its
// noise drawn while this pass runs) fit beside this kernel's on every SM.
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? 3 : (LN > 0 && (TWO || !FAST) ? 2 : 1))
fused_step_kernel(const LaunchFused A) {
    using C2 = typename Cx<R>::T;
    constexpr int NC = MODEL == CLV_MODEL_REF4 ? 4 : 3;
    constexpr int NPS = MODEL == CLV_MODEL_REF4 ? 3 : 2;  // psi slots (REF4 also reads psi(tau+1))
    constexpr int NQS = 2;                                // psibar slots
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int abort_cta;
    // a kernel launched after this one with a programmatic launch (the stored-drift
    // update) may start now; it waits for this grid's end before it reads its results
    asm volatile("griddepcontrol.launch_dependents;");
    const FusedTask task = A.tasks[blockIdx.x];
    const ChainDev &ch = A.chains[task.chain];
    // fields this CTA steps (the production variant always takes both)
    const int side = FAST ? 0 : task.side;
    const bool do_psi = side != 2, do_bar = side != 1;
    // components of this CTA (all unless the chunk is split by component halves)
    const int cmask = (FAST || task.cmask == 0) ? 0xF : task.cmask;
    auto own = [&](int c) { return ((cmask >> c) & 1) != 0; };
    ChainState *st = A.state + task.chain;
    if (A.mode == FUSED_APPLY && A.only_rejected && st->accepted) return;  // uniform per CTA

    const int V = LN ? LN : ch.V, T = ch.nt, cs = LN ? padded_line(LN) : A.comp_stride;
    const int TV = T * V;  // elements of one component of the chain
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem);  // NPS + NQS barriers
    // slot geometry: compile-time for 1D lines of LN sites (the host's formulas, tables of
    // the one filtered axis), so slot addresses are constant offsets
    const int tab_bytes = LN ? fused_tab_bytes(LN, (int)sizeof(C2), LN) : A.tab_bytes;
    const int slot_stride = LN ? fused_slot_stride(NC, LN, (int)sizeof(C2)) : A.slot_stride;
    C2 *slots = reinterpret_cast<C2 *>(smem + tab_bytes);
    auto slot = [&](int i) { return slots + (size_t)i * slot_stride; };
    // slots 0..NPS-1: psi ring; NPS..NPS+NQS-1: psibar ring; then the kinetic
    // results of the two fields, two FFT scratch buffers and the noise of one tau
    C2 *part0 = slot(NPS + NQS), *part1 = slot(NPS + NQS + 1);
    C2 *ybuf0 = slot(NPS + NQS + 2), *ybuf1 = slot(NPS + NQS + 3), *nzbuf = slot(NPS + NQS + (TWO ? 2 : 4));
    const C2 *gpsi = reinterpret_cast<const C2 *>(A.psi_in) + ch.off;
    const C2 *gpsic = reinterpret_cast<const C2 *>(A.psic_in) + ch.off;
    C2 *opsi = reinterpret_cast<C2 *>(A.psi_out) + ch.off;
    C2 *opsic = reinterpret_cast<C2 *>(A.psic_out) + ch.off;
    static_assert(!FAST || LN > 0, "the production variant needs compile-time lines");
    const bool tma = FAST || A.use_tma != 0;
    const bool writes = FAST || A.mode != FUSED_MAXONLY;

    R dt = 0;
    uint64_t nstep = 0;
    if (A.mode == FUSED_SPEC) { dt = (R)ch.dt_max; nstep = st->step; }
    else if (A.mode == FUSED_APPLY) { dt = (R)st->dt; nstep = st->noise_step; }
    const R sd = (R)sqrt((double)dt);

    if (threadIdx.x == 0) {
        abort_cta = 0;
        for (int i = 0; i < NPS + NQS; ++i) mbar_init(&bars[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const LineFilter<R, LN> lines(smem, ch, V, NC, A.kinetic);  // shared twiddle and filter tables
    __syncthreads();

    uint32_t phase = 0, pending = 0;
    auto issue = [&](int sl, const C2 *g, int tau) {
        // periodic wrap: the CTA reads imaginary times tau0 - 1 .. tau1 + 1 of [0, T)
        const int t = tau < 0 ? tau + T : (tau >= T ? tau - T : tau);
        if (tma) {
            if (threadIdx.x == 0) {
                mbar_expect_tx(&bars[sl], (uint32_t)(NC * V * sizeof(C2)));
                for (int c = 0; c < NC; ++c)
                    tma_load_1d(slot(sl) + c * cs, g + ((long long)c * T + t) * V,
                                (uint32_t)(V * sizeof(C2)), &bars[sl]);
            }
            pending |= 1u << sl;
        } else {
            C2 *d = slot(sl);
            for (int e = threadIdx.x; e < NC * V; e += blockDim.x) {
                const int c = e / V, s = e - c * V;
                d[c * cs + s] = g[((long long)c * T + t) * V + s];
            }
        }
    };
    // Only warp 0 polls a copy's barrier; the block barrier that follows every wait
    // orders the landed slice before the other warps' reads (the copy's completion
    // happens before warp 0 passes the wait, which happens before the block barrier).
    auto wait_slot = [&](int sl) {
        if (!(pending & (1u << sl))) return;
        if (threadIdx.x < 32 && !mbar_wait(&bars[sl], (phase >> sl) & 1u)) {
            mbar_wait(&bars[sl], (phase >> sl) & 1u);  // second bounded chance for the copy
            if (threadIdx.x == 0) {
                atomicOr(&st->flags, CLV_FLAG_TIMEOUT);
                abort_cta = 1;
            }
        }
        phase ^= 1u << sl;
        pending &= ~(1u << sl);
    };

    const int tau0 = task.tau0, tau1 = task.tau1;
    const int last_psi = MODEL == CLV_MODEL_REF4 ? tau1 : tau1 - 1;  // last psi time read
    C2 Pp[NC], Kp[NC], Qc[NC];  // psi(tau-1), kin(tau-1), psibar(tau)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = FAST ? 8 : blockDim.x >> 5;
    // One warp per line (2 NC lines); the remaining warps draw the Philox noise of the
    // imaginary time into shared memory meanwhile.
    constexpr int SMEM_PAIRS = (NC + 1) / 2;
    const bool noise_smem =
        writes && (FAST || A.noise == CLV_NOISE_PHILOX) && 2 * NC < nwarps;
    const bool wc = A.kinetic == CLV_KIN_EXP;
    // Filter the lines of `mask` (bit job * NC + c: job 0 = psi of src0 -> X0, job 1 =
    // psibar of src1 -> X1), one warp per line; FP64 lines of 256 on two warps when they fit
    // (the chunks split by field and component halves of the few-CTA problems).
    constexpr bool kPairLines = sizeof(R) == 8 && LN == 256 && !FAST;
    auto filter_lines = [&](int mask, const C2 *src0, C2 *X0, C2 *Y0, const C2 *src1, C2 *X1, C2 *Y1) {
        if constexpr (kPairLines) {
            const int nl = __popc(mask), g = warp >> 1;
            if (2 * nl <= nwarps) {
                if (g < nl) {
                    int m = mask;
                    for (int i = 0; i < g; ++i) m &= m - 1;
                    const int bit = __ffs(m) - 1, job = bit >= NC, c = bit - job * NC;
                    lines.template run<64>(ch, wc, c, (job ? src1 : src0) + c * cs, (job ? X1 : X0) + c * cs,
                                           (job ? Y1 : Y0) + c * cs, threadIdx.x & 63, g);
                }
                return;
            }
        }
        if (warp < 2 * NC && ((mask >> warp) & 1)) {
            const int job = warp >= NC, c = warp - job * NC;
            lines.template run<32, TWO>(ch, wc, c, (job ? src1 : src0) + c * cs, (job ? X1 : X0) + c * cs, (job ? Y1 : Y0) + c * cs, lane);
        }
    };

    // prologue: psi(tau0-1) and its kinetic term, psibar(tau0)
    if (A.withhold && tma && blockIdx.x == 0)
        pending |= 1u;  // test hook: the copy is never issued, so its bounded wait runs out
    else
        issue(0, gpsi, tau0 - 1);
    issue(NPS, gpsic, tau0);
    wait_slot(0);
    wait_slot(NPS);
    __syncthreads();
    const int s = threadIdx.x;
    if (s < V)
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            Pp[c] = slot(0)[c * cs + s];
            Qc[c] = slot(NPS)[c * cs + s];
        }
    filter_lines(do_psi ? cmask & ((1 << NC) - 1) : 0, slot(0), part0, ybuf0, nullptr, nullptr, nullptr);
    __syncthreads();
    if (s < V)
#pragma unroll
        for (int c = 0; c < NC; ++c) Kp[c] = part0[c * cs + s];
    __syncthreads();
    if (!abort_cta) {  // a CTA whose prologue copy timed out issues nothing more and leaves
        for (int i = 0; i < NPS; ++i)
            if (tau0 + i <= last_psi) issue(i, gpsi, tau0 + i);
        for (int i = 0; i < NQS; ++i)
            if (tau0 + 1 + i <= tau1) issue(NPS + i, gpsic, tau0 + 1 + i);
    }

    // step-rule reduction in the working precision per thread (the max is exact;
    // the REF mean sums at most tau1 - tau0 values), FP64 across the CTA
    R mxr = 0, smr = 0;
    int bad = 0;
    const DriftConsts<R> dk(ch);
    // FP64: the pair (psibar(tau), psi(tau-1)) carried from the previous imaginary time (44
    // of the site's 740 FP64 operations; FP32 recomputes it: the registers cost occupancy)
    constexpr bool kCarry = FAST && MODEL == CLV_MODEL_SPIN1 && sizeof(R) == 8;
    Spin1Link<C2> link;
    if constexpr (kCarry) link = spin1_link<R>(dk, Qc, Pp);
    const uint64_t seed = ch.seed;
    const int ref_rule = !FAST && A.dt_rule == CLV_DT_REF_MEANMAX;
    int ia = 0, ic = 0;  // ring positions of psi(tau) and psibar(tau+1)
    for (int tau = tau0; tau < tau1; ++tau) {
        const int sp = ia, spp = (ia + 1) % NPS, sq = NPS + ic;
        wait_slot(sp);
        if (MODEL == CLV_MODEL_REF4) wait_slot(spp);
        wait_slot(sq);
        // every thread is past the previous imaginary time's drift: its slots and
        // the kinetic buffers may be reused from here on
        __syncthreads();
        if (abort_cta) break;
        if (tau > tau0) {
            const int fp = (ia + NPS - 1) % NPS, fq = NPS + (ic + NQS - 1) % NQS;
            if (tau - 1 + NPS <= last_psi) issue(fp, gpsi, tau - 1 + NPS);
            if (tau + NQS <= tau1) issue(fq, gpsic, tau + NQS);
        }
        C2 vpc[NC], vcp[NC], vpp[NC];
        {
            // kin(tau) -> part0, kinbar(tau+1) -> part1; the field slots stay intact
            // (kin(tau) only feeds the next imaginary time: the chunk's last skips it)
            if (warp < 2 * NC || (kPairLines && !noise_smem)) {
                const int own_lines = cmask & ((1 << NC) - 1);
                filter_lines(((do_psi && tau + 1 < tau1) ? own_lines : 0) | (do_bar ? own_lines << NC : 0),
                             slot(sp), part0, ybuf0, slot(sq), part1, ybuf1);
            } else if (noise_smem && LN > 0 && (NC & 1) && NC - 1 < 2 * SMEM_PAIRS) {
                // even lines with a lone component: site pairs (2j, 2j + 1) of the slice, the
                // pair blocks of both sites and their shared lone block drawn together (three
                // independent Philox chains per iteration, a compile-time trip count)
                const int nthr = (nwarps - 2 * NC) * 32, t = (warp - 2 * NC) * 32 + lane;
                constexpr int c = NC - 1;
#pragma unroll 1
                for (int j = t; j < LN / 2; j += nthr) {
                    const int s0 = 2 * j;
                    const uint32_t site = (uint32_t)(tau * LN + s0);
                    uint4 o0[(NC - 1) / 2], o1[(NC - 1) / 2];
#pragma unroll
                    for (int p = 0; p < (NC - 1) / 2; ++p) {
                        o0[p] = philox_block(seed, (uint32_t)task.chain, nstep, p, site);
                        o1[p] = philox_block(seed, (uint32_t)task.chain, nstep, p, site + 1);
                    }
                    const uint4 ol = philox_block(seed, (uint32_t)task.chain, nstep, c >> 1, site >> 1);
#pragma unroll
                    for (int p = 0; p < (NC - 1) / 2; ++p) {
                        nzbuf[2 * p * cs + s0] = unit_normal<R, C2>(o0[p].x, o0[p].y);
                        nzbuf[(2 * p + 1) * cs + s0] = unit_normal<R, C2>(o0[p].z, o0[p].w);
                        nzbuf[2 * p * cs + s0 + 1] = unit_normal<R, C2>(o1[p].x, o1[p].y);
                        nzbuf[(2 * p + 1) * cs + s0 + 1] = unit_normal<R, C2>(o1[p].z, o1[p].w);
                    }
                    nzbuf[c * cs + s0] = unit_normal<R, C2>(ol.x, ol.y);
                    nzbuf[c * cs + s0 + 1] = unit_normal<R, C2>(ol.z, ol.w);
                }
            } else if (noise_smem) {
                const int nthr = (nwarps - 2 * NC) * 32, t = (warp - 2 * NC) * 32 + lane;
                // component pairs: one Philox block per site
                for (int s = t; s < V; s += nthr) {
                    const uint32_t site = (uint32_t)(tau * V + s);
#pragma unroll
                    for (int c = 0; c + 1 < NC && c < 2 * SMEM_PAIRS; c += 2) {
                        const uint4 o = philox_block(seed, (uint32_t)task.chain, nstep, c >> 1, site);
                        nzbuf[c * cs + s] = unit_normal<R, C2>(o.x, o.y);
                        nzbuf[(c + 1) * cs + s] = unit_normal<R, C2>(o.z, o.w);
                    }
                }
                // the lone component of an odd count: one block per two consecutive sites
                // (noise_words); a block straddling the slice's ends serves one site here
                if constexpr ((NC & 1) && NC - 1 < 2 * SMEM_PAIRS) {
                    constexpr int c = NC - 1;
                    const int first = tau * V, last = first + V - 1;
                    for (int j = (first >> 1) + t; j <= (last >> 1); j += nthr) {
                        const uint4 o = philox_block(seed, (uint32_t)task.chain, nstep, c >> 1, (uint32_t)j);
                        const int s0 = 2 * j - first;
                        if (s0 >= 0) nzbuf[c * cs + s0] = unit_normal<R, C2>(o.x, o.y);
                        if (s0 + 1 < V) nzbuf[c * cs + s0 + 1] = unit_normal<R, C2>(o.z, o.w);
                    }
                }
            }
        }
        __syncthreads();
        if (s < V) {
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                vpc[c] = slot(sp)[c * cs + s];
                vcp[c] = slot(sq)[c * cs + s];
                if (MODEL == CLV_MODEL_REF4) vpp[c] = slot(spp)[c * cs + s];
            }
            C2 kp[NC], K[NC], Kc[NC];
            if (!FAST && side) {
#pragma unroll
                for (int c = 0; c < NC; ++c) K[c] = Kc[c] = mk<C2>(0.0, 0.0);
            }
#pragma unroll
            for (int c = 0; c < NC; ++c) kp[c] = part1[c * cs + s];
            if (MODEL == CLV_MODEL_REF4)
                drift_ref4_vals<R>(dk, Pp, vpc, vpp, Qc, vcp, Kp, kp, K, Kc,
                                   FAST ? 3 : (do_psi ? 1 : 0) | (do_bar ? 2 : 0), cmask);
            else if constexpr (kCarry) {
                spin1_drift_psi<R>(link, Pp, vpc, Kp, K);
                link = spin1_link<R>(dk, vcp, vpc);
                spin1_drift_bar<R>(link, vcp, Qc, kp, Kc);
            } else
                drift_spin1_vals<R>(dk, Pp, vpc, Qc, vcp, Kp, kp, K, Kc,
                                    FAST ? 3 : (do_psi ? 1 : 0) | (do_bar ? 2 : 0));
            if (!FAST && A.mode == FUSED_MAXONLY && A.drift_out) {
                // the apply step reads the drift instead of recomputing filter and drift
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    if (!own(c)) continue;
                    const long long gi = ((long long)c * T + tau) * V + s;
                    if (do_psi) reinterpret_cast<C2 *>(A.drift_out)[ch.off + gi] = K[c];
                    if (do_bar) reinterpret_cast<C2 *>(A.driftc_out)[ch.off + gi] = Kc[c];
                }
            }
            if (A.mode != FUSED_APPLY) {
                if (ref_rule) {
                    if (own(0)) {  // (a psibar CTA's K is zero)
                        const R a0 = abs_drift(K[0]);
                        mxr = max_nan(mxr, a0);
                        smr += a0;
                        bad |= not_finite(a0);
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < NC; ++c)
                        if (own(c)) mxr = max_nan(mxr, max_nan(abs2<R>(K[c]), abs2<R>(Kc[c])));
                }
            }
            if (writes) {
                const uint32_t site = (uint32_t)(tau * V + s);
#pragma unroll
                for (int c = 0; c < NC; c += 2) {
                    C2 z[2];
                    if (noise_smem && (c >> 1) < SMEM_PAIRS) {
                        z[0] = nzbuf[c * cs + s];
                        if (c + 1 < NC) z[1] = nzbuf[(c + 1) * cs + s];
                    } else if (FAST || A.noise == CLV_NOISE_PHILOX) {
                        if (c + 1 < NC) {
                            const uint4 o = philox_block(seed, (uint32_t)task.chain, nstep, c >> 1, site);
                            z[0] = unit_normal<R, C2>(o.x, o.y);
                            z[1] = unit_normal<R, C2>(o.z, o.w);
                        } else {
                            const uint2 w = noise_words(seed, (uint32_t)task.chain, nstep, c, NC, site);
                            z[0] = unit_normal<R, C2>(w.x, w.y);
                        }
                    } else {
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            if (c + u >= NC) break;
                            const long long r = ch.noise_off + (((long long)(c + u) * V + s) * T + tau) * 2;
                            z[u].x = (R)A.noise_buf[r];
                            z[u].y = (R)A.noise_buf[r + 1];
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int cc = c + u;
                        if (cc >= NC) break;
                        C2 zz;
                        zz.x = mul_rn<R>(sd, z[u].x);
                        zz.y = mul_rn<R>(sd, z[u].y);
                        const int gi = cc * TV + tau * V + s;  // < 2^31 (plan_fused)
                        if (!own(cc)) continue;
                        if (do_psi) opsi[gi] = langevin_update<R>(vpc[cc], K[cc], dt, zz, false);
                        if (do_bar) opsic[gi] = langevin_update<R>(Qc[cc], Kc[cc], dt, zz, true);
                    }
                }
            }
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                Pp[c] = vpc[c];
                Kp[c] = part0[c * cs + s];
                Qc[c] = vcp[c];
            }
        }
        ia = (ia + 1) % NPS;
        ic = (ic + 1) % NQS;
    }
    // no copy may be in flight when the CTA exits (warp 0 keeps the CTA resident)
    for (int sl = 0; sl < NPS + NQS; ++sl)
        if (pending & (1u << sl)) {
            if (threadIdx.x < 32) mbar_wait(&bars[sl], (phase >> sl) & 1u);
            phase ^= 1u << sl;
        }
    bad |= abort_cta;
    if (A.mode == FUSED_APPLY) return;

    // chain-wide reduction: partial per CTA, the last CTA of the chain finishes the step
    double mx = (double)mxr, sm = (double)smr;
    bad |= !isfinite(mx) || !isfinite(sm);
    bad = __syncthreads_or(bad);
    block_max_sum(mx, sm);
    __shared__ int am_last;
    if (threadIdx.x == 0) {
        A.partials[ch.fused_block0 + task.part] =
            make_double2(mx, bad ? __longlong_as_double(0x7ff8000000000000ll) : sm);
        __threadfence();
        const unsigned prev = atomicAdd(&st->arrive, 1u);
        am_last = prev == (unsigned)ch.fused_nblocks - 1;
    }
    __syncthreads();
    if (!am_last) return;
    __threadfence();
    mx = 0.0;
    sm = 0.0;
    bad = 0;
    for (int i = threadIdx.x; i < ch.fused_nblocks; i += blockDim.x) {
        const double2 p = __ldcg(&A.partials[ch.fused_block0 + i]);
        mx = fmax(mx, p.x);
        sm += p.y;
        bad |= !isfinite(p.y) || !isfinite(p.x);
    }
    bad = __syncthreads_or(bad);
    block_max_sum(mx, sm);
    if (threadIdx.x == 0) {
        double mean;
        const double dtn = step_rule(ch, *st, A.dt_rule, mx, sm, mean);
        if (bad || !isfinite(mx) || !isfinite(sm)) st->flags |= CLV_FLAG_NONFINITE;
        st->dt = dtn;
        st->max = mx;
        st->mean = mean;
        st->t += dtn;
        st->noise_step = st->step;
        st->step += 1;
        st->accepted = (A.mode == FUSED_SPEC && dtn == ch.dt_max) ? 1 : 0;
        if (!st->accepted) st->rejected += (A.mode == FUSED_SPEC);
        st->arrive = 0;
    }
}

// Kernel pointer of one instantiation (defined in k_fused_<precision>_<model>.cu); two: the
// TWO form of the production variant (FP64 spin-1).
void *fused_kernel_f32_ref4(int ln, bool fast);
void *fused_kernel_f32_spin1(int ln, bool fast);
void *fused_kernel_f64_ref4(int ln, bool fast);
void *fused_kernel_f64_spin1(int ln, bool fast, bool two);

template <class R, int MODEL, bool HAS_TWO = false>
void *fused_fn(int ln, bool fast, bool two = false) {
    auto of = [&](auto len) {
        constexpr int LN = decltype(len)::value;
        if (fast && two) return (void *)fused_step_kernel<R, MODEL, LN, true, HAS_TWO>;
        return fast ? (void *)fused_step_kernel<R, MODEL, LN, true> : (void *)fused_step_kernel<R, MODEL, LN>;
    };
    switch (ln) {
        case 64: return of(std::integral_constant<int, 64>{});
        case 128: return of(std::integral_constant<int, 128>{});
        case 256: return of(std::integral_constant<int, 256>{});
        default: break;
    }
    return (void *)fused_step_kernel<R, MODEL, 0>;
}

}  // namespace clv
