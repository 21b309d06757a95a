// k_tile.cuh -- kinetic filter of lattices without a kernel of their own: lines of any
// length 2^a 3^b 5^c, whole small slices, and strided or contiguous tiles of large ones.
//
// A task is a tile of one field held in shared memory: `rows` rows of `cols` elements at
// a pitch without bank conflicts (tile_pitch).  It is one of
//   * whole slices: consecutive (component, imaginary time) slices of a chain, rows along
//     the innermost axis; every filtered axis is transformed while the slice is on chip, so
//     a 2D or 3D slice is read and written once;
//   * a strided tile: all n sites of one axis (the rows) for `cols` adjacent lines;
//   * a contiguous tile: `rows` lines of the innermost axis.
// Lines are filtered in place (decimation in frequency, the filter at the digit-reversed
// frequencies, decimation in time; see inplace_fft.cuh) with a plan of two or three
// radices of 2 .. 16 that the host chose for the length: 60 = 10 x 6 takes three passes
// over shared memory.  Butterfly b of a pass is butterfly b / NL of line b mod NL, so a
// warp works on 32 lines at a time however short they are, conflict-free along rows and
// across them; the divisions are multiplications by a reciprocal that the
// thread computes once per pass.
//
// FP64 lines run in block floating point on the integer pipes (fft_int.cuh): a pass over the
// raw tile finds every line's largest component (every slice's, when several axes are
// filtered), the first pass converts as it reads and the last one converts back as it
// writes.  A filter that vanishes at zero frequency (k^2: the reference's kinetic term and all
// kinetic energies) does not see a constant, so its lines are taken relative to their first
// site: a condensate would fill the top bits at a frequency that is then thrown away (lines of 1250
// sites: 2.2 times the FP64 butterflies' error, now 0.4 to 0.8; kBasedSites).  128-site lines, 4 components x 128 x 128 x 128 imaginary times, both fields: 1.37
// (butterflies on the FP64 pipe, at its rate) -> 0.58 ms; 48-site lines of 48 x 40 x 36 x 24:
// 0.93 -> 0.39 ms.  Bound by integer issue (48 % of the ALU) and instruction fetch.
//
// FP32 is bound by instruction issue (61 %, 170 instructions an element, a third of them
// addresses) and the latency between its barriers.  64 ragged chains, 1.6 M sites: 78 us.
#pragma once

#include "clv_internal.cuh"
#include "clv_launch.h"
#include "fft_radix.cuh"

namespace clv {

// x / d for x d < 2^32 by the reciprocal ceil(2^32 / d) (0 stands for d = 1).
struct FastDiv {
    uint32_t m;
    __device__ __forceinline__ explicit FastDiv(int d) : m(d > 1 ? 0xFFFFFFFFu / (uint32_t)d + 1u : 0u) {}
    __device__ __forceinline__ int div(int x) const { return m ? (int)__umulhi((uint32_t)x, m) : x; }
};

// Geometry of the lines of one axis of a tile: the rows themselves (along), or element a of
// line l at hi n es + y PZ + x + a es, l = hi I + y cols + x, I the lines between two
// blocks of the axis.
struct TileLines {
    int NL, n, es, PZ, I, cols;
    bool along;
    FastDiv dI, dcols, dNL;
    __device__ __forceinline__ TileLines(int rows, int cols_, int PZ_, int n_, int I_, bool along_)
        : NL(along_ ? rows : rows * cols_ / n_), n(n_), es(along_ ? 1 : PZ_ * (I_ / cols_)), PZ(PZ_), I(I_), cols(cols_),
          along(along_), dI(I_), dcols(cols_), dNL(NL) {}
    __device__ __forceinline__ int base(int l) const {
        if (along) return l * PZ;
        const int hi = dI.div(l), lo = l - hi * I;
        const int y = I > cols ? dcols.div(lo) : 0;
        return hi * n * es + y * (PZ - cols) + lo;
    }
};

// Arithmetic of the tile's passes: element type, twiddle and filter types.
template <class R> struct TileMath;
template <> struct TileMath<float> { using E = float2; using W = float2; using F = float; };
template <> struct TileMath<double> { using E = I2; using W = WCplx; using F = long long; };

// FP64: the lines' scale.  Line l belongs to group l / lines per group; of each group, raw: the
// high word of the largest component as the doubles came in; cur, next: of the largest one
// after the pass before this one and after this one (zero: cleared for the pass after);
// exps: the shifts so far.  first: the pass reads doubles; last: it writes them.  eg: the
// filters' power of two.
struct TileScale {
    unsigned *raw, *cur, *next, *zero;
    int *exps;
    FastDiv group;
    int ng, eg;
    bool first, last;
    __device__ __forceinline__ void advance() {
        unsigned *t = cur;
        cur = next; next = zero; zero = t;
        first = false;
    }
};

enum { TILE_DIF = 0, TILE_MID = 1, TILE_DIT = 2, TILE_MAX = 3 };

__host__ __device__ constexpr int ceil_log2(int n) { return n <= 1 ? 0 : 1 + ceil_log2((n + 1) / 2); }

// One pass of radix R over the tile.  TILE_DIF: forward pass of span L (S = L / R), twiddles
// after the butterfly unless S = 1.  TILE_MID: the last forward pass, the filter (f in the
// passes' order of frequencies, plus the line's share fo of the other axes when it is not
// null), the first inverse pass.  TILE_DIT: the inverse of TILE_DIF.  TILE_MAX (FP64): the
// largest component of every group.
template <class RR, int R, int KIND>
__device__ __forceinline__ void tile_pass(typename Cx<RR>::T *t, const TileLines &g, int L, int S,
                                          const typename TileMath<RR>::W *tw, const typename TileMath<RR>::F *f,
                                          const typename TileMath<RR>::F *fo, const TileScale &sc) {
    using C2 = typename Cx<RR>::T;
    using E = typename TileMath<RR>::E;
    constexpr bool kInt = sizeof(RR) == 8;
    constexpr int LR = ceil_log2(R);
    const int NB = g.NL * (g.n / R), ts = g.n / L;
    const FastDiv dS(S);
    const int st = S * g.es;
#pragma unroll 1
    for (int b = threadIdx.x; b < NB; b += blockDim.x) {
        const int j = g.dNL.div(b), l = b - j * g.NL;
        const int blk = KIND == TILE_MID ? j : dS.div(j), k = KIND == TILE_MID ? 0 : j - blk * S;
        C2 *p = t + g.base(l) + (blk * L + k) * g.es;
        if constexpr (KIND == TILE_MAX) {
            if constexpr (kInt) {
                unsigned mx = 0;
#pragma unroll
                for (int m = 0; m < R; ++m) {
                    const unsigned v = mag_bits(p[m * st]);
                    mx = v > mx ? v : mx;
                }
                atomicMax(&sc.raw[sc.group.div(l)], mx);
            }
        } else {
            E v[R];
            int gr = 0;
            if constexpr (kInt) {
                gr = sc.group.div(l);
                if (sc.first) {
                    const int em = (int)(sc.raw[gr] >> 20), sf = ifirst_for(sc.raw[gr], R);
#pragma unroll
                    for (int m = 0; m < R; ++m) {
                        const double2 d = p[m * st];
                        v[m] = I2{to_fixed(d.x, em, sf), to_fixed(d.y, em, sf)};
                    }
                } else {
                    const int sh = ishift_for(sc.cur[gr], R);
#pragma unroll
                    for (int m = 0; m < R; ++m) v[m] = ishift(*reinterpret_cast<const I2 *>(p + m * st), sh);
                }
            } else {
#pragma unroll
                for (int m = 0; m < R; ++m) v[m] = p[m * st];
            }
            if constexpr (KIND == TILE_DIF) {
                Radix<E, R>::template run<-1>(v);
                if (S > 1) {
                    const int step = k * ts;
#pragma unroll
                    for (int q = 1; q < R; ++q) v[q] = vmul(v[q], tw[q * step]);
                }
            } else if constexpr (KIND == TILE_DIT) {
                if (S > 1) {
                    const int step = k * ts;
#pragma unroll
                    for (int q = 1; q < R; ++q) v[q] = vmulc(v[q], tw[q * step]);
                }
                Radix<E, R>::template run<1>(v);
            } else {
                Radix<E, R>::template run<-1>(v);
                typename TileMath<RR>::F o = 0;
                if (fo) o = fo[l];
#pragma unroll
                for (int q = 0; q < R; ++q) {
                    if constexpr (kInt) v[q] = ifilter<LR>(f[blk * R + q] + o, v[q]);
                    else v[q] = vscale(f[blk * R + q] + o, v[q]);
                }
                Radix<E, R>::template run<1>(v);
            }
            if constexpr (kInt) {
                if (KIND != TILE_DIF && sc.last) {
                    const int em = (int)(sc.raw[gr] >> 20);
                    const int e = sc.eg + sc.exps[gr] + (KIND == TILE_MID ? LR : 0) +
                                  (sc.first ? ifirst_for(sc.raw[gr], R) : ishift_for(sc.cur[gr], R));
#pragma unroll
                    for (int m = 0; m < R; ++m) p[m * st] = make_double2(from_fixed(v[m].x, em, e), from_fixed(v[m].y, em, e));
                } else {
                    unsigned mx = 0;
#pragma unroll
                    for (int m = 0; m < R; ++m) {
                        const unsigned u = imag_bits(v[m]);
                        mx = u > mx ? u : mx;
                        *reinterpret_cast<I2 *>(p + m * st) = v[m];
                    }
                    atomicMax(&sc.next[gr], mx);
                }
            } else {
#pragma unroll
                for (int m = 0; m < R; ++m) p[m * st] = v[m];
            }
        }
    }
    if constexpr (kInt && KIND != TILE_MAX) {
        if (!sc.last)  // (the last pass reads exps)
            for (int i = threadIdx.x; i < sc.ng; i += blockDim.x) {
                sc.exps[i] += (KIND == TILE_MID ? LR : 0) + (sc.first ? ifirst_for(sc.raw[i], R) : ishift_for(sc.cur[i], R));
                sc.zero[i] = 0;
            }
    }
    __syncthreads();
}

template <class RR, int KIND>
__device__ __forceinline__ void tile_pass_any(int R, typename Cx<RR>::T *t, const TileLines &g, int L, int S,
                                              const typename TileMath<RR>::W *tw, const typename TileMath<RR>::F *f,
                                              const typename TileMath<RR>::F *fo, const TileScale &sc) {
    switch (R) {
        case 2: tile_pass<RR, 2, KIND>(t, g, L, S, tw, f, fo, sc); break;
        case 3: tile_pass<RR, 3, KIND>(t, g, L, S, tw, f, fo, sc); break;
        case 4: tile_pass<RR, 4, KIND>(t, g, L, S, tw, f, fo, sc); break;
        case 5: tile_pass<RR, 5, KIND>(t, g, L, S, tw, f, fo, sc); break;
        case 6: tile_pass<RR, 6, KIND>(t, g, L, S, tw, f, fo, sc); break;
        case 8: tile_pass<RR, 8, KIND>(t, g, L, S, tw, f, fo, sc); break;
        case 9: tile_pass<RR, 9, KIND>(t, g, L, S, tw, f, fo, sc); break;
        case 10: tile_pass<RR, 10, KIND>(t, g, L, S, tw, f, fo, sc); break;
        default:
            if constexpr (tile_radix_max<RR>() >= 16) {
                if (R == 12) tile_pass<RR, 12, KIND>(t, g, L, S, tw, f, fo, sc);
                else if (R == 15) tile_pass<RR, 15, KIND>(t, g, L, S, tw, f, fo, sc);
                else tile_pass<RR, 16, KIND>(t, g, L, S, tw, f, fo, sc);
            }
    }
}

template <class R> __device__ __forceinline__ const typename TileMath<R>::W *tile_tw(const AxisDev &ax);
template <> __device__ __forceinline__ const WCplx *tile_tw<double>(const AxisDev &ax) { return static_cast<const WCplx *>(ax.tw62); }
template <> __device__ __forceinline__ const float2 *tile_tw<float>(const AxisDev &ax) { return ax.tw32; }
template <class R> __device__ __forceinline__ const R *tile_filt(const AxisDev &ax, int energy);
template <> __device__ __forceinline__ const double *tile_filt<double>(const AxisDev &ax, int energy) {
    return energy ? ax.tefilt64 : ax.tfilt64;
}
template <> __device__ __forceinline__ const float *tile_filt<float>(const AxisDev &ax, int energy) {
    return energy ? ax.tefilt32 : ax.tfilt32;
}

// Global to shared without registers (8 or 16 bytes per thread), and the wait for it.
#if defined(__CUDACC__)
template <class C2>
__device__ __forceinline__ void copy_async(C2 *s, const C2 *g) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(s)), "l"(g),
                 "n"((int)sizeof(C2))
                 : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
#else  // host build of the tests
template <class C2> inline void copy_async(C2 *s, const C2 *g) { *s = *g; }
inline void copy_async_commit() {}
inline void copy_async_wait() {}
#endif

// TH threads: 128, or 256 for the large slices.
template <class R, int TH>
__global__ void __launch_bounds__(TH, tile_min_ctas<R>(TH)) tile_filter_kernel(const LaunchTileFilter A) {
    using C2 = typename Cx<R>::T;
    using W = typename TileMath<R>::W;
    using F = typename TileMath<R>::F;
    constexpr bool kInt = sizeof(R) == 8;
    static_assert(sizeof(W) == sizeof(C2) && sizeof(F) == sizeof(R), "tables take the elements' sizes");
    extern __shared__ __align__(128) unsigned char smem[];
    const int bid = A.nfields == 2 ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
    const int field = A.nfields == 2 ? (int)(blockIdx.x & 1) : 0;
    const TileFilterTask task = A.tasks[bid];
    const TileFilterPlan &P = A.plans[task.plan];
    const ChainDev &ch = A.chains[task.chain];
    const int rows = task.rows, cols = task.cols, PZ = P.pitch, nax = P.naxes;
    const bool energy = A.filter != 0, summed = energy && nax > 1;
    C2 *tile = reinterpret_cast<C2 *>(smem);
    W *tw0 = reinterpret_cast<W *>(tile + P.tile_elems);
    const long long off = ch.off + (long long)task.slice * ch.V + task.off;
    const C2 *src = reinterpret_cast<const C2 *>(field ? A.src1 : A.src0) + off;
    C2 *dst = reinterpret_cast<C2 *>(field ? A.dst1 : A.dst0) + off;
    const int total = rows * cols;
    const FastDiv dc(cols);
    // element e of the tile: row e / cols, column e % cols; rows follow one another in global
    // memory (gstride = cols) or lie an axis stride apart
    const int gs = P.gstride ? P.gstride : cols;
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
        const int r = dc.div(e), c = e - r * cols;
        copy_async(tile + r * PZ + c, src + (long long)r * gs + c);
    }
    copy_async_commit();
    // tables of the filtered axes: twiddles, then the filters in the passes' order of
    // frequencies, the component constant folded into the first axis' one
    int nsum = 0;
    for (int a = 0; a < nax; ++a) nsum += ch.axis[P.axis[a]].n;
    // (FP64, a filter that vanishes at zero frequency: the groups' first sites between them)
    F *f0 = reinterpret_cast<F *>(tw0 + nsum + (kInt && P.based ? (nax == 1 ? total / ch.axis[P.axis[0]].n : total / ch.V) : 0));
    F *fo = f0 + nsum;  // summed filters: the rows' shares of the other axes
    TileScale sc{nullptr, nullptr, nullptr, nullptr, nullptr, FastDiv(1), 0, 0, false, false};
    {
        // FP64: the filters relative to the power of two at or above their largest value (of
        // each axis, or of the sum)
        if constexpr (kInt) {
            if (summed) {
                double most = 0, n = 1;
                for (int a = 0; a < nax; ++a) n *= ch.axis[P.axis[a]].n;
                for (int a = 0; a < nax; ++a) most += ch.axis[P.axis[a]].efmax * (ch.axis[P.axis[a]].n / n);
                sc.eg = exp_above(most);
            }
        }
        int o = 0;
        for (int a = 0; a < nax; ++a) {
            const AxisDev &ax = ch.axis[P.axis[a]];
            const W *tw = tile_tw<R>(ax);
            const R *f = tile_filt<R>(ax, energy);
            // energy: sum of the axes' k^2/2; each axis' table carries 1/n, and the sum over
            // axes of a slice's transforms needs the product of all 1/n on every term
            R cst = (a == 0 && P.with_const && !energy) ? (R)ch.comp_const[task.slice / ch.nt] : (R)1;
            if (energy)
                for (int b = 0; b < nax; ++b)
                    if (b != a) cst /= (R)ch.axis[P.axis[b]].n;
            if constexpr (kInt) {
                int e = sc.eg;
                if (!summed) {
                    e = exp_above((energy ? ax.efmax : ax.fmax) * cst);
                    sc.eg += e;
                }
                cst *= pow2(kFiltQ - e);
            }
            for (int i = threadIdx.x; i < ax.n; i += blockDim.x) {
                tw0[o + i] = tw[i];
                if constexpr (kInt) f0[o + i] = __double2ll_rn(f[i] * cst);
                else f0[o + i] = f[i] * cst;
            }
            o += ax.n;
        }
    }
    // lines of axis a (P.inner: tile elements, padding aside, between two of its sites)
    auto lines = [&](int a) {
        return TileLines(rows, cols, PZ, ch.axis[P.axis[a]].n, P.inner[a] == 0 ? cols : P.inner[a], P.inner[a] == 1);
    };
    // FP64: one scale per line, or per slice when several axes mix its lines
    auto group = [&](int a) {
        if constexpr (kInt) sc.group = FastDiv(nax == 1 ? 1 : ch.V / ch.axis[P.axis[a]].n);
    };
    if constexpr (kInt) {
        sc.ng = nax == 1 ? total / ch.axis[P.axis[0]].n : total / ch.V;
        sc.raw = reinterpret_cast<unsigned *>(fo + (summed ? rows : 0));
        sc.cur = sc.raw + sc.ng;
        sc.next = sc.cur + sc.ng;
        sc.zero = sc.next + sc.ng;
        sc.exps = reinterpret_cast<int *>(sc.zero + sc.ng);
        for (int i = threadIdx.x; i < 5 * sc.ng; i += blockDim.x) sc.raw[i] = 0;
    }
    copy_async_wait();
    __syncthreads();
    if constexpr (kInt) {
        const AxisDev &ax = ch.axis[P.axis[0]];
        group(0);
        if (P.based) {
            // element e: line (slice of a sum) hi I + (e mod I), whose first one is hi per + (e mod I)
            double2 *base = reinterpret_cast<double2 *>(tw0 + nsum);
            const int I = nax > 1 ? 1 : (P.inner[0] == 0 ? cols : P.inner[0]), per = nax > 1 ? ch.V : ax.n * I;
            const FastDiv dp(per), dI(I);
            auto at = [&](int e) {
                const int r = dc.div(e);
                return tile + r * PZ + (e - r * cols);
            };
            for (int i = threadIdx.x; i < sc.ng; i += blockDim.x) {
                const int hi = dI.div(i);
                base[i] = *at(hi * per + (i - hi * I));
            }
            __syncthreads();
            for (int e = threadIdx.x; e < total; e += blockDim.x) {
                const int hi = dp.div(e), lo = e - hi * per;
                C2 *p = at(e);
                *p = vsub(*p, base[hi * I + (lo - dI.div(lo) * I)]);
            }
            __syncthreads();
        }
        tile_pass_any<R, TILE_MAX>(ax.tfac[0], tile, lines(0), ax.n, ax.n / ax.tfac[0], nullptr, nullptr, nullptr, sc);
    }
    // forward passes of one axis (all of them when `whole`), the middle one, the inverse ones
    auto forward = [&](const TileLines &g, const AxisDev &ax, const W *tw, bool whole) {
        int L = ax.n;
        for (int p = 0; p < (whole ? ax.tnf : ax.tnf - 1); ++p) {
            const int rad = ax.tfac[p];
            tile_pass_any<R, TILE_DIF>(rad, tile, g, L, L / rad, tw, nullptr, nullptr, sc);
            sc.advance();
            L /= rad;
        }
    };
    auto middle = [&](const TileLines &g, const AxisDev &ax, const W *tw, const F *f, const F *fr, bool end) {
        const int rad = ax.tfac[ax.tnf - 1];
        sc.last = end && ax.tnf == 1;
        tile_pass_any<R, TILE_MID>(rad, tile, g, rad, 1, tw, f, fr, sc);
        sc.advance();
    };
    auto inverse = [&](const TileLines &g, const AxisDev &ax, const W *tw, bool whole, bool end) {
        int S = whole ? 1 : ax.tfac[ax.tnf - 1];
        for (int p = (whole ? ax.tnf : ax.tnf - 1) - 1; p >= 0; --p) {
            const int rad = ax.tfac[p];
            sc.last = end && p == 0;
            tile_pass_any<R, TILE_DIT>(rad, tile, g, S * rad, S, tw, nullptr, nullptr, sc);
            sc.advance();
            S *= rad;
        }
    };
    sc.first = true;
    if (!summed) {
        // product of the axes' filters: one axis after the other
        int o = 0;
        for (int a = 0; a < nax; ++a) {
            const AxisDev &ax = ch.axis[P.axis[a]];
            const TileLines g = lines(a);
            group(a);
            const bool end = a == nax - 1;
            forward(g, ax, tw0 + o, false);
            middle(g, ax, tw0 + o, f0 + o, nullptr, end);
            inverse(g, ax, tw0 + o, false, end);
            o += ax.n;
        }
    } else {
        // sum of the axes' filters: every axis forward, the sum at each frequency, and back
        // (the last axis is the innermost: its lines are the tile's rows, whose share of the
        // other axes' filters goes into fo)
        int o = 0;
        for (int a = 0; a + 1 < nax; ++a) {
            const AxisDev &ax = ch.axis[P.axis[a]];
            group(a);
            forward(lines(a), ax, tw0 + o, true);
            o += ax.n;
        }
        for (int r = threadIdx.x; r < rows; r += blockDim.x) {
            F v = 0;
            int o2 = 0;
            for (int a = 0; a + 1 < nax; ++a) {
                const int n = ch.axis[P.axis[a]].n, I = P.inner[a] == 0 ? cols : P.inner[a];
                v += f0[o2 + r / (I / cols) % n];
                o2 += n;
            }
            fo[r] = v;
        }
        __syncthreads();
        {
            const AxisDev &ax = ch.axis[P.axis[nax - 1]];
            const TileLines g = lines(nax - 1);
            group(nax - 1);
            forward(g, ax, tw0 + o, false);
            middle(g, ax, tw0 + o, f0 + o, fo, false);
            inverse(g, ax, tw0 + o, false, false);
        }
        for (int a = nax - 2; a >= 0; --a) {
            const AxisDev &ax = ch.axis[P.axis[a]];
            o -= ax.n;
            group(a);
            inverse(lines(a), ax, tw0 + o, true, a == 0);
        }
    }
    const bool acc = A.accumulate != 0;
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
        const int r = dc.div(e), c = e - r * cols;
        C2 *d = dst + (long long)r * gs + c;
        const C2 v = tile[r * PZ + c];
        *d = acc ? cadd(*d, v) : v;
    }
}

// Allows the kernel the device's whole opt-in shared memory: it serves every shape, and a limit
// raised by one engine could be lowered again by another that is created beside it.
template <class R>
cudaError_t setup_tile_filter(size_t smem_bytes, int threads, int *ctas_per_sm) {
    const void *fn = threads == 128 ? (const void *)tile_filter_kernel<R, 128> : (const void *)tile_filter_kernel<R, 256>;
    int dev = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaFuncAttributes fa{};
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, fn);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes);
    if (e != cudaSuccess) return e;
    *ctas_per_sm = 0;
    if (smem_bytes + fa.sharedSizeBytes > (size_t)optin) return cudaSuccess;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas_per_sm, fn, threads, smem_bytes);
}

template <class R>
cudaError_t launch_tile_filter(const LaunchTileFilter &L, cudaStream_t s) {
    if (L.ntasks == 0) return cudaSuccess;
    void *args[] = {const_cast<LaunchTileFilter *>(&L)};
    const void *fn = L.threads == 128 ? (const void *)tile_filter_kernel<R, 128> : (const void *)tile_filter_kernel<R, 256>;
    return cudaLaunchKernel(fn, dim3(L.nfields * L.ntasks), dim3(L.threads), args, L.smem_bytes, s);
}

}  // namespace clv
