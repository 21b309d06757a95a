// k_tile.cuh -- kinetic filter of lattices without a kernel of their own: lines of any
// length 2^a 3^b 5^c, whole small slices, and strided or contiguous tiles of large ones.
//
// A task is a tile of one field held in shared memory: `rows` rows of `cols` elements at
// an odd pitch.  It is one of
//   * whole slices: consecutive (component, imaginary time) slices of a chain, rows along
//     the innermost axis; every filtered axis is transformed while the slice is on chip, so
//     a 2D or 3D slice is read and written once;
//   * a strided tile: all n sites of one axis (the rows) for `cols` adjacent lines;
//   * a contiguous tile: `rows` lines of the innermost axis.
// Lines are filtered in place (decimation in frequency, the filter at the digit-reversed
// frequencies, decimation in time; see inplace_fft.cuh) with a plan of two or three
// radices of 2 .. 16 that the host chose for the length: 60 = 10 x 6 takes three passes
// over shared memory.  Butterfly b of a pass is butterfly b / NL of line b mod NL, so a
// warp works on 32 lines at a time however short they are, conflict-free along rows (odd
// pitch) and across them; the divisions are multiplications by a reciprocal that the
// thread computes once per pass.
//
// Bound by the passes over shared memory and the latency between their barriers.  Against
// the one-warp-per-line plans that these lengths had (a 60-site line gave a warp 15
// butterflies of radix 4): see plan_tiled for the paths and figures.
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

enum { TILE_DIF = 0, TILE_MID = 1, TILE_DIT = 2 };

// One pass of radix R over the tile.  TILE_DIF: forward pass of span L (S = L / R), twiddles
// after the butterfly unless S = 1.  TILE_MID: the last forward pass, the filter (f in the
// passes' order of frequencies, plus the line's share fo of the other axes when it is not
// null), the first inverse pass.  TILE_DIT: the inverse of TILE_DIF.
template <class C2, class RR, int R, int KIND>
__device__ __forceinline__ void tile_pass(C2 *t, const TileLines &g, int L, int S, const C2 *tw, const RR *f,
                                          const RR *fo) {
    const int NB = g.NL * (g.n / R), ts = g.n / L;
    const FastDiv dS(S);
    const int st = S * g.es;
#pragma unroll 1
    for (int b = threadIdx.x; b < NB; b += blockDim.x) {
        const int j = g.dNL.div(b), l = b - j * g.NL;
        const int blk = KIND == TILE_MID ? j : dS.div(j), k = KIND == TILE_MID ? 0 : j - blk * S;
        C2 *p = t + g.base(l) + (blk * L + k) * g.es;
        C2 v[R];
#pragma unroll
        for (int m = 0; m < R; ++m) v[m] = p[m * st];
        if constexpr (KIND == TILE_DIF) {
            Radix<C2, R>::template run<-1>(v);
            if (S > 1) {
                const int step = k * ts;
#pragma unroll
                for (int q = 1; q < R; ++q) v[q] = vmul(v[q], tw[q * step]);
            }
        } else if constexpr (KIND == TILE_DIT) {
            if (S > 1) {
                const int step = k * ts;
#pragma unroll
                for (int q = 1; q < R; ++q) {
                    C2 w = tw[q * step];
                    w.y = -w.y;
                    v[q] = vmul(v[q], w);
                }
            }
            Radix<C2, R>::template run<1>(v);
        } else {
            Radix<C2, R>::template run<-1>(v);
            const RR o = fo ? fo[l] : (RR)0;
            RR h[R];
#pragma unroll
            for (int q = 0; q < R; ++q) h[q] = f[blk * R + q] + o;
            radix_scaled<C2, R, 1>(v, h);
        }
#pragma unroll
        for (int m = 0; m < R; ++m) p[m * st] = v[m];
    }
    __syncthreads();
}

template <class C2, class RR, int KIND>
__device__ __forceinline__ void tile_pass_any(int R, C2 *t, const TileLines &g, int L, int S, const C2 *tw, const RR *f,
                                              const RR *fo) {
    switch (R) {
        case 2: tile_pass<C2, RR, 2, KIND>(t, g, L, S, tw, f, fo); break;
        case 3: tile_pass<C2, RR, 3, KIND>(t, g, L, S, tw, f, fo); break;
        case 4: tile_pass<C2, RR, 4, KIND>(t, g, L, S, tw, f, fo); break;
        case 5: tile_pass<C2, RR, 5, KIND>(t, g, L, S, tw, f, fo); break;
        case 6: tile_pass<C2, RR, 6, KIND>(t, g, L, S, tw, f, fo); break;
        case 8: tile_pass<C2, RR, 8, KIND>(t, g, L, S, tw, f, fo); break;
        case 9: tile_pass<C2, RR, 9, KIND>(t, g, L, S, tw, f, fo); break;
        case 10: tile_pass<C2, RR, 10, KIND>(t, g, L, S, tw, f, fo); break;
        case 12: tile_pass<C2, RR, 12, KIND>(t, g, L, S, tw, f, fo); break;
        case 15: tile_pass<C2, RR, 15, KIND>(t, g, L, S, tw, f, fo); break;
        default: tile_pass<C2, RR, 16, KIND>(t, g, L, S, tw, f, fo); break;
    }
}

template <class R> __device__ __forceinline__ const typename Cx<R>::T *tile_tw(const AxisDev &ax);
template <> __device__ __forceinline__ const double2 *tile_tw<double>(const AxisDev &ax) { return ax.tw64; }
template <> __device__ __forceinline__ const float2 *tile_tw<float>(const AxisDev &ax) { return ax.tw32; }
template <class R> __device__ __forceinline__ const R *tile_filt(const AxisDev &ax, int energy);
template <> __device__ __forceinline__ const double *tile_filt<double>(const AxisDev &ax, int energy) {
    return energy ? ax.tefilt64 : ax.tfilt64;
}
template <> __device__ __forceinline__ const float *tile_filt<float>(const AxisDev &ax, int energy) {
    return energy ? ax.tefilt32 : ax.tfilt32;
}

// Global to shared without registers (8 or 16 bytes per thread).
template <class C2>
__device__ __forceinline__ void copy_async(C2 *s, const C2 *g) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(s)), "l"(g),
                 "n"((int)sizeof(C2))
                 : "memory");
}

template <class R>
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? 3 : 2) tile_filter_kernel(const LaunchTileFilter A) {
    using C2 = typename Cx<R>::T;
    extern __shared__ __align__(128) unsigned char smem[];
    const int bid = A.nfields == 2 ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
    const int field = A.nfields == 2 ? (int)(blockIdx.x & 1) : 0;
    const TileFilterTask task = A.tasks[bid];
    const TileFilterPlan &P = A.plans[task.plan];
    const ChainDev &ch = A.chains[task.chain];
    const int rows = task.rows, cols = task.cols, PZ = P.pitch, nax = P.naxes;
    const bool energy = A.filter != 0;
    C2 *tile = reinterpret_cast<C2 *>(smem);
    C2 *tw0 = tile + P.tile_elems;
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
    asm volatile("cp.async.commit_group;" ::: "memory");
    // tables of the filtered axes: twiddles, then the filters in the passes' order of
    // frequencies, the component constant folded into the first axis' one
    int nsum = 0;
    for (int a = 0; a < nax; ++a) nsum += ch.axis[P.axis[a]].n;
    R *f0 = reinterpret_cast<R *>(tw0 + nsum);
    {
        int o = 0;
        for (int a = 0; a < nax; ++a) {
            const AxisDev &ax = ch.axis[P.axis[a]];
            const C2 *tw = tile_tw<R>(ax);
            const R *f = tile_filt<R>(ax, energy);
            // energy: sum of the axes' k^2/2; each axis' table carries 1/n, and the sum over
            // axes of a slice's transforms needs the product of all 1/n on every term
            R cst = (a == 0 && P.with_const && !energy) ? (R)ch.comp_const[task.slice / ch.nt] : (R)1;
            if (energy)
                for (int b = 0; b < nax; ++b)
                    if (b != a) cst /= (R)ch.axis[P.axis[b]].n;
            for (int i = threadIdx.x; i < ax.n; i += blockDim.x) {
                tw0[o + i] = tw[i];
                f0[o + i] = f[i] * cst;
            }
            o += ax.n;
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // forward passes of one axis (all of them when `whole`), inverse passes
    auto forward = [&](const TileLines &g, const AxisDev &ax, const C2 *tw, bool whole) {
        int L = ax.n;
        for (int p = 0; p < (whole ? ax.tnf : ax.tnf - 1); ++p) {
            const int rad = ax.tfac[p];
            tile_pass_any<C2, R, TILE_DIF>(rad, tile, g, L, L / rad, tw, (const R *)nullptr, (const R *)nullptr);
            L /= rad;
        }
    };
    auto inverse = [&](const TileLines &g, const AxisDev &ax, const C2 *tw, bool whole) {
        int S = whole ? 1 : ax.tfac[ax.tnf - 1];
        for (int p = (whole ? ax.tnf : ax.tnf - 1) - 1; p >= 0; --p) {
            const int rad = ax.tfac[p];
            tile_pass_any<C2, R, TILE_DIT>(rad, tile, g, S * rad, S, tw, (const R *)nullptr, (const R *)nullptr);
            S *= rad;
        }
    };
    // I of axis a: the tile elements (padding aside) between two of its sites
    auto lines = [&](int a) {
        return TileLines(rows, cols, PZ, ch.axis[P.axis[a]].n, P.inner[a] == 0 ? cols : P.inner[a], P.inner[a] == 1);
    };
    auto middle = [&](const TileLines &g, const AxisDev &ax, const C2 *tw, const R *f, const R *fo) {
        const int rad = ax.tfac[ax.tnf - 1];
        tile_pass_any<C2, R, TILE_MID>(rad, tile, g, rad, 1, tw, f, fo);
    };
    if (!energy || nax == 1) {
        // product of the axes' filters: one axis after the other
        int o = 0;
        for (int a = 0; a < nax; ++a) {
            const AxisDev &ax = ch.axis[P.axis[a]];
            const TileLines g = lines(a);
            forward(g, ax, tw0 + o, false);
            middle(g, ax, tw0 + o, f0 + o, nullptr);
            inverse(g, ax, tw0 + o, false);
            o += ax.n;
        }
    } else {
        // sum of the axes' filters: every axis forward, the sum at each frequency, and back
        // (the last axis is the innermost: its lines are the tile's rows, whose share of the
        // other axes' filters goes into fo)
        R *fo = f0 + nsum;
        int o = 0;
        for (int a = 0; a + 1 < nax; ++a) {
            const AxisDev &ax = ch.axis[P.axis[a]];
            forward(lines(a), ax, tw0 + o, true);
            o += ax.n;
        }
        for (int r = threadIdx.x; r < rows; r += blockDim.x) {
            R v = 0;
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
            forward(g, ax, tw0 + o, false);
            middle(g, ax, tw0 + o, f0 + o, fo);
            inverse(g, ax, tw0 + o, false);
        }
        for (int a = nax - 2; a >= 0; --a) {
            const AxisDev &ax = ch.axis[P.axis[a]];
            o -= ax.n;
            inverse(lines(a), ax, tw0 + o, true);
        }
    }
    const bool acc = A.accumulate != 0;
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
        const int r = dc.div(e), c = e - r * cols;
        C2 *d = dst + (long long)r * gs + c;
        const C2 v = tile[r * PZ + c];
        *d = acc ? vadd(*d, v) : v;
    }
}

template <class R>
cudaError_t setup_tile_filter(size_t smem_bytes, int *ctas_per_sm) {
    const void *fn = (const void *)tile_filter_kernel<R>;
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, fn);
    if (e != cudaSuccess) return e;
    if ((int)smem_bytes > fa.maxDynamicSharedSizeBytes) {  // serves every shape: keep the largest request
        e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes);
        if (e != cudaSuccess) return e;
    }
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas_per_sm, fn, 256, smem_bytes);
}

template <class R>
cudaError_t launch_tile_filter(const LaunchTileFilter &L, cudaStream_t s) {
    if (L.ntasks == 0) return cudaSuccess;
    void *args[] = {const_cast<LaunchTileFilter *>(&L)};
    return cudaLaunchKernel((const void *)tile_filter_kernel<R>, dim3(L.nfields * L.ntasks), dim3(L.threads), args, L.smem_bytes, s);
}

}  // namespace clv
