// k_plane.cu -- kinetic filter of a whole square plane (both of its axes) in one
// pass over HBM, for the tiled path's 2D slices (n x n) and the (y, z) planes of
// 3D slices (n x n at each x), n = 32, 64, 96 or 128.
//
// The spin-1 kinetic factor exp(-eps k^2/2) is a product over the axes, so the
// plane's filter is the line filter along one axis followed by the line filter
// along the other (the same operator as two axis_filter_kernel launches,
// Propagator_without_cutoff.cu:410-424 for the reference's transform sequence).
// One CTA (plane_threads(n, esz) threads) holds one plane of one (component, tau)
// slice of one field in shared memory (n rows at an odd pitch n + 1) and filters
// its lines in place (inplace_fft.cuh: decimation in frequency, the filter at the
// digit-reversed frequencies, decimation in time; one block barrier per pass).
// The first pass (along the slower axis, whose lines are columns) reads its
// butterflies straight from global memory, 32 consecutive columns a warp; the
// plane is written back from shared memory in row order.  FP32 planes of 64 take
// one thread per line instead, the line in registers (plane_lines_in_registers), FP32
// planes of 128 2D blocks of it (plane_blocks_128).
// The plane is read once and written once: half the traffic of the two axis
// launches it replaces.
#include "clv_internal.cuh"
#include "clv_launch.h"
#include "fused_impl.cuh"
#include "inplace_fft.cuh"

namespace clv {

// Butterflies whose global loads the first pass issues together: all of a thread's
// where one CTA fills the SM (FP32 planes of 128, FP64 planes of 96), else one (the
// other resident CTAs keep loads in flight).
__host__ __device__ constexpr int plane_first_group(int n, int esz) {
    return (n == 128 && esz == 8) || (n == 96 && esz == 16) ? n * (n / plane_fac(n, 0)) / plane_threads(n, esz) : 1;
}

// Butterflies of a pass unrolled together: all of a thread's (at most 8) for the FP64
// planes of 96 (one CTA per SM), else one at a time, streamed (several resident CTAs).
__host__ __device__ constexpr int plane_unroll(int n, int esz) { return n == 96 && esz == 16 ? 8 : 1; }

// Two-radix line plans of the plane (clv_launch.h plane_fac).
struct PlanePlan {
    static __host__ __device__ constexpr int nfac(int n) { return plane_nfac(n); }
    static __host__ __device__ constexpr int fac(int n, int p) { return plane_fac(n, p); }
};

// Resident CTAs per SM the registers are budgeted for (shared memory allows as many).
__host__ __device__ constexpr int plane_min_ctas(int n, int esz) {
    return esz == 8 ? (n == 32 ? 8 : (n == 64 ? 6 : (n == 96 ? 3 : 1))) : (n == 32 ? 4 : (n == 64 ? 3 : 1));
}

// The filter's planes in blocks (plane_blocks): its threads and CTAs per SM.
__host__ __device__ constexpr bool plane_in_blocks(int n, int esz) { return esz == 8 && (n == 96 || n == 128); }
__host__ __device__ constexpr int filter_threads(int n, int esz) {
    return plane_in_blocks(n, esz) && n == 96 ? 192 : plane_threads(n, esz);
}
__host__ __device__ constexpr int filter_min_ctas(int n, int esz) {
    return plane_in_blocks(n, esz) && n == 96 ? 2 : plane_min_ctas(n, esz);
}

// One thread per line with the whole line in registers (FP32 planes of 64): thread l
// loads column l straight from global memory (a warp: 32 consecutive columns), runs the
// 64-point transform, the filter and the inverse in registers and writes the column into
// the tile; after a barrier it does the same for row l, and the plane goes back in row
// order: 4 shared-memory accesses per element instead of the 12 of the in-place passes.
template <class R, int N>
__device__ __forceinline__ void plane_lines_in_registers(const LaunchAxis &A) {
    using C2 = typename Cx<R>::T;
    constexpr int PL = plane_pitch(N);
    extern __shared__ __align__(128) unsigned char smem[];
    const AxisTask task = A.tasks[blockIdx.x >> 1];
    const int field = (int)(blockIdx.x & 1);
    const ChainDev &ch = A.chains[task.chain];
    const AxisDev &axr = ch.axis[A.axis], &axc = ch.axis[A.axis + 1];
    R *fr = reinterpret_cast<R *>(smem + N * sizeof(C2));
    R *fc = fr + N;
    C2 *tile = reinterpret_cast<C2 *>(smem + plane_tab_bytes(N, sizeof(C2)));
    const long long soff = ch.off + (long long)task.slice * ch.V + (long long)task.l0 * (N * N);
    const C2 *src = reinterpret_cast<const C2 *>(field ? A.src1 : A.src0) + soff;
    C2 *dst = reinterpret_cast<C2 *>(field ? A.dst1 : A.dst0) + soff;
    const int l = threadIdx.x;
    const R cst = A.with_const ? (R)ch.comp_const[task.slice / ch.nt] : (R)1;
    // phase 0 along column l (the slower axis), phase 1 along row l (the contiguous axis):
    // one copy of the transforms' code for both (the unrolled transforms are large)
#pragma unroll 1
    for (int ph = 0; ph < 2; ++ph) {
        C2 v[N];
        if (ph == 0) {
#pragma unroll
            for (int a = 0; a < N; ++a) v[a] = src[a * N + l];
            fr[l] = filt_of<R>(axr)[l];
            fc[l] = filt_of<R>(axc)[l] * cst;
            __syncthreads();
        } else {
#pragma unroll
            for (int a = 0; a < N; ++a) v[a] = tile[l * PL + a];
        }
        Radix<C2, N>::template run<-1>(v);
        const R *f = ph ? fc : fr;
#pragma unroll
        for (int k = 0; k < N; ++k) v[k] = vscale(f[k], v[k]);
        Radix<C2, N>::template run<1>(v);
        const int s0 = ph ? l * PL : l, sa = ph ? 1 : PL;  // element a of the line in the tile
#pragma unroll
        for (int a = 0; a < N; ++a) tile[s0 + a * sa] = v[a];
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < N; ++i) dst[i * N + l] = tile[i * PL + l];
}

// FP32 planes of 96 and 128: few CTAs fill an SM's shared memory, so every access to the tile
// counts.  2D blocks in registers: columns 8 x CB, rows RA x RB, with the columns' last inverse
// pass (8 rows) and the rows' first forward pass (RA columns) done on one 8 x RA block, the
// first pass read from and the last written to global memory: 8 shared accesses an element and
// four barriers instead of the in-place passes' 12 and six.  In the blocks a thread's
// twiddles serve all its rows or columns.
//   A  columns forward, radix 8:  rows k + CB m of column c                  -> tile
//   B  columns middle, radix CB:  rows CB j + m                              tile
//   C  columns inverse, radix 8 and rows forward, radix RA: rows k + CB m, columns l + RB n  tile
//   D  rows middle, radix RB:     columns RB q + i of row r                  tile
//   E  rows inverse, radix RA:    columns l + RB n of 8 rows                 -> global
// 768 planes of 128 (one chain, 3 components x 128 slices x 2 fields): 97 us in place -> 79
// us (floor 30); 3840 planes of 96: 463 -> 422 us (floor 250).  Blocks of 128 (512 threads, one
// CTA) prefetch the plane that follows on the SM into L2 (940 -> 902 us for 3840 planes); of 96
// (192 threads, two CTAs that overlap) do not (422 -> 447 us).
template <int N>
struct PlaneBlocks {
    static constexpr int CB = N / 8, RA = N == 128 ? 4 : 6, RB = N / RA, T = CB * RB, G = T / N, RPT = T / RB;
    static constexpr int NA = CB / G, NB = 8 / G, ND = RA / G, NE = N / RPT;
};

template <int N>
__device__ __forceinline__ void plane_blocks(const LaunchAxis &A) {
    using C2 = float2;
    using P = PlaneBlocks<N>;
    constexpr int PL = plane_pitch(N), CB = P::CB, RA = P::RA, RB = P::RB, G = P::G;
    extern __shared__ __align__(128) unsigned char smem[];
    C2 *tw = reinterpret_cast<C2 *>(smem);
    float *fr = reinterpret_cast<float *>(smem + N * sizeof(C2));
    float *fc = fr + N;
    C2 *tile = reinterpret_cast<C2 *>(smem + plane_tab_bytes(N, sizeof(C2)));
    const int c = threadIdx.x % N, g = threadIdx.x / N, l = threadIdx.x % RB, w = threadIdx.x / RB;
    C2 v[P::NA][8];
    C2 *dst;
    auto load = [&](int t) {
        const AxisTask task = A.tasks[t >> 1];
        const ChainDev &ch = A.chains[task.chain];
        const long long off = ch.off + (long long)task.slice * ch.V + (long long)task.l0 * (N * N);
        const C2 *src = reinterpret_cast<const C2 *>(t & 1 ? A.src1 : A.src0) + off + c;
#pragma unroll
        for (int i = 0; i < P::NA; ++i)
#pragma unroll
            for (int m = 0; m < 8; ++m) v[i][m] = src[(g + G * i + CB * m) * N];
    };
    const int t = blockIdx.x;
    load(t);
    if (threadIdx.x < N) tw[c] = A.chains[A.tasks[t >> 1].chain].axis[A.axis + 1].tw32[c];
    __syncthreads();
    {
        const AxisTask task = A.tasks[t >> 1];
        const ChainDev &ch = A.chains[task.chain];
        dst = reinterpret_cast<C2 *>(t & 1 ? A.dst1 : A.dst0) + ch.off + (long long)task.slice * ch.V +
              (long long)task.l0 * (N * N);
        if (threadIdx.x < N) {
            fr[c] = ch.axis[A.axis].filt32[c];
            fc[c] = ch.axis[A.axis + 1].filt32[c] * (A.with_const ? (float)ch.comp_const[task.slice / ch.nt] : 1.0f);
        }
    }
#pragma unroll
    for (int i = 0; i < P::NA; ++i) {
        const int k = g + G * i;
        Radix<C2, 8>::run<-1>(v[i]);
        tile[k * PL + c] = v[i][0];
#pragma unroll
        for (int q = 1; q < 8; ++q) tile[(k + CB * q) * PL + c] = vmul(v[i][q], tw[q * k]);
    }
    // the plane that follows on this SM, into L2
    if (const int tn = t + A.resident; N == 128 && tn < 2 * A.ntasks) {
        const AxisTask task = A.tasks[tn >> 1];
        const ChainDev &ch = A.chains[task.chain];
        const long long off = ch.off + (long long)task.slice * ch.V + (long long)task.l0 * (N * N);
        const C2 *src = reinterpret_cast<const C2 *>(tn & 1 ? A.src1 : A.src0) + off;
        for (int i = threadIdx.x * 16; i < N * N; i += P::T * 16) asm volatile("prefetch.global.L2 [%0];" ::"l"(src + i));
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < P::NB; ++i) {
        const int j = g + G * i;
        C2 *x = tile + j * CB * PL + c;
        C2 u[CB];
#pragma unroll
        for (int m = 0; m < CB; ++m) u[m] = x[m * PL];
        Radix<C2, CB>::template run<-1>(u);
#pragma unroll
        for (int q = 0; q < CB; ++q) u[q] = vscale(fr[j + 8 * q], u[q]);
        Radix<C2, CB>::template run<1>(u);
#pragma unroll
        for (int m = 0; m < CB; ++m) x[m * PL] = u[m];
    }
    __syncthreads();
    {
        C2 *x = tile + w * PL + l;
        C2 b[RA][8];
#pragma unroll
        for (int m = 0; m < 8; ++m)
#pragma unroll
            for (int n = 0; n < RA; ++n) b[n][m] = x[CB * m * PL + RB * n];
#pragma unroll
        for (int m = 1; m < 8; ++m) {
            const C2 z = tw[m * w];
#pragma unroll
            for (int n = 0; n < RA; ++n) b[n][m] = vmulc(b[n][m], z);
        }
#pragma unroll
        for (int n = 0; n < RA; ++n) Radix<C2, 8>::run<1>(b[n]);
        C2 z[RA];
#pragma unroll
        for (int n = 1; n < RA; ++n) z[n] = tw[n * l];
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            C2 u[RA];
#pragma unroll
            for (int n = 0; n < RA; ++n) u[n] = b[n][m];
            Radix<C2, RA>::template run<-1>(u);
            C2 *o = x + CB * m * PL;
            o[0] = u[0];
#pragma unroll
            for (int n = 1; n < RA; ++n) o[RB * n] = vmul(u[n], z[n]);
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < P::ND; ++i) {
        const int q = g + G * i;
        C2 *x = tile + c * PL + RB * q;  // row c
        C2 u[RB];
#pragma unroll
        for (int m = 0; m < RB; ++m) u[m] = x[m];
        Radix<C2, RB>::template run<-1>(u);
#pragma unroll
        for (int m = 0; m < RB; ++m) u[m] = vscale(fc[q + RA * m], u[m]);
        Radix<C2, RB>::template run<1>(u);
#pragma unroll
        for (int m = 0; m < RB; ++m) x[m] = u[m];
    }
    __syncthreads();
    C2 z[RA];
#pragma unroll
    for (int n = 1; n < RA; ++n) z[n] = tw[n * l];
#pragma unroll
    for (int i = 0; i < P::NE; ++i) {
        const int r = w + P::RPT * i;
        const C2 *x = tile + r * PL + l;
        C2 u[RA];
        u[0] = x[0];
#pragma unroll
        for (int n = 1; n < RA; ++n) u[n] = vmulc(x[RB * n], z[n]);
        Radix<C2, RA>::template run<1>(u);
        C2 *o = dst + r * N + l;
#pragma unroll
        for (int n = 0; n < RA; ++n) o[RB * n] = u[n];
    }
}

// In-place passes over the plane in shared memory (inplace_fft.cuh).
template <class R, int N>
__device__ __forceinline__ void plane_in_place(const LaunchAxis &A) {
    using C2 = typename Cx<R>::T;
    constexpr int T = plane_threads(N, (int)sizeof(C2)), PL = plane_pitch(N), EPT = N * N / T, R0 = plane_fac(N, 0);
    constexpr int PER0 = N * (N / R0) / T, G = plane_first_group(N, (int)sizeof(C2));
    using IP = InPlace<PlanePlan, N, N, T, plane_unroll(N, (int)sizeof(C2))>;
    extern __shared__ __align__(128) unsigned char smem[];
    const AxisTask task = A.tasks[blockIdx.x >> 1];
    const int field = (int)(blockIdx.x & 1);
    const ChainDev &ch = A.chains[task.chain];
    const AxisDev &axr = ch.axis[A.axis], &axc = ch.axis[A.axis + 1];
    C2 *twS = reinterpret_cast<C2 *>(smem);
    R *fr = reinterpret_cast<R *>(smem + N * sizeof(C2));
    R *fc = fr + N;
    C2 *tile = reinterpret_cast<C2 *>(smem + plane_tab_bytes(N, sizeof(C2)));
    const long long soff = ch.off + (long long)task.slice * ch.V + (long long)task.l0 * (N * N);
    const C2 *src = reinterpret_cast<const C2 *>(field ? A.src1 : A.src0) + soff;
    C2 *dst = reinterpret_cast<C2 *>(field ? A.dst1 : A.dst0) + soff;
    const C2 *tw = tw_of<R>(axc);  // both axes have n sites: one twiddle table
    // first forward pass along the columns, straight from global memory (twiddles from
    // the global table); the shared tables are filled meanwhile
#pragma unroll 1
    for (int p0 = 0; p0 < PER0; p0 += G) {
        C2 v[G][R0];
        IP::template first_load<C2, G>(v, src, 1, N, p0);
        IP::template first_finish<C2, G>(v, tile, 1, PL, tw, p0);
    }
    {
        const R *f0 = filt_of<R>(axr), *f1 = filt_of<R>(axc);
        const R cst = A.with_const ? (R)ch.comp_const[task.slice / ch.nt] : (R)1;
        for (int i = threadIdx.x; i < N; i += T) {
            twS[i] = tw[i];
            fr[i] = f0[i];
            fc[i] = f1[i] * cst;
        }
    }
    __syncthreads();
    IP::template filter<C2, R, 1>(tile, 1, PL, twS, fr);  // along the columns (the slower axis)
    IP::template filter<C2, R, 0>(tile, PL, 1, twS, fc);  // along the rows (contiguous axis)
#pragma unroll
    for (int i = 0; i < EPT; ++i) {
        const int e = threadIdx.x + i * T;
        dst[threadIdx.x + i * T] = tile[(e / N) * PL + e % N];
    }
}

// Kinetic energy of the planes: (k_r^2 + k_c^2) / 2, a sum over the axes, so both axes go
// forward, the sum multiplies at every frequency pair, and both come back.  One field
// (A.src0 -> A.dst0, added to it when A.accumulate): the planes of a 3D slice follow its x
// axis.  An evaluation of 64^3 x 64, FP32, three axis launches and the sums: 1.70 -> 0.58 ms;
// of 128^2 x 128: 161 -> 87 us.
__device__ __forceinline__ const float *plane_efilt(const AxisDev &ax, float) { return ax.efilt32; }
__device__ __forceinline__ const double *plane_efilt(const AxisDev &ax, double) { return ax.efilt64; }

// FP32 planes of 64, a line per thread: columns forward, rows forward, multiplied and back,
// columns back.
template <class R, int N>
__device__ __forceinline__ void plane_energy_in_registers(const LaunchAxis &A) {
    using C2 = typename Cx<R>::T;
    constexpr int PL = plane_pitch(N);
    extern __shared__ __align__(128) unsigned char smem[];
    const AxisTask task = A.tasks[blockIdx.x];
    const ChainDev &ch = A.chains[task.chain];
    const AxisDev &axr = ch.axis[A.axis], &axc = ch.axis[A.axis + 1];
    R *fr = reinterpret_cast<R *>(smem + N * sizeof(C2));
    R *fc = fr + N;
    C2 *tile = reinterpret_cast<C2 *>(smem + plane_tab_bytes(N, sizeof(C2)));
    const long long soff = ch.off + (long long)task.slice * ch.V + (long long)task.l0 * (N * N);
    const C2 *src = reinterpret_cast<const C2 *>(A.src0) + soff;
    C2 *dst = reinterpret_cast<C2 *>(A.dst0) + soff;
    const int l = threadIdx.x;
    fr[l] = plane_efilt(axr, R(0))[l] / N;
    fc[l] = plane_efilt(axc, R(0))[l] / N;
    C2 v[N];
#pragma unroll
    for (int a = 0; a < N; ++a) v[a] = src[a * N + l];
    // phases 0 and 1 forward along columns and rows, 1 and 2 backward along rows and columns:
    // one copy of each transform's code
#pragma unroll 1
    for (int ph = 0; ph < 3; ++ph) {
        if (ph < 2) Radix<C2, N>::template run<-1>(v);
        if (ph == 1) {
            const R o = fr[l];
#pragma unroll
            for (int k = 0; k < N; ++k) v[k] = vscale(fc[k] + o, v[k]);
        }
        if (ph > 0) Radix<C2, N>::template run<1>(v);
        if (ph == 2) break;
        const int s0 = ph ? l * PL : l, sa = ph ? 1 : PL;
#pragma unroll
        for (int a = 0; a < N; ++a) tile[s0 + a * sa] = v[a];
        __syncthreads();
        const int t0 = ph ? l : l * PL, ta = ph ? PL : 1;
#pragma unroll
        for (int a = 0; a < N; ++a) v[a] = tile[t0 + a * ta];
    }
    if (A.accumulate) {
#pragma unroll
        for (int a = 0; a < N; ++a) dst[a * N + l] = cadd(dst[a * N + l], v[a]);
    } else {
#pragma unroll
        for (int a = 0; a < N; ++a) dst[a * N + l] = v[a];
    }
}

template <class R, int N>
__device__ __forceinline__ void plane_energy_in_place(const LaunchAxis &A) {
    using C2 = typename Cx<R>::T;
    constexpr int T = plane_threads(N, (int)sizeof(C2)), PL = plane_pitch(N), EPT = N * N / T, R0 = plane_fac(N, 0);
    constexpr int PER0 = N * (N / R0) / T, G = plane_first_group(N, (int)sizeof(C2));
    using IP = InPlace<PlanePlan, N, N, T, plane_unroll(N, (int)sizeof(C2))>;
    extern __shared__ __align__(128) unsigned char smem[];
    const AxisTask task = A.tasks[blockIdx.x];
    const ChainDev &ch = A.chains[task.chain];
    const AxisDev &axr = ch.axis[A.axis], &axc = ch.axis[A.axis + 1];
    C2 *twS = reinterpret_cast<C2 *>(smem);
    R *fr = reinterpret_cast<R *>(smem + N * sizeof(C2));
    R *fc = fr + N;
    C2 *tile = reinterpret_cast<C2 *>(smem + plane_tab_bytes(N, sizeof(C2)));
    const long long soff = ch.off + (long long)task.slice * ch.V + (long long)task.l0 * (N * N);
    const C2 *src = reinterpret_cast<const C2 *>(A.src0) + soff;
    C2 *dst = reinterpret_cast<C2 *>(A.dst0) + soff;
    const C2 *tw = tw_of<R>(axc);
#pragma unroll 1
    for (int p0 = 0; p0 < PER0; p0 += G) {
        C2 v[G][R0];
        IP::template first_load<C2, G>(v, src, 1, N, p0);
        IP::template first_finish<C2, G>(v, tile, 1, PL, tw, p0);
    }
    for (int i = threadIdx.x; i < N; i += T) {
        twS[i] = tw[i];
        fr[i] = plane_efilt(axr, R(0))[IP::freq(i)] / N;  // row i holds the columns' frequency freq(i)
        fc[i] = plane_efilt(axc, R(0))[i] / N;
    }
    __syncthreads();
    IP::template forward<C2, 1>(tile, 1, PL, twS);
    IP::template fwd<C2, 0>(tile, PL, 1, twS);
    IP::template mid<C2, R, true>(tile, PL, 1, fc, fr);
    __syncthreads();
    IP::template inv<C2, IP::NF - 2>(tile, PL, 1, twS);
    IP::template backward<C2>(tile, 1, PL, twS);
    const bool acc = A.accumulate != 0;
#pragma unroll
    for (int i = 0; i < EPT; ++i) {
        const int e = threadIdx.x + i * T;
        const C2 v = tile[(e / N) * PL + e % N];
        dst[e] = acc ? cadd(dst[e], v) : v;
    }
}

template <class R, int N>
__global__ void __launch_bounds__(plane_threads(N, (int)sizeof(R) * 2), plane_min_ctas(N, (int)sizeof(R) * 2))
plane_energy_kernel(const LaunchAxis A) {
    if constexpr (plane_line_per_thread(N, (int)sizeof(R) * 2)) plane_energy_in_registers<R, N>(A);
    else plane_energy_in_place<R, N>(A);
}

// Task: AxisTask {chain, slice = c * nt + tau, l0 = plane index within the slice
// (the x index of a 3D slice, 0 for 2D)}; blockIdx.x % 2 selects the field.
// Axes A.axis (rows, the slower one) and A.axis + 1 (columns, contiguous).
template <class R, int N>
__global__ void __launch_bounds__(filter_threads(N, (int)sizeof(R) * 2), filter_min_ctas(N, (int)sizeof(R) * 2))
plane_filter_kernel(const LaunchAxis A) {
    if constexpr (plane_line_per_thread(N, (int)sizeof(R) * 2)) plane_lines_in_registers<R, N>(A);
    else if constexpr (plane_in_blocks(N, (int)sizeof(R) * 2)) plane_blocks<N>(A);
    else plane_in_place<R, N>(A);
}

// FP64 planes of 128 need 264 KB of shared memory: the engine never selects them.
template <class R, int N>
static const void *plane_kernel_of(int energy) {
    return energy ? (const void *)plane_energy_kernel<R, N> : (const void *)plane_filter_kernel<R, N>;
}
template <class R>
static const void *plane_kernel_ptr(int n, int energy) {
    if (n == 32) return plane_kernel_of<R, 32>(energy);
    if (n == 64) return plane_kernel_of<R, 64>(energy);
    if (n == 96) return plane_kernel_of<R, 96>(energy);
    if constexpr (sizeof(R) == 4) {
        if (n == 128) return plane_kernel_of<R, 128>(energy);
    }
    return nullptr;
}

template <class R>
cudaError_t setup_plane_filter(int n, int energy, size_t smem_bytes, int *ctas_per_sm) {
    const void *fn = plane_kernel_ptr<R>(n, energy);
    if (!fn) return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes);
    if (e != cudaSuccess) return e;
    const int esz = (int)sizeof(R) * 2;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas_per_sm, fn, energy ? plane_threads(n, esz) : filter_threads(n, esz),
                                                         smem_bytes);
}

template <class R>
cudaError_t launch_plane_filter(const LaunchAxis &L, cudaStream_t s) {
    if (L.ntasks == 0) return cudaSuccess;
    const void *fn = plane_kernel_ptr<R>(L.n, L.filter);
    if (!fn) return cudaErrorInvalidValue;
    void *args[] = {(void *)&L};
    const int esz = (int)sizeof(R) * 2, blocks = L.nfields * L.ntasks;
    if (L.filter || !plane_in_blocks(L.n, esz))
        return cudaLaunchKernel(fn, dim3(blocks), dim3(plane_threads(L.n, esz)), args, L.smem_bytes, s);
    return cudaLaunchKernel(fn, dim3(blocks), dim3(filter_threads(L.n, esz)), args, L.smem_bytes, s);
}

template cudaError_t setup_plane_filter<float>(int, int, size_t, int *);
template cudaError_t setup_plane_filter<double>(int, int, size_t, int *);
template cudaError_t launch_plane_filter<float>(const LaunchAxis &, cudaStream_t);
template cudaError_t launch_plane_filter<double>(const LaunchAxis &, cudaStream_t);

}  // namespace clv
