// k_obs.cu -- observables accumulated on the device in FP64.
//
// Reference observables (Observables::evaluate, Observables_without_cutoff.cu:1155-1382):
//   F_x, F_y, F_z real-space profiles summed over tau (kernel
//   evaluate_spin_density_realspace, :456-488) and n_tot, n_11..n_22 (kernels
//   :35-101 evaluated on FFT'd fields and reduced with thrust).  The particle
//   numbers are computed in real space here: with the reference's transform
//   directions, sum_k psibar~(k) psi~(k) = V sum_x psibar(x) psi(x) (Parseval),
//   so no FFT and no host round trip is needed.  One thread sums a site over a chunk of
//   imaginary times (29 FP64 operations each; the products of two times are summed among
//   themselves and added to the running sum once: added one by one, each would be rounded at
//   that sum's size, 2 to 3 times the error), a second kernel adds the chunks in order.
//   Bound by the FP64 pipe on large lattices (4 components, 128^2 x 128: 405 -> 171 us), by
//   latency on small ones, where a thread per site left one CTA to walk through imaginary
//   time (256 x 32: 105 -> 17 us).
// Spin-1 observables: density, F_z, F^2 = Fz^2 + F+F- and energy
//   psibar (k^2/2 - q m^2) psi + c0/2 n^2 + c1/2 F^2, all with the point split
//   (psibar(tau+1), psi(tau)); one FP64 sample per evaluate call and chain,
//   reduced without atomics on the sums.
#include "clv_internal.cuh"
#include "clv_launch.h"

namespace clv {

__device__ __forceinline__ long long oidx(const ChainDev &ch, int c, int tau, int s) {
    return ch.off + ((long long)c * ch.nt + tau) * ch.V + s;
}

// The CTA's (chunk, site) pair of this thread and its imaginary times [tau0, tau1).
struct ObsRange {
    int s, tau0, tau1;
    bool act;
    __device__ __forceinline__ ObsRange(const ChainDev &ch, const ObsTask &task, int pair) {
        const int flat = task.flat0 + pair, k = flat / ch.V;
        s = flat - k * ch.V;
        act = k < ch.obs_nchunk;
        tau0 = (int)((long long)ch.nt * k / ch.obs_nchunk);
        tau1 = (int)((long long)ch.nt * (k + 1) / ch.obs_nchunk);
    }
};

// a += Re(x y), a += Im(x y) and a -= Im(x y)
__device__ __forceinline__ void add_re(double &a, double2 x, double2 y) { a = fma(x.x, y.x, fma(-x.y, y.y, a)); }
__device__ __forceinline__ void add_im(double &a, double2 x, double2 y) { a = fma(x.x, y.y, fma(x.y, y.x, a)); }
__device__ __forceinline__ void sub_im(double &a, double2 x, double2 y) { a = fma(-x.x, y.y, fma(-x.y, y.x, a)); }

// Sums of M values over a warp: every step halves the values a lane carries (8 values take 9
// FP64 additions a lane instead of 40).  Lanes that are multiples of 32 / M return value
// lane M / 32.
template <int M>
__device__ __forceinline__ double warp_sums(double (&v)[M]) {
    const int lane = threadIdx.x & 31;
    int o = 16;
#pragma unroll
    for (int n = M / 2; n >= 1; n /= 2, o /= 2) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const double send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
#pragma unroll
    for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    return v[0];
}

template <class R>
__global__ void __launch_bounds__(256)
obs_ref_kernel(const ChainDev *__restrict__ chains, const ObsTask *__restrict__ tasks,
               const typename Cx<R>::T *__restrict__ psi, const typename Cx<R>::T *__restrict__ psic,
               double *__restrict__ scratch, double *__restrict__ partials) {
    __shared__ double sh[8][4];
    const ObsTask task = tasks[blockIdx.x];
    const ChainDev &ch = chains[task.chain];
    const ObsRange o(ch, task, threadIdx.x);
    double n[4] = {0, 0, 0, 0}, fx = 0, fy = 0, fz = 0;
    if (o.act) {
        for (int tau = o.tau0; tau < o.tau1; tau += 2) {
            double x = 0, y = 0, d[4] = {0, 0, 0, 0};
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int t = tau + u, tp = t == ch.nt - 1 ? 0 : t + 1;
                if (t >= o.tau1) break;
                double2 pc[4], cp[4];
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    const auto v = psi[oidx(ch, a, t, o.s)];
                    const auto w = psic[oidx(ch, a, tp, o.s)];
                    pc[a] = make_double2(v.x, v.y);
                    cp[a] = make_double2(w.x, w.y);
                }
                add_re(x, cp[2], pc[0]); add_re(x, cp[0], pc[2]);
                add_re(x, cp[3], pc[1]); add_re(x, cp[1], pc[3]);
                // Re(i w) = -Im(w) of t20 - t02 + t31 - t13
                sub_im(y, cp[2], pc[0]); add_im(y, cp[0], pc[2]);
                sub_im(y, cp[3], pc[1]); add_im(y, cp[1], pc[3]);
#pragma unroll
                for (int a = 0; a < 4; ++a) add_re(d[a], cp[a], pc[a]);
            }
            fx += x;
            fy += y;
            fz += (d[0] + d[1]) - (d[2] + d[3]);
#pragma unroll
            for (int a = 0; a < 4; ++a) n[a] += d[a];
        }
        const long long nv = (long long)ch.obs_nchunk * ch.V;
        double *F = scratch + ch.obs_scr + task.flat0 + threadIdx.x;
        F[0] = fx;
        F[nv] = fy;
        F[2 * nv] = fz;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const double w = warp_sums<4>(n) * ch.a_x;
    if (lane % 8 == 0) sh[warp][lane / 8] = w;
    __syncthreads();
    if (threadIdx.x < 4) {
        double v = 0.0;
        for (int w = 0; w < 8; ++w) v += sh[w][threadIdx.x];
        partials[(size_t)blockIdx.x * 8 + threadIdx.x] = v;
    }
}

// Sum of value i < M of a chain's partials (8 doubles per CTA) over its CTAs: 256 / M threads
// per value, then those in order; result valid in threads i < M.
template <int M>
__device__ __forceinline__ double sum_partials(const ChainDev &ch, const double *partials) {
    constexpr int G = 256 / M;
    __shared__ double sh[G][M];
    const int i = threadIdx.x % M, g = threadIdx.x / M;
    double v = 0.0;
    for (int b = g; b < ch.obs_nblocks; b += G) v += __ldcg(&partials[(size_t)(ch.obs_block0 + b) * 8 + i]);
    sh[g][i] = v;
    __syncthreads();
    v = 0.0;
    if (threadIdx.x < M)
        for (int k = 0; k < G; ++k) v += sh[k][threadIdx.x];
    return v;
}

// Adds the chunks of 32 sites to the profiles and, in the chain's first CTA, the CTAs'
// particle numbers to the accumulators.  A warp takes every eighth chunk, and the warps' sums
// are added in order (a thread per site summing all chunks: 11 chains of 64 sites and up to
// 100 imaginary times: an evaluation 82 us, so 21; one of 256 x 32 32 and 16).
__global__ void __launch_bounds__(256)
obs_ref_finish_kernel(const ChainDev *__restrict__ chains, const SiteTask *__restrict__ sites,
                      const double *__restrict__ scratch, const double *__restrict__ partials,
                      double *__restrict__ accF, double *__restrict__ accN) {
    const SiteTask task = sites[blockIdx.x >> 3];
    const ChainDev &ch = chains[task.chain];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, site0 = task.site0 + 32 * (int)(blockIdx.x & 7);
    const int s = site0 + lane, V = ch.V, nc = ch.obs_nchunk;
    if (site0 >= V) return;
    __shared__ double sh[8][3][32];
    double v[3] = {0.0, 0.0, 0.0};
    if (s < V) {
        const double *F = scratch + ch.obs_scr + s;
#pragma unroll 4
        for (int c = warp; c < nc; c += 8)
#pragma unroll
            for (int k = 0; k < 3; ++k) v[k] += __ldcg(&F[((long long)k * nc + c) * V]);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) sh[warp][k][lane] = v[k];
    __syncthreads();
    if (warp < 3 && s < V) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < 8; ++w) t += sh[w][warp][lane];
        accF[ch.obs_off + warp * V + s] += t;
    }
    if (site0 == 0) {
        const double n = sum_partials<4>(ch, partials);
        // the threads of a warp's first four lanes hold n_11 .. n_22
        double t = n;
        t += __shfl_xor_sync(0xffffffffu, t, 1);
        t += __shfl_xor_sync(0xffffffffu, t, 2);
        if (threadIdx.x < 4) accN[task.chain * 5 + 1 + threadIdx.x] += n * (double)V;
        if (threadIdx.x == 0) accN[task.chain * 5] += t * (double)V;
    }
}

template <class R>
cudaError_t launch_obs_ref(const LaunchObs &L, cudaStream_t s) {
    using C2 = typename Cx<R>::T;
    obs_ref_kernel<R><<<L.ntasks, 256, 0, s>>>(L.chains, L.tasks, (const C2 *)L.psi, (const C2 *)L.psic, L.scratch,
                                               L.partials);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    obs_ref_finish_kernel<<<8 * L.nsites, 256, 0, s>>>(L.chains, L.sites, L.scratch, L.partials, L.accF, L.accN);
    return cudaGetLastError();
}

// A CTA takes 256 (chunk, site) pairs of one chain, chunks of at most 16 imaginary times
// (ObsTask); tpsi = (k^2/2) psi from the kinetic-energy filter.  Per-site
// products in the working precision R, summed per thread over the CTA's tau
// range, then in FP64 across the CTA (one partial of the 8 sums per CTA); the
// chain's last CTA adds its partials (no atomics on the sums, the same result for every
// run) and writes the sample.
// GROUP (FP32, few pairs): 16 pairs by 16 threads, one imaginary time each; a thread then adds
// a pair's values in the order and precision of the streaming form, whose sums it repeats bit
// for bit (two chains of 256 x 32: an evaluation 28 us streaming 16 imaginary times, 17 so; the
// streaming form is the faster one from 0.3 M sites on).
template <class R, bool GROUP>
__global__ void __launch_bounds__(256)
obs_spin1_kernel(const ChainDev *__restrict__ chains, const ObsTask *__restrict__ tasks,
                 const typename Cx<R>::T *__restrict__ psi, const typename Cx<R>::T *__restrict__ psic,
                 const typename Cx<R>::T *__restrict__ tpsi, double *__restrict__ partials,
                 unsigned int *__restrict__ arrive, double *__restrict__ samples, int slot, int nchains) {
    using C2 = typename Cx<R>::T;
    __shared__ double sh[8][8];
    __shared__ int am_last;
    const ObsTask task = tasks[blockIdx.x];
    const ChainDev &ch = chains[task.chain];
    const ObsRange o(ch, task, GROUP ? threadIdx.x & 15 : threadIdx.x);
    const int s = o.s, mine = o.tau0 + (int)(threadIdx.x >> 4);
    const int from = GROUP ? mine : o.tau0, to = GROUP ? min(mine + 1, o.tau1) : o.tau1;
    R acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (o.act) {
        const R r2 = (R)1.41421356237309504880, q = (R)ch.q, c0h = (R)(0.5 * ch.c0),
                c1h = (R)(0.5 * ch.c1);
        for (int tau = from; tau < to; ++tau) {
            const int tp = tau == ch.nt - 1 ? 0 : tau + 1;
            C2 bar[3], ket[3], tk[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                bar[a] = psic[oidx(ch, a, tp, s)];
                ket[a] = psi[oidx(ch, a, tau, s)];
                tk[a] = tpsi[oidx(ch, a, tau, s)];
            }
            const C2 n = cadd(cadd(cmul(bar[0], ket[0]), cmul(bar[1], ket[1])), cmul(bar[2], ket[2]));
            const C2 Fz = csub(cmul(bar[0], ket[0]), cmul(bar[2], ket[2]));
            const C2 Fp = cscale(r2, cadd(cmul(bar[0], ket[1]), cmul(bar[1], ket[2])));
            const C2 Fm = cscale(r2, cadd(cmul(bar[1], ket[0]), cmul(bar[2], ket[1])));
            const C2 F2 = cadd(cmul(Fz, Fz), cmul(Fp, Fm));
            C2 e1 = cmul(bar[1], tk[1]);  // m = 0
            e1 = cadd(e1, cmul(bar[0], csub(tk[0], cscale(q, ket[0]))));
            e1 = cadd(e1, cmul(bar[2], csub(tk[2], cscale(q, ket[2]))));
            const C2 e = cadd(cadd(e1, cscale(c0h, cmul(n, n))), cscale(c1h, F2));
            acc[0] += n.x; acc[1] += n.y; acc[2] += Fz.x; acc[3] += Fz.y;
            acc[4] += F2.x; acc[5] += F2.y; acc[6] += e.x; acc[7] += e.y;
        }
    }
    if constexpr (GROUP) {
        __shared__ R val[8][16][16];
#pragma unroll
        for (int i = 0; i < 8; ++i) val[i][threadIdx.x >> 4][threadIdx.x & 15] = acc[i];
        __syncthreads();
        const int i = threadIdx.x >> 4, p = threadIdx.x & 15;
        if (i < 8) {
            R t = 0;
            if (o.act)
                for (int j = 0; j < o.tau1 - o.tau0; ++j) t += val[i][j][p];
            double v = (double)t;
#pragma unroll
            for (int b = 8; b > 0; b >>= 1) v += __shfl_xor_sync(0xffffffffu, v, b);
            if (p == 0) partials[(size_t)blockIdx.x * 8 + i] = v;
        }
    } else {
        // FP64 above the thread: warp shuffles, then the CTA's 8 warps in order
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        double part[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) part[i] = (double)acc[i];
        const double sum = warp_sums<8>(part);
        if (lane % 4 == 0) sh[warp][lane / 4] = sum;
        __syncthreads();
        if (threadIdx.x < 8) {
            double v = 0.0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v += sh[w][threadIdx.x];
            partials[(size_t)blockIdx.x * 8 + threadIdx.x] = v;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        am_last = atomicAdd(&arrive[task.chain], 1u) == (unsigned)ch.obs_nblocks - 1;
    }
    __syncthreads();
    if (!am_last) return;
    __threadfence();
    const double v = sum_partials<8>(ch, partials);
    if (threadIdx.x < 8)
        samples[((size_t)slot * nchains + task.chain) * 8 + threadIdx.x] = v / ((double)ch.V * ch.nt);
    if (threadIdx.x == 0) arrive[task.chain] = 0u;
}

template <class R>
cudaError_t launch_obs_spin1(const LaunchObs &L, cudaStream_t s) {
    using C2 = typename Cx<R>::T;
    if (L.ntasks == 0) return cudaSuccess;
    auto run = [&](auto kern) {
        kern<<<L.ntasks, 256, 0, s>>>(L.chains, L.tasks, (const C2 *)L.psi, (const C2 *)L.psic, (const C2 *)L.tpsi,
                                      L.partials, L.arrive, L.samples, L.slot, L.nchains);
    };
    if (sizeof(R) == 4 && L.group) run(obs_spin1_kernel<R, sizeof(R) == 4>);
    else run(obs_spin1_kernel<R, false>);
    return cudaGetLastError();
}

template cudaError_t launch_obs_ref<double>(const LaunchObs &, cudaStream_t);
template cudaError_t launch_obs_ref<float>(const LaunchObs &, cudaStream_t);
template cudaError_t launch_obs_spin1<double>(const LaunchObs &, cudaStream_t);
template cudaError_t launch_obs_spin1<float>(const LaunchObs &, cudaStream_t);

}  // namespace clv
