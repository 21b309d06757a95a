// k_tiled.cu -- the Langevin step of every lattice that the fused kernel does not
// take, after the kinetic terms have been filtered along every axis
// (k_axis.cu writes kin = e^{-eps H_kin} psi and kinbar for all imaginary times).
//
// A thread owns one spatial site of one chain over a chunk of imaginary times
// [tau0, tau1) and streams through it; a CTA takes 256 consecutive (chunk, site) pairs.  psi(tau-1), psi(tau)
// and psibar(tau) are carried in registers from the previous tau;
// each iteration loads psi(tau+1), psibar(tau+1), kin(tau-1) and kinbar(tau+1),
// prefetched one tau ahead, so every array is read once per step (plus one halo
// slice per CTA).  Drift (Propagator_without_cutoff.cu:1-129 for the reference
// model; the spin-1 drift otherwise), the step-rule reduction, the noise
// (in-register Philox or an injected buffer in the reference's ind_rand layout)
// and the update psi + dt K + sqrt(dt) xi (:131-157, Lattice.cu:32-36) happen
// in registers, and the new state goes to the other buffer of the ping-pong
// pair.  The step size follows the same protocol as the fused kernel:
// speculative update with dt_max and an exact redo of rejected chains (K/max
// rule), or a reduce-only pass and an apply pass (the reference's rule; at FP64
// the reduce pass stores the drift and the site-parallel update applies it).
#include "clv_internal.cuh"
#include "clv_launch.h"
#include "drift_math.cuh"

namespace clv {

template <class R, class C2>
__device__ __forceinline__ void normal_pair(uint64_t seed, uint32_t chain, uint64_t step, int pair,
                                            uint32_t site, C2 &z0, C2 &z1) {
    const uint4 o = philox_block(seed, chain, step, pair, site);
    if constexpr (sizeof(R) == 8) {
        const double2 g0 = box_muller64(o.x, o.y), g1 = box_muller64(o.z, o.w);
        z0.x = g0.x; z0.y = g0.y; z1.x = g1.x; z1.y = g1.y;
    } else {
        const float2 g0 = box_muller32(o.x, o.y), g1 = box_muller32(o.z, o.w);
        z0.x = g0.x; z0.y = g0.y; z1.x = g1.x; z1.y = g1.y;
    }
}


// One task: 256 consecutive (chunk, site) pairs of one chain.  LEAN (large FP64 problems): an
// imaginary time's loads are not issued one ahead, which leaves two CTAs an SM their
// registers, so that one warp's drift (FP64 pipe) covers another's normals (integer pipes):
// 45 spin-1 chains of up to 27 x 20 sites, 0.57 M sites: 301 -> 229 us.  REDUCE: the reduce
// pass that stores the drift and the step's unit normals (tiled_reduce_kernel).
template <class R, int MODEL, bool LEAN, bool REDUCE>
__device__ __forceinline__ void tiled_task(const LaunchTiled &A, const TileTask task) {
    using C2 = typename Cx<R>::T;
    constexpr int NC = MODEL == CLV_MODEL_REF4 ? 4 : 3;
    const ChainDev &ch = A.chains[task.chain];
    ChainState *st = A.state + task.chain;
    const int mode = REDUCE ? FUSED_MAXONLY : A.mode;
    if (mode == FUSED_APPLY && A.only_rejected && st->accepted) return;  // uniform per CTA

    const int V = ch.V, T = ch.nt;
    const int flat = task.flat0 + threadIdx.x;
    const int chunk = flat / V, s = flat - chunk * V;
    const bool act = chunk < task.nchunk;
    const C2 *gpsi = reinterpret_cast<const C2 *>(A.psi_in) + ch.off;
    const C2 *gpsic = reinterpret_cast<const C2 *>(A.psic_in) + ch.off;
    const C2 *gkin = reinterpret_cast<const C2 *>(A.kin) + ch.off;
    const C2 *gkinc = reinterpret_cast<const C2 *>(A.kinc) + ch.off;
    C2 *opsi = reinterpret_cast<C2 *>(A.psi_out) + ch.off;
    C2 *opsic = reinterpret_cast<C2 *>(A.psic_out) + ch.off;
    const bool writes = mode != FUSED_MAXONLY;

    R dt = 0;
    uint64_t nstep = 0;
    if (mode == FUSED_SPEC) dt = (R)ch.dt_max;
    if (mode != FUSED_APPLY) nstep = st->step;
    else { dt = (R)st->dt; nstep = st->noise_step; }
    const R sd = (R)sqrt((double)dt);

    auto at = [&](int c, int tau) -> long long {
        const int t = tau < 0 ? tau + T : (tau >= T ? tau - T : tau);
        return ((long long)c * T + t) * V + s;
    };
    const DriftConsts<R> dk(ch);
    const int tau0 = (int)((long long)T * chunk / task.nchunk), tau1 = (int)((long long)T * (chunk + 1) / task.nchunk);
    // carried: psi(tau-1), psibar(tau), psi(tau) and the pair (psibar(tau), psi(tau-1))
    C2 Pp[NC], Qc[NC], Pc[NC];
    Spin1Link<C2> Bm;
    Ref4Pair<C2> Sm;
    // prefetched for the next tau: psi(tau+1), psibar(tau+1), kin(tau-1), kinbar(tau+1)
    C2 nP[NC], nQ[NC], nK[NC], nKc[NC];
    auto load_next = [&](int tau) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            nP[c] = gpsi[at(c, tau + 1)];
            nQ[c] = gpsic[at(c, tau + 1)];
            nK[c] = gkin[at(c, tau - 1)];
            nKc[c] = gkinc[at(c, tau + 1)];
        }
    };
    if (act) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            Pp[c] = gpsi[at(c, tau0 - 1)];
            Qc[c] = gpsic[at(c, tau0)];
            Pc[c] = gpsi[at(c, tau0)];
        }
        if constexpr (MODEL == CLV_MODEL_SPIN1) Bm = spin1_link<R>(dk, Qc, Pp);
        else Sm = ref4_pair<R>(dk.g2, Pp, Qc);
        if (!LEAN) load_next(tau0);
    }

    R mxr = 0, smr = 0;
    int bad = 0;
    const uint64_t seed = ch.seed;
    const int ref_rule = A.dt_rule == CLV_DT_REF_MEANMAX;
    if (act) {
        for (int tau = tau0; tau < tau1; ++tau) {
            if (LEAN) load_next(tau);
            C2 vpp[NC], vcp[NC], km[NC], kp[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) { vpp[c] = nP[c]; vcp[c] = nQ[c]; km[c] = nK[c]; kp[c] = nKc[c]; }
            if (!LEAN && tau + 1 < tau1) load_next(tau + 1);
            C2 K[NC], Kc[NC];
            if constexpr (MODEL == CLV_MODEL_REF4) {
                drift_ref4_psi<R>(dk, Sm, Pp, Pc, km, K);
                Sm = ref4_pair<R>(dk.g2, Pc, vcp);
                drift_ref4_bar<R>(dk, Sm, vpp, Qc, vcp, kp, Kc);
            } else {
                spin1_drift_psi<R>(Bm, Pp, Pc, km, K);
                Bm = spin1_link<R>(dk, vcp, Pc);
                spin1_drift_bar<R>(Bm, vcp, Qc, kp, Kc);
            }
            if (REDUCE || (mode == FUSED_MAXONLY && A.drift_out)) {
                // the stored-drift update reads the drift instead of a second drift pass
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const long long gi = ((long long)c * T + tau) * V + s;
                    reinterpret_cast<C2 *>(A.drift_out)[ch.off + gi] = K[c];
                    reinterpret_cast<C2 *>(A.driftc_out)[ch.off + gi] = Kc[c];
                }
            }
            if (mode != FUSED_APPLY) {
                if (REDUCE || ref_rule) {
                    const R a0 = abs_drift(K[0]);
                    mxr = max_nan(mxr, a0);
                    smr += a0;
                    bad |= not_finite(a0);
                } else {
#pragma unroll
                    for (int c = 0; c < NC; ++c) mxr = max_nan(mxr, max_nan(abs2<R>(K[c]), abs2<R>(Kc[c])));
                }
            }
            if (writes || REDUCE) {
                const uint32_t site = (uint32_t)(tau * V + s);
                C2 z[NC];
                if (REDUCE || A.noise == CLV_NOISE_PHILOX) {
#pragma unroll
                    for (int c = 0; c < NC; c += 2) {
                        if (c + 1 < NC) {
                            normal_pair<R>(seed, (uint32_t)task.chain, nstep, c >> 1, site, z[c], z[c + 1]);
                        } else {
                            const uint2 w = noise_words(seed, (uint32_t)task.chain, nstep, c, NC, site);
                            z[c] = unit_normal<R, C2>(w.x, w.y);
                        }
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        const long long r = ch.noise_off + (((long long)c * V + s) * T + tau) * 2;
                        z[c].x = (R)A.noise_buf[r];
                        z[c].y = (R)A.noise_buf[r + 1];
                    }
                }
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    if (!writes) {
                        opsi[((long long)c * T + tau) * V + s] = z[c];
                        continue;
                    }
                    C2 zz;
                    zz.x = mul_rn<R>(sd, z[c].x);
                    zz.y = mul_rn<R>(sd, z[c].y);
                    const long long gi = ((long long)c * T + tau) * V + s;
                    opsi[gi] = langevin_update<R>(Pc[c], K[c], dt, zz, false);
                    opsic[gi] = langevin_update<R>(Qc[c], Kc[c], dt, zz, true);
                }
            }
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                Pp[c] = Pc[c];
                Pc[c] = vpp[c];
                Qc[c] = vcp[c];
            }
        }
    }
    if (mode == FUSED_APPLY) return;

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
        st->accepted = (mode == FUSED_SPEC && dtn == ch.dt_max) ? 1 : 0;
        if (!st->accepted) st->rejected += (mode == FUSED_SPEC);
        st->arrive = 0;
    }
}

// One CTA per task.  (Persistent CTAs walking the task list measured slower:
// every task start exposes its first loads, which resident CTAs otherwise hide.)
template <class R, int MODEL, bool LEAN>
__global__ void __launch_bounds__(256, LEAN || sizeof(R) == 4 ? 2 : 1) tiled_step_kernel(const LaunchTiled A) {
    // a stored-drift update launched programmatically after this reduce pass may start
    // drawing its noise now; it waits for this grid's end before it reads the results
    asm volatile("griddepcontrol.launch_dependents;");
    tiled_task<R, MODEL, LEAN, false>(A, A.tasks[blockIdx.x]);
}

// The reference rule's reduce pass at FP64 that also draws the step's unit normals: the drift
// keeps the FP64 pipe busy and the normals the integer pipes
// (128 x 128 x 128: 754 us for the drift alone, at one CTA an SM, 783 with the normals; the FP64
// operations 560).
template <int MODEL>
__global__ void __launch_bounds__(256, 2) tiled_reduce_kernel(const LaunchTiled A) {
    tiled_task<double, MODEL, true, true>(A, A.tasks[blockIdx.x]);
}

template <class R>
static const void *tiled_kernel_ptr(int model, int lean, int draw) {
    const bool ref4 = model == CLV_MODEL_REF4;
    if constexpr (sizeof(R) == 8) {
        if (draw) return ref4 ? (const void *)tiled_reduce_kernel<CLV_MODEL_REF4> : (const void *)tiled_reduce_kernel<CLV_MODEL_SPIN1>;
        if (lean && !ref4) return (const void *)tiled_step_kernel<R, CLV_MODEL_SPIN1, true>;
    }
    return ref4 ? (const void *)tiled_step_kernel<R, CLV_MODEL_REF4, false> : (const void *)tiled_step_kernel<R, CLV_MODEL_SPIN1, false>;
}

template <class R>
cudaError_t launch_tiled(const LaunchTiled &L, cudaStream_t s) {
    if (L.ntasks == 0) return cudaSuccess;
    void *args[] = {(void *)&L};
    return cudaLaunchKernel(tiled_kernel_ptr<R>(L.model, L.lean, L.draw), dim3(L.ntasks), dim3(256), args, 0, s);
}

template <class R>
cudaError_t setup_tiled(int model, int lean, int draw, int *ctas_per_sm) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas_per_sm, tiled_kernel_ptr<R>(model, lean, draw), 256, 0);
}

template cudaError_t setup_tiled<float>(int, int, int, int *);
template cudaError_t setup_tiled<double>(int, int, int, int *);
template cudaError_t launch_tiled<float>(const LaunchTiled &, cudaStream_t);
template cudaError_t launch_tiled<double>(const LaunchTiled &, cudaStream_t);

}  // namespace clv
