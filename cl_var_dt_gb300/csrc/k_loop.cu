// k_loop.cu -- many Langevin steps of a small problem in one cooperative launch,
// under the reference's step rule or the K/max rule (exact there without
// speculation: dt is known before any update).
//
// On the reference's own lattices (one chain of 256 x 32: 128 CTAs of one
// imaginary time each) a step of the two-kernel form -- the filter/drift/reduce
// pass, then the update with its noise -- costs more in launches, in the drift's
// round trip and in the update's wait for the reduce pass than in arithmetic.
// Here every CTA keeps its task (one imaginary time, one field, the components
// of FusedTask::cmask) for all steps of the launch and, per step,
//   1. copies the slices it needs from the current buffer set (L2-resident, cp.async),
//   2. filters its lines (the fused kernel's line filters), while its idle warps
//      draw its half of the unit normals of its (imaginary time, components) and
//      store them for the partner CTA of the other field,
//   3. computes the drift of its sites and its step-rule partial,
//   -- every CTA of the chain has arrived --
//   4. derives dt from the chain's partials (every CTA, in the order of the fused
//      kernel's last CTA; the chain's first CTA also advances ChainState),
//   5. updates its sites with dt K + sqrt(dt) xi into the other buffer set,
//   -- the CTAs of its imaginary time and the two next to it have arrived --
// The results are those of the two-kernel form bit for bit: the same filters,
// drift, reduction order, noise stream (Philox block per component pair, the
// update kernel's words) and update rounding.
//
// On these lattices a step is a chain of latencies.  Arrivals are one flag word per CTA
// (a release store), and the waiting CTA's threads poll one flag each: an atomic counter
// serialised 128 arrivals.  The second wait covers only the CTAs whose slices step k + 1
// reads (and whose reads of step k its stores must follow); the partials alternate between
// two sets, since another CTA may still read the last step's.  Step 4 runs in one warp
// without block barriers: the maximum by integer reductions, the sum through the same
// tree as the fused kernel's, and under the K/max rule neither root nor quotient unless
// the maximum is near K / dt_max.  256 x 32, FP64: 25.1 -> 20.3 us a step; 64 x 64: 17.5 -> 13.3.
// Every wait is bounded (0.5 s), after which the CTA raises CLV_FLAG_TIMEOUT and an abort
// flag that makes every CTA leave at its next wait.  A cooperative launch guarantees
// that all CTAs are resident.
#include "fused_impl.cuh"

namespace clv {

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ int ld_volatile_i32(const int *p) {
    return *reinterpret_cast<const volatile int *>(p);
}

// L2 to shared memory without registers (cp.async.cg passes the SM's own cache by, which may
// hold a slice of two steps ago; it takes 16 bytes, so FP32 elements go through registers)
__device__ __forceinline__ void copy_l2(double2 *s, const double2 *g) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(s)), "l"(g) : "memory");
}
__device__ __forceinline__ void copy_l2(float2 *s, const float2 *g) { *s = __ldcg(g); }

// Largest of a warp's values that are not negative (NaN: the largest of all), by integers.
__device__ __forceinline__ double max_warp(double v) {
    const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
    const unsigned h = __reduce_max_sync(0xffffffffu, hi);
    const unsigned l = __reduce_max_sync(0xffffffffu, hi == h ? lo : 0u);
    return __hiloint2double((int)h, (int)l);
}

// This CTA's writes so far are visible to whoever sees the flag (call by all threads).
__device__ __forceinline__ void loop_arrive(unsigned *flag, unsigned gen) {
    __syncthreads();
    if (threadIdx.x == 0) asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(flag), "r"(gen) : "memory");
}

// Waits for n flags to reach gen (thread i polls flag i of `flag(i)`); true when all did.
template <class Flag>
__device__ __forceinline__ bool loop_wait(const LaunchLoop &A, int n, unsigned gen, ChainState *st, Flag flag) {
    int good = 1;
    uint64_t t0 = 0;
    for (int i = threadIdx.x; i < n && good; i += blockDim.x) {
        const unsigned *p = flag(i);
        for (int k = 0;; ++k) {
            if (ld_acquire_u32(p) >= gen) break;
            if (k == 0) t0 = globaltimer_ns();
            if ((k & 63) == 63 &&
                (ld_volatile_i32(A.abort) || k >= (1 << 26) || globaltimer_ns() - t0 > 500000000ull)) {
                good = 0;
                break;
            }
        }
    }
    if (__syncthreads_and(good)) return true;
    if (threadIdx.x == 0) {
        atomicExch(A.abort, 1);
        atomicOr(&st->flags, CLV_FLAG_TIMEOUT);
    }
    return false;
}

template <class R, int MODEL, int LN>
__global__ void __launch_bounds__(256, 1) loop_step_kernel(const LaunchLoop A) {
    using C2 = typename Cx<R>::T;
    constexpr int NC = MODEL == CLV_MODEL_REF4 ? 4 : 3;
    constexpr int CS = padded_line(LN);
    constexpr int SLOT = fused_slot_stride(NC, LN, (int)sizeof(C2));
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ double s_dt, s_sd;
    __shared__ double s_mx[8], s_sm[8];

    const FusedTask task = A.tasks[blockIdx.x];
    const ChainDev &ch = A.chains[task.chain];
    ChainState *st = A.state + task.chain;
    const int side = task.side;  // 1: psi, 2: psibar (the loop needs split tasks)
    const bool do_psi = side == 1, do_bar = side == 2;
    const int cmask = task.cmask ? task.cmask : (1 << NC) - 1;
    auto own = [&](int c) { return ((cmask >> c) & 1) != 0; };
    const int tau = task.tau0, T = ch.nt, TV = T * LN;
    const int tm = tau == 0 ? T - 1 : tau - 1, tp = tau == T - 1 ? 0 : tau + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, s = threadIdx.x;
    const bool leader = task.part == 0;  // advances the chain's ChainState

    C2 *slots = reinterpret_cast<C2 *>(smem + fused_tab_bytes(LN, (int)sizeof(C2), LN));
    C2 *sPm = slots, *sPc = slots + SLOT, *sPp = slots + 2 * SLOT, *sQc = slots + 3 * SLOT,
       *sQp = slots + 4 * SLOT, *sX = slots + 5 * SLOT, *sY = slots + 6 * SLOT;
    const LineFilter<R, LN> lines(smem, ch, LN, NC, A.kinetic);
    const bool wc = A.kinetic == CLV_KIN_EXP;
    const DriftConsts<R> dk(ch);
    const uint64_t seed = ch.seed, nstep0 = __ldcg(&st->step);
    C2 *nz = reinterpret_cast<C2 *>(A.noise) + ch.off;

    // lines of this CTA (bit job * NC + c) and the warps that filter them; the others
    // draw the CTA's half of the unit normals meanwhile
    const int own_lines = cmask & ((1 << NC) - 1);
    const int mask = do_psi ? own_lines : own_lines << NC;
    // FP64 lines of 256 take two warps each when they fit (no more than four of them)
    const int nl = __popc(mask);
    const bool pair = sizeof(R) == 8 && LN == 256 && 2 * nl <= 8;
    const int used = pair ? (1 << (2 * nl)) - 1 : (mask & 0xFF);
    const int idle = ~used & 0xFF;
    const bool noise_warp = (idle >> warp) & 1;
    const int nthr = __popc(idle) * 32, tn = __popc(idle & ((1 << warp) - 1)) * 32 + lane;
    const int n0 = do_psi ? 0 : LN / 2, n1 = do_psi ? LN / 2 : LN;

    auto draw = [&](int x, uint64_t nstep) {
        const uint32_t site = (uint32_t)(tau * LN + x);
#pragma unroll
        for (int p = 0; p < (NC + 1) / 2; ++p) {
            if (!((cmask >> (2 * p)) & 3)) continue;
            const bool lone = lone_component(2 * p, NC);  // (noise_words)
            const uint4 o = philox_block(seed, (uint32_t)task.chain, nstep, p, lone ? site >> 1 : site);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int c = 2 * p + u;
                if (c >= NC || !own(c)) continue;
                const bool hi = lone ? (site & 1) != 0 : u != 0;
                const uint32_t wx = hi ? o.z : o.x, wy = hi ? o.w : o.y;
                C2 z;
                if constexpr (sizeof(R) == 8) {
                    const double2 g = box_muller64(wx, wy);
                    z.x = (R)g.x; z.y = (R)g.y;
                } else {
                    const float2 g = box_muller32(wx, wy);
                    z.x = (R)g.x; z.y = (R)g.y;
                }
                nz[(c * T + tau) * LN + x] = z;
            }
        }
    };

    int buf = A.from;
    const double sd_max = sqrt((double)(R)ch.dt_max);
    const double cap2 = ch.K > 0 && ch.dt_max > 0 ? ch.K / ch.dt_max * (ch.K / ch.dt_max) * (1.0 - 9.1e-13) : 0.0;
    for (int k = 0; k < A.nsteps; ++k) {
        const uint64_t nstep = nstep0 + (uint64_t)k;
        const C2 *psi = reinterpret_cast<const C2 *>(A.fld[buf][0]) + ch.off;
        const C2 *psic = reinterpret_cast<const C2 *>(A.fld[buf][1]) + ch.off;
        C2 *opsi = reinterpret_cast<C2 *>(A.fld[buf ^ 1][0]) + ch.off;
        C2 *opsic = reinterpret_cast<C2 *>(A.fld[buf ^ 1][1]) + ch.off;
        // 1. slices (from L2: other CTAs wrote them in the previous step)
        for (int e = threadIdx.x; e < NC * LN; e += blockDim.x) {
            const int c = e / LN, x = e - c * LN, o = c * CS + x;
            const long long b = (long long)c * TV + x;
            if (do_psi) copy_l2(&sPm[o], &psi[b + tm * LN]);
            copy_l2(&sQp[o], &psic[b + tp * LN]);
            copy_l2(&sPc[o], &psi[b + tau * LN]);
            copy_l2(&sQc[o], &psic[b + tau * LN]);
            if (MODEL == CLV_MODEL_REF4 && do_bar) copy_l2(&sPp[o], &psi[b + tp * LN]);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        // 2. kinetic term of the filtered field (psi side: kin(tau-1); psibar side:
        //    kinbar(tau+1)) into sX; unit normals by the idle warps
        {
            const C2 *src = do_psi ? sPm : sQp;
            if (pair) {
                const int g = warp >> 1;
                if (g < nl) {
                    int m = mask;
                    for (int i = 0; i < g; ++i) m &= m - 1;
                    const int bit = __ffs(m) - 1, c = bit - (bit >= NC ? NC : 0);
                    if constexpr (sizeof(R) == 8 && LN == 256)
                        lines.template run<64>(ch, wc, c, src + c * CS, sX + c * CS, sY + c * CS, threadIdx.x & 63, g);
                }
            } else if ((mask >> warp) & 1) {
                const int c = warp - (warp >= NC ? NC : 0);
                lines.run(ch, wc, c, src + c * CS, sX + c * CS, sY + c * CS, lane);
            }
            if (noise_warp)
                for (int x = n0 + tn; x < n1; x += nthr) draw(x, nstep);
        }
        if (nthr == 0)
            for (int x = n0 + threadIdx.x; x < n1; x += blockDim.x) draw(x, nstep);
        __syncthreads();
        // 3. drift of site s and the step-rule partial (the fused kernel's REF-rule code)
        C2 K[NC], Kc[NC], pc[NC], qc[NC];
        R mxr = 0, smr = 0;
        int bad = 0;
        if (s < LN) {
            C2 pm[NC], pp[NC], cp[NC], km[NC], kp[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                K[c] = Kc[c] = mk<C2>(0.0, 0.0);
                pc[c] = sPc[c * CS + s];
                qc[c] = sQc[c * CS + s];
                cp[c] = sQp[c * CS + s];
                pm[c] = do_psi ? sPm[c * CS + s] : mk<C2>(0.0, 0.0);
                pp[c] = (MODEL == CLV_MODEL_REF4 && do_bar) ? sPp[c * CS + s] : mk<C2>(0.0, 0.0);
                km[c] = do_psi ? sX[c * CS + s] : mk<C2>(0.0, 0.0);
                kp[c] = do_bar ? sX[c * CS + s] : mk<C2>(0.0, 0.0);
            }
            if (MODEL == CLV_MODEL_REF4)
                drift_ref4_vals<R>(dk, pm, pc, pp, qc, cp, km, kp, K, Kc, do_psi ? 1 : 2, cmask);
            else
                drift_spin1_vals<R>(dk, pm, pc, qc, cp, km, kp, K, Kc, do_psi ? 1 : 2);
            if (A.dt_rule == CLV_DT_REF_MEANMAX) {
                if (own(0)) {  // (a psibar CTA's K is zero)
                    const R a0 = abs_drift(K[0]);
                    mxr = max_nan(mxr, a0);
                    smr += a0;
                    bad |= not_finite(a0);
                }
            } else {
                // K/max rule: max |K|^2 over this CTA's field and components (the chain's
                // maximum is the same whichever CTA finds it)
#pragma unroll
                for (int c = 0; c < NC; ++c)
                    if (own(c)) mxr = max_nan(mxr, abs2<R>(do_psi ? K[c] : Kc[c]));
            }
        }
        // the CTA's partial, in the order of block_max_sum (the sum only under the reference's rule)
        const bool ref_rule = A.dt_rule == CLV_DT_REF_MEANMAX;
        double mx = max_warp((double)mxr), sm = (double)smr;
        if (ref_rule) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sm += __shfl_xor_sync(0xffffffffu, sm, o);
        }
        if (lane == 0) {
            s_mx[warp] = mx;
            s_sm[warp] = sm;
        }
        bad = __syncthreads_or(bad | (lane == 0 && (not_finite(mx) || not_finite(sm))));
        double2 *parts = A.partials + ((k & 1) ? A.part_stride : 0);
        if (warp == 0) {
            mx = max_warp(lane < 8 ? s_mx[lane] : 0.0);
            sm = lane < 8 ? s_sm[lane] : 0.0;
            if (ref_rule) {
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) sm += __shfl_xor_sync(0xffffffffu, sm, o);
            }
            if (lane == 0)
                __stcg(&parts[ch.fused_block0 + task.part],
                       make_double2(mx, bad ? __longlong_as_double(0x7ff8000000000000ll) : sm));
        }
        if (A.withhold && blockIdx.x == 0 && k == 0) {
            // test hook: this CTA leaves without arriving, so the others' waits run out
            if (threadIdx.x == 0) atomicOr(&st->flags, CLV_FLAG_TIMEOUT);
            return;
        }
        const unsigned gen = (unsigned)k + 1;
        loop_arrive(A.bar + blockIdx.x, gen);
        if (!loop_wait(A, ch.fused_nblocks, gen, st, [&](int i) { return A.bar + ch.fused_block0 + i; })) return;
        // the normals of this CTA's sites (half of them drawn by the partner) on their way
        C2 z[NC];
        if (s < LN) {
#pragma unroll
            for (int c = 0; c < NC; ++c)
                if (own(c)) z[c] = __ldcg(&nz[(c * T + tau) * LN + s]);
        }
        // 4. dt from the chain's partials, in the fused kernel's order: thread i of 256 would hold
        //    partial i (+ 256, ...); lane l here holds those of threads l, l + 32, ...
        int finish_bad = 0;
        double fin_dt = 0, fin_mean = 0;
        if (warp == 0) {
            double2 p[4];
            const int nb = ch.fused_nblocks;
#pragma unroll
            for (int g = 0; g < 4; ++g) p[g] = lane + 32 * g < nb ? __ldcg(&parts[ch.fused_block0 + lane + 32 * g]) : make_double2(0.0, 0.0);
            int b = 0;
            mx = 0.0;
            auto take = [&](double2 v) {
                b |= not_finite(v.x) || not_finite(v.y);
                if (!(__double2hiint(v.x) > 0x7ff00000)) mx = max_nan(mx, v.x);  // (fmax drops a NaN)
            };
#pragma unroll
            for (int g = 0; g < 4; ++g) take(p[g]);
            sm = 0.0;
            if (ref_rule) {
                double ts[8];
#pragma unroll
                for (int g = 0; g < 8; ++g) ts[g] = g < 4 ? p[g].y : 0.0;
                for (int i = lane + 128; i < nb; i += 32) {
                    const double2 v = __ldcg(&parts[ch.fused_block0 + i]);
                    take(v);
#pragma unroll
                    for (int g = 0; g < 8; ++g)
                        if (((i >> 5) & 7) == g) ts[g] += v.y;
                }
                // eight warps' xor trees at once (each step halves the sums a lane carries), then
                // the tree over the warps
                int o = 16;
#pragma unroll
                for (int n = 4; n >= 1; n /= 2, o /= 2) {
                    const bool up = (lane & o) != 0;
#pragma unroll
                    for (int i = 0; i < n; ++i) {
                        const double send = up ? ts[i] : ts[i + n], keep = up ? ts[i + n] : ts[i];
                        ts[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                    }
                }
                sm = ts[0] + __shfl_xor_sync(0xffffffffu, ts[0], 2);
                sm += __shfl_xor_sync(0xffffffffu, sm, 1);
                // lane 4 w holds warp w's sum
                sm += __shfl_xor_sync(0xffffffffu, sm, 16);
                sm += __shfl_xor_sync(0xffffffffu, sm, 8);
                sm += __shfl_xor_sync(0xffffffffu, sm, 4);
            } else {
                for (int i = lane + 128; i < nb; i += 32) take(__ldcg(&parts[ch.fused_block0 + i]));
            }
            finish_bad = __any_sync(0xffffffffu, b);
            mx = max_warp(mx);
            if (lane == 0) {
                // K/max: K / sqrt(mx) >= dt_max for certain below this (2^-40 relative margin)
                const bool capped = !ref_rule && mx < cap2;
                double m = mx;
                if (capped) {
                    fin_dt = ch.dt_max;
                } else {
                    ChainState scratch{};
                    fin_dt = step_rule(ch, leader ? *st : scratch, A.dt_rule, m, sm, fin_mean);
                }
                s_dt = fin_dt;
                s_sd = capped ? sd_max : sqrt((double)(R)fin_dt);
            }
        }
        __syncthreads();
        // 5. update (the rounding of the stored-drift update at FP64 and of the fused
        //    apply pass at FP32, whose sqrt takes the step rounded to FP32)
        const R dt = (R)s_dt, sd = (R)s_sd;
        if (s < LN) {
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                if (!own(c)) continue;
                const long long gi = (long long)c * TV + tau * LN + s;
                z[c].x = mul_rn<R>(sd, z[c].x);
                z[c].y = mul_rn<R>(sd, z[c].y);
                if (do_psi) opsi[gi] = langevin_update<R>(pc[c], K[c], dt, z[c], false);
                else opsic[gi] = langevin_update<R>(qc[c], Kc[c], dt, z[c], true);
            }
        }
        loop_arrive(A.bar + A.ntasks + blockIdx.x, gen);
        if (leader && threadIdx.x == 0) {  // (off the others' path: nobody waits for it)
            if (finish_bad || not_finite(mx) || not_finite(sm)) st->flags |= CLV_FLAG_NONFINITE;
            st->dt = fin_dt;
            st->max = ref_rule ? mx : sqrt(mx);
            st->mean = fin_mean;
            st->t += fin_dt;
            st->noise_step = nstep;
            st->step = nstep + 1;
            st->accepted = 0;
        }
        // the CTAs of imaginary times tau - 1, tau, tau + 1 of this chain (parts per time each)
        const int per = ch.fused_nblocks / T;
        if (!loop_wait(A, 3 * per, gen, st, [&](int i) {
                const int u = i / per, t = u == 0 ? tm : (u == 1 ? tau : tp);
                return A.bar + A.ntasks + ch.fused_block0 + t * per + (i - u * per);
            }))
            return;
        buf ^= 1;
    }
}

template <class R, int MODEL>
static void *loop_kernel_of(int ln) {
    switch (ln) {
        case 64: return (void *)loop_step_kernel<R, MODEL, 64>;
        case 128: return (void *)loop_step_kernel<R, MODEL, 128>;
        case 256: return (void *)loop_step_kernel<R, MODEL, 256>;
        default: return nullptr;
    }
}
template <class R>
static void *loop_kernel(int model, int ln) {
    return model == CLV_MODEL_REF4 ? loop_kernel_of<R, CLV_MODEL_REF4>(ln) : loop_kernel_of<R, CLV_MODEL_SPIN1>(ln);
}

size_t loop_smem_bytes(int model, int ln, int esz) {
    const int nc = model == CLV_MODEL_REF4 ? 4 : 3;
    return (size_t)fused_tab_bytes(ln, esz, ln) + 7 * (size_t)fused_slot_stride(nc, ln, esz) * esz;
}

template <class R>
cudaError_t setup_loop(int model, int ln, int *ctas_per_sm) {
    *ctas_per_sm = 0;
    void *fn = loop_kernel<R>(model, ln);
    if (!fn) return cudaSuccess;
    const size_t smem = loop_smem_bytes(model, ln, (int)sizeof(typename Cx<R>::T));
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas_per_sm, fn, 256, smem);
}

template <class R>
cudaError_t launch_loop(const LaunchLoop &L, cudaStream_t s) {
    void *fn = loop_kernel<R>(L.model, L.ln);
    if (!fn) return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(L.ntasks);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = loop_smem_bytes(L.model, L.ln, (int)sizeof(typename Cx<R>::T));
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    void *args[] = {const_cast<LaunchLoop *>(&L)};
    return cudaLaunchKernelExC(&cfg, fn, args);
}

template cudaError_t setup_loop<double>(int, int, int *);
template cudaError_t setup_loop<float>(int, int, int *);
template cudaError_t launch_loop<double>(const LaunchLoop &, cudaStream_t);
template cudaError_t launch_loop<float>(const LaunchLoop &, cudaStream_t);

}  // namespace clv
