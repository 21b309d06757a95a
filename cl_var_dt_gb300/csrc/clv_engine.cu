// clv_engine.cu -- host side of the engine and the C ABI declared in include/clv.h.
//
// An engine owns, on one GPU, the fields of a batch of chains (packed one after
// another, each chain in the reference layout [c][tau][x][y][z]), the scratch
// for the kinetic term and the drift, per-chain constant tables (FFT twiddles,
// kinetic filters), per-chain device step state, and the work tables that map
// CTAs to (chain, lines) and (chain, sites).  A Langevin step is a fixed
// sequence of launches on one stream with no host synchronisation; repeated
// steps replay a captured CUDA graph.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <string>
#include <tuple>
#include <utility>
#include <vector>

#include "clv_internal.cuh"
#include "clv_launch.h"
#include "tile_plan.h"

using namespace clv;

namespace {

thread_local std::string g_last_error;

int fail(int code, const std::string &msg) {
    g_last_error = msg;
    return code;
}

#define CK(call)                                                                          \
    do {                                                                                  \
        cudaError_t _e = (call);                                                          \
        if (_e != cudaSuccess)                                                            \
            return fail(CLV_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(_e)); \
    } while (0)

// Signed momentum of compute_kinetic_part (Propagator_without_cutoff.cu:169-194).
double pmom(int j, int L) {
    if (j < L / 2 || L == 1) return 2. * M_PI * double(j) / double(L);
    return -2. * M_PI * double(L - j) / double(L);
}

bool factorize(int n, int *fac, int &nf) {
    nf = 0;
    while (n % 8 == 0 && nf < kMaxFactors) { fac[nf++] = 8; n /= 8; }
    while (n % 4 == 0 && nf < kMaxFactors) { fac[nf++] = 4; n /= 4; }
    while (n % 2 == 0 && nf < kMaxFactors) { fac[nf++] = 2; n /= 2; }
    while (n % 3 == 0 && nf < kMaxFactors) { fac[nf++] = 3; n /= 3; }
    while (n % 5 == 0 && nf < kMaxFactors) { fac[nf++] = 5; n /= 5; }
    return n == 1;
}

}  // namespace

namespace clv {
// Sets the message clv_last_error() returns, for entry points defined in other
// translation units.
int record_failure(int code, const std::string &msg) { return fail(code, msg); }
}  // namespace clv

struct clv_engine {
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    int model = 0, kinetic = 0, dt_rule = 0, noise = 0, precision = 0, ncomp = 4;
    std::vector<clv_chain_params> params;
    std::vector<ChainDev> chains_h;
    ChainDev *chains_d = nullptr;
    ChainState *state_d = nullptr;
    size_t elem_bytes = 16;
    long long total_elems = 0;  // per field, all chains
    long long max_chain_elems = 0;
    long long noise_total = 0;  // doubles of an external noise buffer, all chains
    void *fld[2][2] = {{nullptr, nullptr}, {nullptr, nullptr}};  // [buffer set][psi, psibar]
    int cur = 0;                    // buffer set holding the current state
    void *kin = nullptr, *kinc = nullptr;
    void *drift = nullptr, *driftc = nullptr;
    // fused path (every chain's slice fits in shared memory)
    bool fused = false, speculate = true, use_tma = true;
    bool withhold_copy = false;  // CLV_TEST_WITHHOLD_COPY: exercise the bounded-wait timeout
    // two-pass (reference dt rule) fused steps: the reduce pass stores the drift and a
    // streaming update applies it, instead of a second filter + drift pass
    bool store_drift = false;
    bool tiled_lean = false;      // tiled, FP64: enough sites for two CTAs an SM (k_tiled.cu)
    bool draw_in_reduce = false;  // tiled: the reduce pass draws the normals of the stored-drift update
    std::vector<FusedTask> fused_tasks_h;
    FusedTask *fused_tasks = nullptr;
    double2 *fused_partials = nullptr;
    int slot_stride = 0, comp_stride = 0;
    int fused_tab_n = 0, fused_tab_bytes = 0, fused_ln = 0;
    size_t fused_smem = 0;
    int fused_ctas_per_sm = 0;
    int num_sms = 0;
    long long all_sites = 0;  // site count over chains and imaginary times
    bool fused_split = false;  // psi and psibar in separate CTAs (build_fused_tasks)
    // step loop (k_loop.cu): resident CTAs of the loop kernel per SM (0: not available)
    int loop_per_sm = 0;
    unsigned int *loop_sync = nullptr;  // the step loop's arrival flags and abort flag
    void *loop_noise = nullptr;         // a step's unit normals (field layout), allocated for problems it fits
    // tiled path (slices too large for the fused kernel): per-axis filter
    // launches grouped by (axis, line length), then the tau-streaming step
    struct AxisGroup {
        int axis, n, pitch, with_const;
        int W;          // lines per tile
        int plane = 0;  // 1: square planes over axes (axis, axis + 1) by the plane filter
        int tile = 0;   // 1: tile filter (k_tile.cuh), tasks in ttasks; n = 0 when lengths differ
        int threads = 128;
        int whole = 0;  // tile filter over whole slices
        int resident = 0;  // plane filter: CTAs the GPU holds
        std::vector<TileFilterTask> ttasks;
        TileFilterTask *td = nullptr;
        int strided = 1;  // every chain's lines of this axis are neighbours in memory (stride > 1)
        size_t smem;
        std::vector<AxisTask> tasks;
        AxisTask *d = nullptr;
        int ntasks() const { return (int)(tile ? ttasks.size() : tasks.size()); }
        int chain_of(int i) const { return tile ? ttasks[i].chain : tasks[i].chain; }
    };
    bool tiled = false;
    // Chains [c0, c1) whose kinetic terms are held at once (tiled path): all of them, or, where
    // kinbar has no memory, as many at a time as kin holds twice (plan_windows); groups: first
    // task and count in every launch group
    struct Window {
        int c0, c1;
        long long off, elems;  // of the chains in a field array
        std::vector<std::pair<int, int>> groups;
    };
    std::vector<Window> windows;
    std::vector<TileFilterPlan> tile_plans_h;
    TileFilterPlan *tile_plans = nullptr;
    std::vector<AxisGroup> axis_groups;
    bool energy_axis = false;             // kinetic energy of the observables by axis filters
    std::vector<AxisGroup> energy_groups;
    // plan knobs (heuristic defaults, CLV_* overrides, or chosen by clv_autotune)
    int chunk = 0;               // imaginary times per CTA of the step kernel
    int fused_ln_static = 0;     // compile-time line length available to the fused path
    bool fused_aligned = false;  // rows 16-byte aligned: bulk copies possible
    size_t task_capacity = 0;    // task/partial slots allocated (finest chunking)
    std::string tune_report;
    std::vector<TileTask> tile_tasks_h;
    TileTask *tile_tasks = nullptr;
    double2 *stage = nullptr;     // complex128 staging (2 * max_chain_elems)
    double2 *stage_all = nullptr; // staging for all-chain copies, allocated on first use
    long long stage_all_elems = 0;
    double *noise_d = nullptr;
    std::vector<SiteTask> site_tasks_h, obs_tasks_h;
    SiteTask *site_tasks = nullptr, *obs_tasks = nullptr;
    std::vector<ObsTask> obs_pairs_h;     // observables
    ObsTask *obs_pairs = nullptr;
    double *obs_partials = nullptr, *obs_scratch = nullptr;
    long long obs_scratch_n = 0;          // doubles (reference model)
    bool obs_group = false;               // 16 pairs a CTA (k_obs.cu)
    unsigned int *obs_arrive = nullptr;
    std::vector<LineTask> line_tasks_h[3];
    LineTask *line_tasks[3] = {nullptr, nullptr, nullptr};
    int max_bundle[3] = {0, 0, 0};
    double2 *partials = nullptr;
    double *accF = nullptr, *accN = nullptr;
    int acc_F_total = 0;
    int counter = 0;
    double *samples = nullptr;
    int sample_cap = 1024, sample_count = 0;
    std::vector<double> sample_spill;  // [k][chain][8] samples moved to the host
    int sample_spilled = 0;
    std::vector<void *> allocs;
    size_t dev_bytes = 0;
    cudaGraphExec_t graph_exec[2] = {nullptr, nullptr};  // keyed by the starting buffer set
    cudaGraph_t graph[2] = {nullptr, nullptr};
    // kStepBlock steps in one graph (an even count: the buffer set returns to its start)
    cudaGraphExec_t block_exec[2] = {nullptr, nullptr};
    cudaGraph_t block_graph[2] = {nullptr, nullptr};

    void *psi() const { return fld[cur][0]; }
    void *psic() const { return fld[cur][1]; }
    void drop_graphs() {
        for (int i = 0; i < 2; ++i) {
            if (graph_exec[i]) cudaGraphExecDestroy(graph_exec[i]);
            if (graph[i]) cudaGraphDestroy(graph[i]);
            if (block_exec[i]) cudaGraphExecDestroy(block_exec[i]);
            if (block_graph[i]) cudaGraphDestroy(block_graph[i]);
            graph_exec[i] = block_exec[i] = nullptr;
            graph[i] = block_graph[i] = nullptr;
        }
    }

    template <class T>
    int alloc(T **p, size_t bytes) {
        void *q = nullptr;
        if (bytes == 0) bytes = 16;
        cudaError_t e = cudaMalloc(&q, bytes);
        if (e != cudaSuccess)
            return fail(CLV_ERR_NOMEM, std::string("cudaMalloc(") + std::to_string(bytes) +
                                           "): " + cudaGetErrorString(e));
        allocs.push_back(q);
        dev_bytes += bytes;
        *p = (T *)q;
        return CLV_OK;
    }

    template <class T>
    void release(T **p, size_t bytes) {
        allocs.erase(std::find(allocs.begin(), allocs.end(), *p));
        dev_bytes -= bytes;
        cudaFree(*p);
        *p = nullptr;
    }

    LaunchObs obs() const {
        LaunchObs L{};
        L.chains = chains_d;
        L.tasks = obs_pairs;
        L.ntasks = (int)obs_pairs_h.size();
        L.psi = psi();
        L.psic = psic();
        L.partials = obs_partials;
        return L;
    }

    LaunchSites sites() const {
        LaunchSites L{};
        L.chains = chains_d;
        L.state = state_d;
        L.tasks = site_tasks;
        L.ntasks = (int)site_tasks_h.size();
        L.model = model;
        L.dt_rule = dt_rule;
        L.noise = noise;
        L.psi = psi(); L.psic = psic(); L.kin = kin; L.kinc = kinc;
        L.psi_w = psi(); L.psic_w = psic();
        L.drift = drift; L.driftc = driftc;
        L.partials = partials;
        L.noise_buf = noise_d;
        return L;
    }
};

namespace {

int build_tables(clv_engine *e) {
    const int nch = (int)e->params.size();
    e->chains_h.resize(nch);
    long long off = 0, noff = 0;
    int obs_off = 0;
    // host staging for every table, uploaded at once
    struct Pending { void **dst; std::vector<unsigned char> bytes; size_t off; };
    std::vector<Pending> pend;
    auto table = [&](auto **dst, auto &&vec) {
        Pending p;
        p.dst = (void **)dst;
        p.bytes.resize(vec.size() * sizeof(vec[0]));
        std::memcpy(p.bytes.data(), vec.data(), p.bytes.size());
        pend.push_back(std::move(p));
    };
    std::map<int, std::vector<WCplx>> fixed;  // by length: a batch has few
    long long &all_sites = e->all_sites;
    all_sites = 0;
    for (auto &p : e->params) all_sites += (long long)p.nx * p.ny * p.nz * p.nt;
    for (int c = 0; c < nch; ++c) {
        const clv_chain_params &p = e->params[c];
        ChainDev &d = e->chains_h[c];
        std::memset(&d, 0, sizeof d);
        d.nx = p.nx; d.ny = p.ny; d.nz = p.nz; d.nt = p.nt;
        d.V = p.nx * p.ny * p.nz;
        d.ncomp = e->ncomp;
        d.off = off;
        d.noise_off = noff;
        d.eps = p.eps; d.a_x = p.a_x; d.mu = p.mu; d.P = p.P; d.Q = p.Q; d.G = p.G;
        d.DT = p.DT; d.dt_min = p.dt_min; d.dt_max_clamp = p.dt_max_clamp; d.alpha = p.alpha;
        d.c0 = p.c0; d.c1 = p.c1; d.q = p.q; d.K = p.K; d.dt_max = p.dt_max;
        d.seed = p.seed;
        for (int a = 0; a < kMaxComp; ++a) {
            const double m = 1.0 - a;
            d.comp_const[a] = std::exp(p.eps * (p.mu + p.q * m * m));
        }
        const long long elems = (long long)e->ncomp * p.nt * d.V;
        off += elems;
        noff += 2 * elems;
        e->max_chain_elems = std::max(e->max_chain_elems, elems);
        d.obs_off = obs_off;
        obs_off += 3 * d.V;
        const int dims[3] = {p.nx, p.ny, p.nz};
        const int inner[3] = {p.ny * p.nz, p.nz, 1};
        for (int a = 0; a < 3; ++a) {
            AxisDev &ax = d.axis[a];
            ax.n = dims[a];
            ax.inner = inner[a];
            if (dims[a] <= 1) continue;
            if (!factorize(dims[a], ax.fac, ax.nf))
                return fail(CLV_ERR_ARG, "lattice extent " + std::to_string(dims[a]) +
                                             " has a prime factor other than 2, 3, 5");
            const int n = dims[a];
            std::vector<double2> tw64(n);
            std::vector<float2> tw32(n);
            const long double twopi = 2.0L * acosl(-1.0L);
            for (int k = 0; k < n; ++k) {
                const long double ang = -twopi * (long double)k / (long double)n;
                tw64[k] = make_double2((double)cosl(ang), (double)sinl(ang));
                tw32[k] = make_float2((float)cosl(ang), (float)sinl(ang));
            }
            std::vector<double> f64(n, 0.0), e64(n);
            for (int k = 0; k < n; ++k) {
                const double pk = pmom(k, n);
                if (e->kinetic == CLV_KIN_REF_LINEAR_PX) {
                    // -px^2 (py, pz terms are commented out in the reference) with the
                    // normalisation 1/(a_x NX) of the x-only transform pair
                    f64[k] = a == 0 ? -(pk * pk) / (p.a_x * n) : 1.0 / n;
                } else {
                    f64[k] = std::exp(-p.eps * 0.5 * pk * pk) / n;
                }
                e64[k] = 0.5 * pk * pk / n;
            }
            std::vector<float> f32(f64.begin(), f64.end()), e32(e64.begin(), e64.end());
            table(&ax.tw64, tw64);
            table(&ax.tw32, tw32);
            if (e->precision == CLV_PREC_F64) {
                const auto it = fixed.find(n);
                table(&ax.tw62, it != fixed.end() ? it->second : fixed.emplace(n, fixed_twiddles(n)).first->second);
            }
            table(&ax.filt64, f64);
            table(&ax.filt32, f32);
            table(&ax.efilt64, e64);
            table(&ax.efilt32, e32);
            // the tile filter's plan, and the filters in the order its forward passes leave
            // the frequencies
            if (!tile_factors(n, e->precision == CLV_PREC_F64 ? tile_radix_max<double>() : tile_radix_max<float>(), ax.tfac, ax.tnf))
                ax.tnf = 0;
            if (ax.tnf) {
                const std::vector<int> order = tile_order(n, ax.tfac, ax.tnf);
                std::vector<double> tf64(n), te64(n);
                for (int i = 0; i < n; ++i) {
                    tf64[i] = f64[order[i]];
                    te64[i] = e64[order[i]];
                }
                std::vector<float> tf32(tf64.begin(), tf64.end()), te32(te64.begin(), te64.end());
                for (int k = 0; k < n; ++k) {
                    ax.fmax = std::max(ax.fmax, std::fabs(f64[k]));
                    ax.efmax = std::max(ax.efmax, e64[k]);
                }
                table(&ax.tfilt64, tf64);
                table(&ax.tfilt32, tf32);
                table(&ax.tefilt64, te64);
                table(&ax.tefilt32, te32);
            }
            // per-pass twiddles of the fused kernel's FP32 line plans, from the same rounded
            // values
            if (n == 64 || n == 128 || n == 256 || n == 512) {
                const int ne = tw_entries(n);
                std::vector<float2> p32(ne);
                for (int i = 0; i < ne; ++i) {
                    bool conj = false;
                    const int m = pass_twiddle_source(n, i, &conj);
                    p32[i] = tw32[m];
                    if (conj) p32[i].y = -p32[i].y;
                }
                table(&ax.ptw32, p32);
            }
        }
        // site tasks: kSiteBlock consecutive (tau, s) sites per CTA
        const int nsites = d.V * p.nt;
        d.site_block0 = (int)e->site_tasks_h.size();
        d.site_nblocks = (nsites + kSiteBlock - 1) / kSiteBlock;
        for (int b = 0; b < d.site_nblocks; ++b) e->site_tasks_h.push_back({c, b * kSiteBlock});
        for (int b = 0; b < (d.V + 255) / 256; ++b) e->obs_tasks_h.push_back({c, b * 256});
        // observables: (chunk, site) pairs, chunks of at most 64 imaginary times for the reference
        // model and 16 for spin-1 at FP64, fewer where that leaves SMs idle.  Spin-1 at FP32, whose
        // threads sum in FP32, takes 16 whatever the batch, so that a chain's sample does not
        // depend on the chains beside it; small problems take a thread per imaginary time
        {
            const long long per = all_sites / (2LL * 256 * e->num_sms);
            const bool ref4 = e->model == CLV_MODEL_REF4;
            e->obs_group = !ref4 && e->precision == CLV_PREC_F32 && per < 4;
            const int L = !ref4 && e->precision == CLV_PREC_F32
                              ? 16 : (int)std::max<long long>(1, std::min<long long>(ref4 ? 64 : 16, per));
            d.obs_nchunk = (p.nt + L - 1) / L;
            d.obs_block0 = (int)e->obs_pairs_h.size();
            d.obs_scr = e->obs_scratch_n;
            const long long pairs = (long long)d.V * d.obs_nchunk;
            e->obs_scratch_n += 3 * pairs;
            for (long long f = 0; f < pairs; f += e->obs_group ? 16 : 256) e->obs_pairs_h.push_back({c, (int)f});
            d.obs_nblocks = (int)e->obs_pairs_h.size() - d.obs_block0;
        }
        // line tasks per axis
        const int budget = e->precision == CLV_PREC_F64 ? kMaxBundleElems64 : kMaxBundleElems32;
        for (int a = 0; a < 3; ++a) {
            const int n = dims[a];
            if (n <= 1) continue;
            if (n > kMaxLine) return fail(CLV_ERR_ARG, "lattice extent above 2048");
            const int lines = e->ncomp * p.nt * (d.V / n);
            int W = std::max(1, budget / n);
            W = std::min(W, lines);
            for (int l0 = 0; l0 < lines; l0 += W) {
                const int nl = std::min(W, lines - l0);
                e->line_tasks_h[a].push_back({c, l0, nl});
                e->max_bundle[a] = std::max(e->max_bundle[a], nl * n);
            }
        }
    }
    e->total_elems = off;
    e->noise_total = noff;
    e->acc_F_total = obs_off;
    // upload the tables in one allocation and one copy, equal ones (chains of one length and
    // imaginary-time step) once; device pointers are patched into the host chain copies
    std::map<std::vector<unsigned char>, size_t> at;
    std::vector<unsigned char> pool;
    for (auto &p : pend) {
        const auto it = at.emplace(std::move(p.bytes), pool.size());
        p.off = it.first->second;
        if (it.second) {
            const auto &b = it.first->first;
            pool.insert(pool.end(), b.begin(), b.end());
            pool.resize((pool.size() + 255) / 256 * 256);
        }
    }
    unsigned char *dptr = nullptr;
    if (int rc = e->alloc(&dptr, pool.size())) return rc;
    if (!pool.empty()) CK(cudaMemcpy(dptr, pool.data(), pool.size(), cudaMemcpyHostToDevice));
    for (auto &p : pend) *p.dst = dptr + p.off;
    return CLV_OK;
}

// Optional event trail of a step: an event is recorded after every launch.
struct EventTrail {
    std::vector<cudaEvent_t> ev;
    cudaError_t mark(cudaStream_t s) {
        cudaEvent_t e;
        cudaError_t r = cudaEventCreate(&e);
        if (r != cudaSuccess) return r;
        ev.push_back(e);
        return cudaEventRecord(e, s);
    }
    ~EventTrail() { for (auto e : ev) cudaEventDestroy(e); }
};

template <class R>
int run_kinetic(clv_engine *e, const void *s0, const void *s1, void *d0, void *d1, int filter,
                int nfields, EventTrail *trail = nullptr) {
    bool first = true;
    for (int a = 0; a < 3; ++a) {
        if (e->line_tasks_h[a].empty()) continue;
        if (e->kinetic == CLV_KIN_REF_LINEAR_PX && filter == 0 && a > 0) break;
        LaunchLineFilter L{};
        L.chains = e->chains_d;
        L.tasks = e->line_tasks[a];
        L.ntasks = (int)e->line_tasks_h[a].size();
        L.max_bundle = e->max_bundle[a];
        L.axis = a;
        L.nfields = nfields;
        L.filter = filter;
        if (filter == 0) {
            // kinetic: product over axes, first pass reads the fields
            L.src0 = first ? s0 : d0;
            L.src1 = first ? s1 : d1;
            L.mode = 0;
            L.with_const = first && e->kinetic == CLV_KIN_EXP;
        } else {
            // kinetic energy: sum over axes of the one-axis operators
            L.src0 = s0;
            L.src1 = s1;
            L.mode = first ? 0 : 1;
            L.with_const = 0;
        }
        L.dst0 = d0;
        L.dst1 = d1;
        CK(launch_line_filter<R>(L, e->stream));
        if (trail) CK(trail->mark(e->stream));
        first = false;
    }
    return CLV_OK;
}

LaunchFused fused_launch(const clv_engine *e, int from, int mode, bool ext) {
    LaunchFused L{};
    L.chains = e->chains_d;
    L.state = e->state_d;
    L.tasks = e->fused_tasks;
    L.ntasks = (int)e->fused_tasks_h.size();
    L.model = e->model;
    L.kinetic = e->kinetic;
    L.dt_rule = e->dt_rule;
    L.noise = ext ? CLV_NOISE_EXTERNAL : CLV_NOISE_PHILOX;
    L.mode = mode;
    L.only_rejected = 0;
    L.use_tma = e->use_tma;
    L.withhold = e->withhold_copy && mode != FUSED_APPLY;
    L.alone = L.ntasks <= e->num_sms;
    L.drift_out = (mode == FUSED_MAXONLY && e->store_drift) ? e->drift : nullptr;
    L.driftc_out = (mode == FUSED_MAXONLY && e->store_drift) ? e->driftc : nullptr;
    L.psi_in = e->fld[from][0];
    L.psic_in = e->fld[from][1];
    L.psi_out = e->fld[from ^ 1][0];
    L.psic_out = e->fld[from ^ 1][1];
    L.partials = e->fused_partials;
    L.noise_buf = e->noise_d;
    L.slot_stride = e->slot_stride;
    L.comp_stride = e->comp_stride;
    L.tab_n = e->fused_tab_n;
    L.tab_bytes = e->fused_tab_bytes;
    L.ln = e->fused_ln;
    L.split = e->fused_split ? 1 : 0;
    L.smem_bytes = e->fused_smem;
    return L;
}

// kin and kinbar of a window's chains, as if of all: kinbar's own array, or behind kin's elements.
std::pair<void *, void *> window_kin(const clv_engine *e, const clv_engine::Window &w) {
    if (e->kinc) return {e->kin, e->kinc};
    char *k = static_cast<char *>(e->kin) - w.off * e->elem_bytes;
    return {k, k + w.elems * e->elem_bytes};
}

LaunchTiled tiled_launch(const clv_engine *e, const clv_engine::Window &w, int from, int mode, bool ext) {
    LaunchTiled L{};
    L.chains = e->chains_d;
    L.state = e->state_d;
    const ChainDev &first = e->chains_h[w.c0], &last = e->chains_h[w.c1 - 1];
    L.tasks = e->tile_tasks + first.fused_block0;
    L.ntasks = last.fused_block0 + last.fused_nblocks - first.fused_block0;
    L.model = e->model;
    L.dt_rule = e->dt_rule;
    L.noise = ext ? CLV_NOISE_EXTERNAL : CLV_NOISE_PHILOX;
    L.mode = mode;
    L.only_rejected = 0;
    L.psi_in = e->fld[from][0];
    L.psic_in = e->fld[from][1];
    std::tie(L.kin, L.kinc) = window_kin(e, w);
    L.psi_out = e->fld[from ^ 1][0];
    L.psic_out = e->fld[from ^ 1][1];
    L.partials = e->fused_partials;
    L.noise_buf = e->noise_d;
    L.drift_out = (mode == FUSED_MAXONLY && e->store_drift) ? e->drift : nullptr;
    L.driftc_out = (mode == FUSED_MAXONLY && e->store_drift) ? e->driftc : nullptr;
    L.lean = e->tiled_lean;
    L.draw = mode == FUSED_MAXONLY && e->draw_in_reduce && !ext;
    return L;
}

// The launches of a group list.  Kinetic filter (two fields, src1 not null): the groups of
// axis 0 read the fields, the others continue in kin/kinbar.  Kinetic energy (src1 null):
// every axis reads src0, the first writes kin and the others add to it.  w: the chains of a
// window only.
template <class R>
int run_groups(clv_engine *e, const std::vector<clv_engine::AxisGroup> &groups, const void *src0, const void *src1,
               const clv_engine::Window *w = nullptr, EventTrail *trail = nullptr) {
    const bool energy = src1 == nullptr;
    const auto kin = w ? window_kin(e, *w) : std::pair<void *, void *>(e->kin, e->kinc);
    for (size_t i = 0; i < groups.size(); ++i) {
        const auto &g = groups[i];
        const void *s0 = (energy || g.axis == 0) ? src0 : kin.first, *s1 = g.axis == 0 ? src1 : kin.second;
        const int first = w ? w->groups[i].first : 0, count = w ? w->groups[i].second : g.ntasks();
        if (g.tile) {
            LaunchTileFilter T{};
            T.chains = e->chains_d;
            T.plans = e->tile_plans;
            T.tasks = g.td + first;
            T.ntasks = count;
            T.src0 = s0;
            T.src1 = s1;
            T.dst0 = kin.first;
            T.dst1 = kin.second;
            T.nfields = energy ? 1 : 2;
            T.filter = energy;
            T.accumulate = energy && g.axis > 0;
            T.threads = g.threads;
            T.smem_bytes = g.smem;
            CK(launch_tile_filter<R>(T, e->stream));
        } else {
            LaunchAxis A{};
            A.chains = e->chains_d;
            A.tasks = g.d + first;
            A.ntasks = count;
            A.axis = g.axis;
            A.n = g.n;
            A.W = g.W;
            A.pitch = g.pitch;
            A.with_const = g.with_const;
            A.src0 = s0;
            A.src1 = s1;
            A.dst0 = kin.first;
            A.dst1 = kin.second;
            A.smem_bytes = g.smem;
            A.nfields = energy ? 1 : 2;
            A.filter = energy;
            A.accumulate = energy && g.axis > 0;
            A.strided = g.strided;
            A.resident = g.resident;
            if (g.plane) CK(launch_plane_filter<R>(A, e->stream));
            else if constexpr (sizeof(R) == 4) CK(launch_axis_filter<R>(A, e->stream));
        }
        if (trail) CK(trail->mark(e->stream));
    }
    return CLV_OK;
}

// Tiled step of a window's chains: kinetic filter axis by axis into kin/kinbar, then the streaming
// drift/noise/update kernel (speculative dt with redo, or reduce then apply).
template <class R>
int enqueue_window(clv_engine *e, const clv_engine::Window &w, bool external_noise, EventTrail *trail, int from) {
    if (int rc = run_groups<R>(e, e->axis_groups, e->fld[from][0], e->fld[from][1], &w, trail)) return rc;
    if (e->speculate && e->dt_rule == CLV_DT_K_OVER_MAX) {
        CK(launch_tiled<R>(tiled_launch(e, w, from, FUSED_SPEC, external_noise), e->stream));
        if (trail) CK(trail->mark(e->stream));
        LaunchTiled L = tiled_launch(e, w, from, FUSED_APPLY, external_noise);
        L.only_rejected = 1;
        CK(launch_tiled<R>(L, e->stream));
    } else {
        const LaunchTiled reduce = tiled_launch(e, w, from, FUSED_MAXONLY, external_noise);
        CK(launch_tiled<R>(reduce, e->stream));
        if (trail) CK(trail->mark(e->stream));
        if (e->store_drift) {
            // the stored drift applied by the site-parallel update, which draws its noise
            // while the reduce pass runs (programmatic launch) unless that pass drew it
            const ChainDev &first = e->chains_h[w.c0], &last = e->chains_h[w.c1 - 1];
            LaunchSites L = e->sites();
            L.tasks += first.site_block0;
            L.ntasks = last.site_block0 + last.site_nblocks - first.site_block0;
            L.psi = e->fld[from][0];
            L.psic = e->fld[from][1];
            L.psi_w = e->fld[from ^ 1][0];
            L.psic_w = e->fld[from ^ 1][1];
            L.noise = external_noise ? CLV_NOISE_EXTERNAL : CLV_NOISE_PHILOX;
            L.drawn = reduce.draw;
            L.pdl = !std::getenv("CLV_NO_PDL");
            CK(launch_update<R>(L, e->stream));
        } else {
            CK(launch_tiled<R>(tiled_launch(e, w, from, FUSED_APPLY, external_noise), e->stream));
        }
    }
    if (trail) CK(trail->mark(e->stream));
    return CLV_OK;
}

template <class R>
int enqueue_tiled(clv_engine *e, bool external_noise, EventTrail *trail, int from) {
    for (const auto &w : e->windows)
        if (int rc = enqueue_window<R>(e, w, external_noise, trail, from)) return rc;
    return CLV_OK;
}

// Small problems run many steps per cooperative launch (k_loop.cu) when every split
// task of the fused plan covers one imaginary time and all of them fit on the GPU at
// once; the trajectory is the two-kernel form's bit for bit (CLV_NO_LOOP=1 keeps the
// two-kernel form).
bool use_loop(const clv_engine *e) {
    if (!e->fused || e->fused_ln <= 0 || !e->fused_split || !e->loop_noise) return false;
    if (e->loop_per_sm < 1 || (long long)e->fused_tasks_h.size() > (long long)e->loop_per_sm * e->num_sms)
        return false;
    for (const auto &t : e->fused_tasks_h)
        if (t.tau1 - t.tau0 != 1 || t.side == 0) return false;
    return !std::getenv("CLV_NO_LOOP");
}

// nsteps Philox steps by the step loop, in launches of at most 2^16 steps.  A
// cooperative launch the GPU refuses (the grid cannot be resident now, e.g. beside
// other work on a shared GPU) turns the loop off for this engine: *done tells the
// caller how many steps ran, and kLoopRefused that the rest is its to run.
constexpr int kLoopRefused = -1000;
template <class R>
int enqueue_loop(clv_engine *e, int nsteps, EventTrail *trail, int *done = nullptr) {
    if (done) *done = 0;
    while (nsteps > 0) {
        const int n = std::min(nsteps, 1 << 16);
        const size_t ntasks = e->fused_tasks_h.size();
        CK(cudaMemsetAsync(e->loop_sync, 0, (2 * ntasks + 1) * sizeof(unsigned int), e->stream));
        if (trail) CK(trail->mark(e->stream));
        LaunchLoop L{};
        L.chains = e->chains_d;
        L.state = e->state_d;
        L.tasks = e->fused_tasks;
        L.ntasks = (int)e->fused_tasks_h.size();
        L.nsteps = n;
        L.model = e->model;
        L.kinetic = e->kinetic;
        L.ln = e->fused_ln;
        L.dt_rule = e->dt_rule;
        for (int b = 0; b < 2; ++b)
            for (int f = 0; f < 2; ++f) L.fld[b][f] = e->fld[b][f];
        L.from = e->cur;
        L.noise = e->loop_noise;
        L.partials = e->fused_partials;
        L.part_stride = (int)e->task_capacity;
        L.bar = e->loop_sync;
        L.abort = reinterpret_cast<int *>(e->loop_sync + 2 * ntasks);
        L.withhold = e->withhold_copy;
        const cudaError_t le = launch_loop<R>(L, e->stream);
        if (le == cudaErrorCooperativeLaunchTooLarge) {
            (void)cudaGetLastError();  // a launch-configuration error: nothing ran
            if (trail) {               // (the mark before the refused launch)
                cudaEventDestroy(trail->ev.back());
                trail->ev.pop_back();
            }
            e->loop_per_sm = 0;
            return kLoopRefused;
        }
        CK(le);
        if (trail) CK(trail->mark(e->stream));
        if (n & 1) e->cur ^= 1;
        nsteps -= n;
        if (done) *done += n;
    }
    return CLV_OK;
}

int enqueue_loop_any(clv_engine *e, int nsteps, EventTrail *trail, int *done = nullptr) {
    return e->precision == CLV_PREC_F64 ? enqueue_loop<double>(e, nsteps, trail, done)
                                        : enqueue_loop<float>(e, nsteps, trail, done);
}

// One step reading buffer set `from` and writing set `from ^ 1`.
template <class R>
int enqueue_step(clv_engine *e, bool external_noise, EventTrail *trail, int from) {
    if (e->tiled) return enqueue_tiled<R>(e, external_noise, trail, from);
    if (e->fused) {
        if (e->speculate && e->dt_rule == CLV_DT_K_OVER_MAX) {
            // update with dt = dt_max; chains whose true dt differs are redone
            CK(launch_fused<R>(fused_launch(e, from, FUSED_SPEC, external_noise), e->stream));
            if (trail) CK(trail->mark(e->stream));
            LaunchFused L = fused_launch(e, from, FUSED_APPLY, external_noise);
            L.only_rejected = 1;
            CK(launch_fused<R>(L, e->stream));
        } else {
            CK(launch_fused<R>(fused_launch(e, from, FUSED_MAXONLY, external_noise), e->stream));
            if (trail) CK(trail->mark(e->stream));
            if (e->store_drift) {
                LaunchSites L = e->sites();
                L.psi = e->fld[from][0];
                L.psic = e->fld[from][1];
                L.psi_w = e->fld[from ^ 1][0];
                L.psic_w = e->fld[from ^ 1][1];
                L.noise = external_noise ? CLV_NOISE_EXTERNAL : CLV_NOISE_PHILOX;
                // its noise is drawn while the reduce pass runs (the pass releases its
                // dependents at its start; the update waits for its end before it reads)
                L.pdl = e->dt_rule == CLV_DT_REF_MEANMAX && !std::getenv("CLV_NO_PDL");
                CK(launch_update<R>(L, e->stream));
            } else {
                CK(launch_fused<R>(fused_launch(e, from, FUSED_APPLY, external_noise), e->stream));
            }
        }
        if (trail) CK(trail->mark(e->stream));
        return CLV_OK;
    }
    // lines beyond the tiled path's: the tile filter, or the line filter where the tile path
    // is switched off (CLV_TILED=0)
    int rc = e->axis_groups.empty() ? run_kinetic<R>(e, e->fld[from][0], e->fld[from][1], e->kin, e->kinc, 0, 2, trail)
                                    : run_groups<R>(e, e->axis_groups, e->fld[from][0], e->fld[from][1], nullptr, trail);
    if (rc) return rc;
    LaunchSites L = e->sites();
    L.psi = e->fld[from][0];
    L.psic = e->fld[from][1];
    L.psi_w = e->fld[from ^ 1][0];
    L.psic_w = e->fld[from ^ 1][1];
    L.noise = external_noise ? CLV_NOISE_EXTERNAL : CLV_NOISE_PHILOX;
    CK(launch_drift<R>(L, e->stream));
    if (trail) CK(trail->mark(e->stream));
    CK(launch_update<R>(L, e->stream));
    if (trail) CK(trail->mark(e->stream));
    return CLV_OK;
}

int enqueue_step_any(clv_engine *e, bool ext, EventTrail *trail, int from) {
    return e->precision == CLV_PREC_F64 ? enqueue_step<double>(e, ext, trail, from)
                                        : enqueue_step<float>(e, ext, trail, from);
}

// Fused step tasks: chunks of L imaginary times.  Under the reference's step rule
// (two passes on the generic kernel), when the chunks are fewer than the SMs (the
// reference's own 256 x 32 lattice: 32 chunks), each chunk becomes a psi CTA and a
// psibar CTA, so twice as many SMs share the FFT and drift work; under the K/max
// rule the production variant on whole chunks measured faster (one 1D 256 x 128
// chain at FP64: 0.086 against 0.129 ms).  CLV_FUSED_SPLIT=0/1 overrides.
void build_fused_tasks(clv_engine *e, int L) {
    e->chunk = L;
    e->fused_tasks_h.clear();
    long long chunks = 0;
    for (auto &d : e->chains_h) chunks += std::max(1, (d.nt + L - 1) / L);
    bool split = e->dt_rule == CLV_DT_REF_MEANMAX && chunks < e->num_sms;
    // under the K/max rule too when the step loop takes the problem: chunks of one
    // imaginary time whose split tasks are all resident at once (the FP64 single chain
    // of 64 sites x 64 imaginary times)
    if (e->dt_rule == CLV_DT_K_OVER_MAX && L == 1 && e->fused_ln > 0 && e->loop_per_sm > 0 &&
        2 * chunks <= (long long)e->loop_per_sm * e->num_sms && !std::getenv("CLV_NO_LOOP"))
        split = true;
    if (const char *sp = std::getenv("CLV_FUSED_SPLIT")) split = sp[0] == '1';
    // fewer still (the reference's 256 x 32 lattice: 64 split CTAs on 152 SMs) and the
    // FP64 pipe the bound: each field's CTA splits again into component halves, so a
    // CTA filters two lines and drifts two components, on 1D lines of the 4-component
    // model (CLV_FUSED_CSPLIT=0/1 overrides)
    bool csplit = split && e->ncomp == 4 && e->precision == CLV_PREC_F64 && 4 * chunks <= e->num_sms;
    for (auto &d : e->chains_h)
        if (d.ny != 1 || d.nz != 1) csplit = false;
    if (const char *cs = std::getenv("CLV_FUSED_CSPLIT")) csplit = split && e->ncomp == 4 && cs[0] == '1';
    e->fused_split = split;
    const int per_chunk = split ? (csplit ? 4 : 2) : 1;
    for (int c = 0; c < (int)e->chains_h.size(); ++c) {
        ChainDev &d = e->chains_h[c];
        const int nchunk = std::max(1, (d.nt + L - 1) / L);
        d.fused_block0 = (int)e->fused_tasks_h.size();
        d.fused_nblocks = per_chunk * nchunk;
        for (int k = 0; k < nchunk; ++k) {
            const int t0 = (int)((long long)d.nt * k / nchunk);
            const int t1 = (int)((long long)d.nt * (k + 1) / nchunk);
            if (csplit) {
                for (int f = 1; f <= 2; ++f)
                    for (int h = 0; h < 2; ++h)
                        e->fused_tasks_h.push_back({c, t0, t1, 4 * k + 2 * (f - 1) + h, f, h ? 0xC : 0x3});
            } else if (split) {
                e->fused_tasks_h.push_back({c, t0, t1, 2 * k, 1, 0});
                e->fused_tasks_h.push_back({c, t0, t1, 2 * k + 1, 2, 0});
            } else {
                e->fused_tasks_h.push_back({c, t0, t1, k, 0, 0});
            }
        }
    }
}

// Tiled step tasks: 256 consecutive (chunk, site) pairs, chunks of L imaginary times.
void build_tiled_tasks(clv_engine *e, int L) {
    e->chunk = L;
    e->tile_tasks_h.clear();
    for (int c = 0; c < (int)e->chains_h.size(); ++c) {
        ChainDev &d = e->chains_h[c];
        const int nchunk = std::max(1, (d.nt + L - 1) / L);
        const int ntile = (int)(((long long)d.V * nchunk + 255) / 256);
        d.fused_block0 = (int)e->tile_tasks_h.size();
        d.fused_nblocks = ntile;
        for (int t = 0; t < ntile; ++t) e->tile_tasks_h.push_back({c, t * 256, nchunk, t});
    }
}

// Imaginary times per CTA of the step kernels: the chunk length whose CTAs, spread over
// `slots`, finish soonest.  A slot's time is its share of the CTAs times a CTA's length plus
// the halo that every chunk pays, and the share is a whole number: 192 CTAs on 152 SMs cost as
// much as 304 (the FP64 reduce pass on 128 x 128 with chunks of 43: 1.11 ms; of 18: 0.75 ms;
// the FP64 step of 32 chains of 256 x 128 with 320 CTAs: 1.32 ms, with 288: 1.02 ms).  Slots:
// the SMs for the fused kernel, whose resident CTAs share the SM's issue slots; resident CTAs
// for the tiled one, bound by memory or, at one per SM, the FP64 pipe (2D 128 x 128, FP32:
// step kernel 78 us counted in SMs, 70 us).  width: sites a CTA takes of a chunk, 0: all.
int choose_chunk(const clv_engine *e, int slots, int width, double halo) {
    int tmax = 1;
    double work = 0;
    for (auto &d : e->chains_h) {
        tmax = std::max(tmax, d.nt);
        work += width ? (double)d.V * d.nt / width : (double)d.nt;
    }
    int best = 1;
    double cost = 0;
    for (int L = 1; L <= std::min(64, tmax); ++L) {
        long long ctas = 0;
        for (auto &d : e->chains_h) {
            const long long nchunk = (d.nt + L - 1) / L;
            ctas += width ? (d.V * nchunk + width - 1) / width : nchunk;
        }
        const double t = (double)((ctas + slots - 1) / slots) * (work / ctas + halo);
        if (L == 1 || t < cost) {
            best = L;
            cost = t;
        }
    }
    return best;
}

bool tiled_off() {
    const char *env = std::getenv("CLV_TILED");
    return env && env[0] == '0';
}

bool tiled_is_faster(const clv_engine *e, int ln) {
    LineBatch b{};
    b.fp64 = e->precision == CLV_PREC_F64;
    b.ref_rule = e->dt_rule == CLV_DT_REF_MEANMAX;
    b.ln = ln;
    b.sites = e->all_sites;
    for (auto &d : e->chains_h) {
        b.largest = std::max(b.largest, (long long)d.V * d.nt);
        b.slices += d.nt;
    }
    b.field_bytes = e->all_sites * e->ncomp * e->elem_bytes;
    b.num_sms = e->num_sms;
    b.loop_ctas = e->loop_per_sm * e->num_sms;
    size_t room = 0, all = 0;  // (the device's memory; what is free of it decides nothing)
    if (cudaMemGetInfo(&room, &all) != cudaSuccess) return false;
    b.device_bytes = (long long)all;
    return lines_on_the_tiled_path(b);
}

int plan_fused(clv_engine *e) {
    const char *env = std::getenv("CLV_FUSED");
    if (env && env[0] == '0') return CLV_OK;
    const size_t esz = e->elem_bytes;
    int vmax = 0;
    bool aligned = true;
    for (auto &d : e->chains_h) {
        vmax = std::max(vmax, d.V);
        if ((d.V * esz) % 16 != 0) aligned = false;
        if (d.nt < 2) return CLV_OK;
        if ((long long)e->ncomp * d.nt * d.V >= (1LL << 31)) return CLV_OK;  // 32-bit element indices
    }
    // component regions padded (one element per 16) for the FFT's padded layouts,
    // even so that every component row stays 16-byte aligned for the bulk copies
    const int cs = padded_line(vmax);
    const int stride = fused_slot_stride(e->ncomp, vmax, (int)esz);
    // every chain a 1D line of one common length of 64, 128 or 256 sites: other shapes and
    // mixed batches take the tiled path, whose filters work on whole tiles of lines (a warp
    // per line and a thread per site of the batch's largest slice left 64 chains of 60-site
    // lines to 30 x 30 planes at 2.43 ms per step; tiled: 0.13 ms)
    int ln = e->chains_h[0].nx;
    for (auto &d : e->chains_h)
        if (d.ny != 1 || d.nz != 1 || d.nx != ln) ln = 0;
    if (ln != 64 && ln != 128 && ln != 256) return CLV_OK;
    // the step loop's resident CTAs per SM
    int coop = 0;
    CK(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, e->device));
    if (coop && !std::getenv("CLV_NO_STATIC_PLAN")) {
        if (e->precision == CLV_PREC_F64) CK(setup_loop<double>(e->model, ln, &e->loop_per_sm));
        else CK(setup_loop<float>(e->model, ln, &e->loop_per_sm));
    }
    if (!env && !tiled_off() && tiled_is_faster(e, ln)) return CLV_OK;
    if (std::getenv("CLV_NO_STATIC_PLAN")) ln = 0;
    const int tab_n = vmax;  // twiddles and filter of the lines
    const int tab_bytes = fused_tab_bytes(tab_n, (int)esz, ln);
    const int nslots = (e->model == CLV_MODEL_REF4 ? 3 : 2) + 2 + 5;
    const size_t smem = tab_bytes + (size_t)nslots * stride * esz;
    int dev_smem = 0, nsm = 0;
    CK(cudaDeviceGetAttribute(&dev_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, e->device));
    CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, e->device));
    e->num_sms = nsm;
    if (smem + 2048 > (size_t)dev_smem) return CLV_OK;  // room for the kernel's static shared memory
    e->slot_stride = stride;
    e->comp_stride = cs;
    e->fused_smem = smem;
    e->fused_tab_n = tab_n;
    e->fused_tab_bytes = tab_bytes;
    e->fused_ln = ln;
    e->use_tma = aligned && !(std::getenv("CLV_NO_TMA"));
    e->speculate = !(std::getenv("CLV_NO_SPECULATE"));
    LaunchFused probe{};
    probe.model = e->model;
    probe.ln = ln;
    probe.smem_bytes = smem;
    probe.slot_stride = stride;
    int per_sm = 0;
    if (e->precision == CLV_PREC_F64) CK(setup_fused<double>(probe, &per_sm));
    else CK(setup_fused<float>(probe, &per_sm));
    if (per_sm < 1) return CLV_OK;
    e->fused_ctas_per_sm = per_sm;
    // chunk length: the halo of a chunk is the filter of psi(tau0 - 1) and its reads
    long long total_slices = 0;
    for (auto &d : e->chains_h) total_slices += d.nt;
    // (CTAs that share an SM share its issue slots; the FP64 spin-1 form of two CTAs an SM waits
    // on its own latencies, so a wave takes both, and a start costs 1.6 imaginary times)
    const bool two = e->precision == CLV_PREC_F64 && e->model == CLV_MODEL_SPIN1 &&
                     e->dt_rule == CLV_DT_K_OVER_MAX && ln > 0 && per_sm > 1;
    int L = two ? choose_chunk(e, per_sm * nsm, 0, 1.6) : choose_chunk(e, nsm, 0, 0.6);
    if (const char *cl = std::getenv("CLV_CHUNK")) L = std::max(1, atoi(cl));
    e->fused_ln_static = std::getenv("CLV_NO_STATIC_PLAN") ? 0 : ln;
    e->withhold_copy = std::getenv("CLV_TEST_WITHHOLD_COPY") != nullptr;
    // FP64 arithmetic is scarce on this part: store the drift rather than recompute it
    e->store_drift = e->dt_rule == CLV_DT_REF_MEANMAX && e->precision == CLV_PREC_F64;
    if (const char *sd = std::getenv("CLV_STORE_DRIFT"))
        e->store_drift = e->dt_rule == CLV_DT_REF_MEANMAX && sd[0] == '1';
    e->fused_aligned = aligned;
    e->task_capacity = 4 * (size_t)total_slices;  // chunks of one imaginary time, split twice
    e->fused = true;
    build_fused_tasks(e, L);
    return CLV_OK;
}

// The tile-filter group for tiles of `elems` shared elements along axis `a` (0 for whole
// slices): tiles of one size class share a launch, whatever their shapes.
clv_engine::AxisGroup &tile_group(const clv_engine *e, std::vector<clv_engine::AxisGroup> &groups, int a, int n,
                                  bool whole, int elems, size_t smem) {
    const bool wide = elems > (e->elem_bytes == 8 ? tile_wide<float>() : tile_wide<double>());
    const int threads = wide ? 256 : 128;
    for (auto &g : groups)
        if (g.tile && g.axis == a && g.threads == threads) {
            if (g.n != n) g.n = 0;
            g.whole |= whole;
            g.smem = std::max(g.smem, smem);
            return g;
        }
    clv_engine::AxisGroup g{};
    g.axis = a;
    g.n = n;
    g.tile = 1;
    g.whole = whole;
    g.threads = threads;
    g.smem = smem;
    groups.push_back(std::move(g));
    return groups.back();
}

// Lines (slices of a sum) of `sites` taken relative to their first site (kBasedSites).
bool tile_based(const clv_engine *e, bool energy, int sites) {
    return e->precision == CLV_PREC_F64 && sites > kBasedSites && (energy || e->kinetic == CLV_KIN_REF_LINEAR_PX);
}

// tile, twiddles, filters, the rows' shares of summed filters, the groups' scales (FP64:
// five words each, and the first site where the filter vanishes at zero frequency)
size_t tile_smem(const clv_engine *e, int elems, int nsum, int rows, int groups, bool based) {
    return (size_t)(elems + nsum) * e->elem_bytes + (size_t)(nsum + rows) * (e->elem_bytes / 2) +
           (e->precision == CLV_PREC_F64 ? 5 * (size_t)groups * sizeof(unsigned) : 0) +
           (based ? (size_t)groups * sizeof(double2) : 0) + 16;
}

int tile_plan(clv_engine *e, const TileFilterPlan &p) {
    for (int i = 0; i < (int)e->tile_plans_h.size(); ++i)
        if (!std::memcmp(&e->tile_plans_h[i], &p, sizeof p)) return i;
    e->tile_plans_h.push_back(p);
    return (int)e->tile_plans_h.size() - 1;
}

// Slices of chain d per tile: about tile_target elements (one slice when it is larger), lines in
// a number that a phase of a warp's access divides evenly when one is near, with two exceptions.
//   * A problem whose tiles of that size would leave three quarters of the CTAs' places empty
//     takes smaller ones, down to an eighth (8 to 32 sites a side, 13 700 sites: step 21.3 ->
//     17.5 us; below that the launch gets longer again).
//   * Few slices a tile, all chains alike (long lines).  FP32 lines: eight, four or two, whichever
//     first leaves two CTAs an SM and fills the GPU (4 x 1500 x 96: two lines 71 us a step, eight
//     52; 143 chains of 1152: 615, 541 with four, 490; 60 x 960 x 96: 501, 424, 374: the tables
//     of a tile cost as much as a line).  FP64, bound by its passes, and 2D or 3D slices: the
//     fewest elements and table entries to go through in all waves, a tile of 256 threads at
//     twice the pace (FP64, 1536 x 64: one line a tile, 1.1 waves, 149 us; two, one wave, 119 us;
//     6 x 675, 431 -> 410 us; 40 x 720 x 64, two lines 1270 us, eight 1120).
int slices_per_tile(const clv_engine *e, const ChainDev &d, int nsum, int rows1, int cols, bool energy) {
    const bool f64 = e->elem_bytes == 16;
    const int base = f64 ? tile_target<double>() : tile_target<float>();
    const int most = f64 ? tile_slice_max<double>() : tile_slice_max<float>();
    const int wide = f64 ? tile_wide<double>() : tile_wide<float>();
    auto resident = [&](int elems, size_t smem) {
        const int th = elems >= wide ? 256 : 128, by_regs = f64 ? tile_min_ctas<double>(th) : tile_min_ctas<float>(th);
        return std::min(by_regs, std::max(1, (int)((size_t)(228 << 10) / (smem + 1024))));
    };
    const double total = (double)e->all_sites * d.ncomp * (energy ? 1 : 2);  // elements
    bool alike = base / d.V <= (f64 || rows1 > 1 ? 4 : 10);
    for (auto &o : e->chains_h) alike = alike && o.V == d.V && o.axis[0].n == d.axis[0].n && o.axis[1].n == d.axis[1].n;
    if (alike) {
        const int last = std::max(1, std::min(d.nt, most / d.V));
        auto of = [&](int ns, double &tiles) {
            const int elems = ns * rows1 * tile_pitch(e->elem_bytes, cols, ns * rows1);
            tiles = 0;
            for (auto &o : e->chains_h) tiles += (double)d.ncomp * ((o.nt + ns - 1) / ns) * (energy ? 1 : 2);
            return resident(elems, tile_smem(e, elems, nsum, ns * rows1, ns * rows1, tile_based(e, energy, d.V)));
        };
        double tiles = 0;
        if (!f64 && rows1 == 1) {
            for (int ns = 8; ns > 1; ns /= 2)
                if (ns <= last && of(ns, tiles) >= 2 && tiles >= 1.4 * e->num_sms) return ns;
            return 1;
        }
        int best = 1;
        double cost = 0;
        for (int ns = 1; ns <= last; ++ns) {
            const int places = of(ns, tiles) * e->num_sms;
            const bool line = rows1 == 1, full = tiles >= places;
            const double t = std::ceil(tiles / places) * (ns * d.V + (line ? 0.72 : 1.0) * nsum) /
                             (line && ns * d.V >= wide ? (full ? 2 : 1.7) : 1);
            if (ns == 1 || t <= (line && full ? 1.05 : 1) * cost) {
                best = ns;
                cost = ns == 1 ? t : std::min(t, cost);
            }
        }
        return best;
    }
    const double share = total / ((f64 ? 5 : 6) * (double)e->num_sms);
    const int target = share < base / 4 ? std::max(base / 8, (int)share) : base;
    int ns = std::max(1, target / d.V);
    if (rows1 == 1) {
        // lines: a power of two, or a multiple of a phase's lines, when one is near
        const int m = f64 ? 8 : 16;
        int r = ns >= m ? (ns + m / 2) / m * m : ns;
        if (r * d.V * 15 > 16 * target) r = ns / m * m;
        while (r < m && (r & (r - 1))) r &= r - 1;
        if (ns < 2 * m ? 5 * r >= 4 * ns : 10 * r >= 9 * ns) ns = r;
    }
    return std::min(d.nt, ns);
}

// Whole slices of chain c: tiles of consecutive imaginary times of one component.
int add_tile_slices(clv_engine *e, int c, bool energy, std::vector<clv_engine::AxisGroup> &groups) {
    const ChainDev &d = e->chains_h[c];
    int last = 0;
    for (int a = 1; a < 3; ++a)
        if (d.axis[a].n > 1) last = a;
    TileFilterPlan p;
    std::memset(&p, 0, sizeof p);
    const int cols = d.axis[last].n, rows1 = d.V / cols;
    int nsum = 0;
    for (int a = 0; a <= last; ++a) {
        if (d.axis[a].n <= 1) continue;
        if (!energy && e->kinetic == CLV_KIN_REF_LINEAR_PX && a > 0) break;
        if (!d.axis[a].tnf) return fail(CLV_ERR_STATE, "tile filter plan");
        p.axis[p.naxes] = a;
        p.inner[p.naxes++] = d.axis[a].inner;
        nsum += d.axis[a].n;
    }
    p.with_const = !energy && e->kinetic == CLV_KIN_EXP;
    p.based = tile_based(e, energy, p.naxes == 1 ? d.axis[p.axis[0]].n : d.V);
    const int ns = slices_per_tile(e, d, nsum, rows1, cols, energy);
    p.pitch = tile_pitch(e->elem_bytes, cols, ns * rows1);
    p.tile_elems = (ns * rows1 * p.pitch + 1) / 2 * 2;
    const int id = tile_plan(e, p);
    auto &g = tile_group(e, groups, 0, p.naxes == 1 ? d.axis[p.axis[0]].n : 0, p.naxes > 1, p.tile_elems,
                         tile_smem(e, p.tile_elems, nsum, ns * rows1,
                                   p.naxes == 1 ? ns * d.V / d.axis[p.axis[0]].n : ns, p.based));
    for (int k = 0; k < d.ncomp; ++k)
        for (int t = 0; t < d.nt; t += ns)
            g.ttasks.push_back({c, id, k * d.nt + t, 0, std::min(ns, d.nt - t) * rows1, cols});
    return CLV_OK;
}

// Tiles of lines of axis a of chain c: a strided axis in tiles of adjacent lines (16-line
// multiples keep the rows' 128-byte segments), the innermost one in tiles of whole lines.
int add_tile_axis(clv_engine *e, int c, int a, bool energy, std::vector<clv_engine::AxisGroup> &groups) {
    const ChainDev &d = e->chains_h[c];
    const AxisDev &ax = d.axis[a];
    if (!ax.tnf) return fail(CLV_ERR_STATE, "tile filter plan");
    const int n = ax.n, lines = d.V / n;
    const int target = e->elem_bytes == 8 ? tile_target<float>() : tile_target<double>();
    TileFilterPlan p;
    std::memset(&p, 0, sizeof p);
    p.naxes = 1;
    p.axis[0] = a;
    p.with_const = !energy && e->kinetic == CLV_KIN_EXP && a == 0;
    p.based = tile_based(e, energy, n);
    if (ax.inner > 1) {
        int W = target / n;
        W = W >= 16 ? W / 16 * 16 : (W >= 8 ? 8 : 4);
        W = std::min(W, ax.inner);
        p.inner[0] = 0;
        p.pitch = W | 1;
        p.gstride = ax.inner;
        p.tile_elems = (n * p.pitch + 1) / 2 * 2;
        const int id = tile_plan(e, p);
        auto &g = tile_group(e, groups, a, n, false, p.tile_elems, tile_smem(e, p.tile_elems, n, 0, W, p.based));
        for (int sl = 0; sl < d.ncomp * d.nt; ++sl)
            for (int hi = 0; hi < lines / ax.inner; ++hi)
                for (int l = 0; l < ax.inner; l += W)
                    g.ttasks.push_back({c, id, sl, hi * n * ax.inner + l, n, std::min(W, ax.inner - l)});
    } else {
        const int W = std::max(1, std::min(lines, target / n));
        p.inner[0] = 1;
        p.pitch = tile_pitch(e->elem_bytes, n, W);
        p.tile_elems = (W * p.pitch + 1) / 2 * 2;
        const int id = tile_plan(e, p);
        auto &g = tile_group(e, groups, a, n, false, p.tile_elems, tile_smem(e, p.tile_elems, n, 0, W, p.based));
        for (int sl = 0; sl < d.ncomp * d.nt; ++sl)
            for (int l = 0; l < lines; l += W)
                g.ttasks.push_back({c, id, sl, l * n, std::min(W, lines - l), n});
    }
    return CLV_OK;
}

// Axis-filter launch groups, one per (axis, line length): kinetic (energy =
// false: the step's filter, every filtered axis, the component constant on the
// first) or kinetic energy (energy = true: k_a^2/2 on every axis, summed).  Square planes
// of 32 to 128 (kinetic) take the plane filter; other slices of up to tile_slice_max sites
// the tile filter with every axis on chip; the axes of larger slices the axis filter where
// it has their length, else the tile filter.  *ok false when a tile does not fit shared
// memory.
int build_axis_groups(clv_engine *e, bool energy, std::vector<clv_engine::AxisGroup> &groups, bool &ok) {
    ok = false;
    groups.clear();
    const size_t esz = e->elem_bytes;
    int dev_smem = 0;
    CK(cudaDeviceGetAttribute(&dev_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, e->device));
    for (int c = 0; c < (int)e->chains_h.size(); ++c) {
        const ChainDev &d = e->chains_h[c];
        // square planes of side 32 to 128 (a 2D slice, or the (y, z) planes of a 3D
        // slice) under the exponential kinetic factor, a product over the axes: one
        // plane-filter launch instead of two axis launches
        int pa = -1, occ = 0;
        if ((energy || e->kinetic == CLV_KIN_EXP) && !std::getenv("CLV_NO_PLANE")) {
            const int n1 = d.axis[1].n, n2 = d.axis[2].n;
            pa = n2 <= 1 ? (d.axis[0].n == n1 ? 0 : -1) : (n1 == n2 ? 1 : -1);
            const int pn = pa >= 0 ? d.axis[pa].n : 0;
            if (pn == 32 || pn == 64 || pn == 96 || pn == 128) {
                const size_t sm = plane_smem_bytes(pn, esz);
                if (sm + 1024 <= (size_t)dev_smem) {
                    if (e->precision == CLV_PREC_F64) CK(setup_plane_filter<double>(pn, energy, sm, &occ));
                    else CK(setup_plane_filter<float>(pn, energy, sm, &occ));
                }
            }
            if (occ < 1) pa = -1;
        }
        // other small slices: every filtered axis while the slice is on chip
        if (pa < 0 && d.V <= (esz == 8 ? tile_slice_max<float>() : tile_slice_max<double>())) {
            if (int rc = add_tile_slices(e, c, energy, groups)) return rc;
            continue;
        }
        for (int a = 0; a < 3; ++a) {
            const AxisDev &ax = d.axis[a];
            if (ax.n <= 1) continue;
            if (!energy && e->kinetic == CLV_KIN_REF_LINEAR_PX && a > 0) break;
            if (pa >= 0 && a == pa + 1) continue;  // filtered with axis pa
            if (pa >= 0 && a == pa) {
                const int n = ax.n;
                int gi = -1;
                for (int g = 0; g < (int)groups.size(); ++g)
                    if (groups[g].plane && groups[g].axis == a && groups[g].n == n) gi = g;
                if (gi < 0) {
                    clv_engine::AxisGroup g;
                    g.axis = a;
                    g.n = n;
                    g.pitch = plane_pitch(n);
                    g.W = 1;
                    g.plane = 1;
                    g.resident = occ * e->num_sms;
                    g.with_const = !energy && a == 0;
                    g.smem = plane_smem_bytes(n, esz);
                    groups.push_back(std::move(g));
                    gi = (int)groups.size() - 1;
                }
                const int planes = d.V / (n * n);
                for (int sl = 0; sl < d.ncomp * d.nt; ++sl)
                    for (int x = 0; x < planes; ++x) groups[gi].tasks.push_back({c, sl, x, 1});
                continue;
            }
            const int n = ax.n, lines = d.V / n;
            // (FP64 always: the tile filter's integer lines against butterflies bound by the FP64
            // pipe, k_tile.cuh)
            if (esz == 16 || !axis_compile_time_plan(n)) {
                if (int rc = add_tile_axis(e, c, a, energy, groups)) return rc;
                continue;
            }
            const int W = axis_tile_lines(n);
            int gi = -1;
            for (int g = 0; g < (int)groups.size(); ++g)
                if (!groups[g].plane && !groups[g].tile && groups[g].axis == a && groups[g].n == n) gi = g;
            if (gi < 0) {
                clv_engine::AxisGroup g;
                g.axis = a;
                g.n = n;
                g.pitch = axis_pitch(n);
                g.W = W;
                g.with_const = !energy && e->kinetic == CLV_KIN_EXP && a == 0;
                g.smem = axis_smem_bytes(n, W, esz);
                if (g.smem + 1024 > (size_t)dev_smem) return CLV_OK;
                int occ = 0;
                CK(setup_axis_filter<float>(n, g.smem, &occ));
                if (occ < 1) return CLV_OK;
                groups.push_back(std::move(g));
                gi = (int)groups.size() - 1;
            }
            groups[gi].strided &= ax.inner > 1;
            if (ax.inner == 1 && !groups[gi].with_const) {
                // contiguous lines run on across slices: tiles of W consecutive lines of
                // the chain (1D chains: W imaginary-time slices per tile)
                const int total = d.ncomp * d.nt * lines;
                for (int gl = 0; gl < total; gl += W)
                    groups[gi].tasks.push_back({c, gl / lines, gl % lines, std::min(W, total - gl)});
            } else {
                // tiles of W lines of one slice, never across an outer block of a strided axis
                for (int sl = 0; sl < d.ncomp * d.nt; ++sl)
                    for (int l0 = 0; l0 < lines;) {
                        const int nl = ax.inner == 1 ? std::min(W, lines - l0)
                                                     : std::min(W, ax.inner - l0 % ax.inner);
                        groups[gi].tasks.push_back({c, sl, l0, nl});
                        l0 += nl;
                    }
            }
        }
    }
    for (auto &g : groups)
        if (g.tile) {
            int occ = 0;
            if (e->precision == CLV_PREC_F64) CK(setup_tile_filter<double>(g.smem, g.threads, &occ));
            else CK(setup_tile_filter<float>(g.smem, g.threads, &occ));
            if (occ < 1) return CLV_OK;
        }
    std::stable_sort(groups.begin(), groups.end(),
                     [](const clv_engine::AxisGroup &x, const clv_engine::AxisGroup &y) { return x.axis < y.axis; });
    ok = true;
    return CLV_OK;
}

int plan_tiled(clv_engine *e) {
    if (e->fused) return CLV_OK;
    const char *env = std::getenv("CLV_TILED");
    if (env && env[0] == '0') return CLV_OK;
    int nsm = 0;
    CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, e->device));
    std::vector<clv_engine::AxisGroup> groups;
    bool ok = false, longer = false;
    if (int rc = build_axis_groups(e, false, groups, ok)) return rc;
    if (!ok) return CLV_OK;
    for (auto &d : e->chains_h) {
        if (d.nt < 2) longer = true;
        for (int a = 0; a < 3; ++a)
            longer |= d.axis[a].n > kTiledMaxLine && !(a > 0 && e->kinetic == CLV_KIN_REF_LINEAR_PX);
    }
    if (longer) {
        e->axis_groups = std::move(groups);
        return CLV_OK;
    }
    // reference rule at FP64, where arithmetic is scarce: the reduce pass stores the drift
    // and the update applies it, instead of a second drift pass; at FP32 in problems bound by
    // latencies, whose update starts on its noise beside the pass (11 chains of 64 sites, 21 800
    // sites: 23 -> 21.5 us a step; 0.43 M sites 68 -> 74, which keep the second pass)
    e->store_drift = e->dt_rule == CLV_DT_REF_MEANMAX &&
                     (e->precision == CLV_PREC_F64 || e->all_sites < 2LL * 256 * nsm);
    if (const char *sd = std::getenv("CLV_STORE_DRIFT"))
        e->store_drift = e->dt_rule == CLV_DT_REF_MEANMAX && sd[0] == '1';
    // Where that pass fills the GPU for a while it is bound by the FP64 pipe, so it also draws
    // the normals (integer pipes) into the buffer that the update overwrites: 128 x 128 x 128,
    // reduce 754 -> 783 us and update 397 -> 190 us.  A short one is bound by latencies, and the
    // update draws them beside it (160 000 sites, 4 blocks an SM: 186 us a step, 200 drawn here).
    // A step kernel that draws beside its drift takes the same two CTAs an SM from 8 blocks on
    // (0.57 M sites, 14: 301 -> 229 us; 0.096 M, 2: 57 us, 70 in that form).
    const long long blocks = e->all_sites / 256;
    e->draw_in_reduce = e->store_drift && e->precision == CLV_PREC_F64 && blocks >= 16LL * nsm;
    e->tiled_lean = e->precision == CLV_PREC_F64 && blocks >= 8LL * nsm;
    int occ = 0;
    if (e->precision == CLV_PREC_F64) CK(setup_tiled<double>(e->model, e->tiled_lean, e->draw_in_reduce, &occ));
    else CK(setup_tiled<float>(e->model, 0, 0, &occ));
    if (occ < 1) return CLV_OK;
    // chunk length: the halo of a chunk is the reads of one imaginary time, which the FP32
    // kernel, bound by memory, pays in full (3D 64^3: 1.04 ms with 16 times a chunk, 1.00 with 64)
    long long tile_taus = 0;
    for (auto &d : e->chains_h) tile_taus += ((long long)d.V * d.nt + 255) / 256;
    // (a reduce pass bound by the FP64 pipe: CTAs that share an SM share its pipe, and the halo
    // costs it one density)
    int L = e->draw_in_reduce ? choose_chunk(e, nsm, 256, 0.15)
                              : choose_chunk(e, occ * nsm, 256, e->precision == CLV_PREC_F32 ? 2.0 : 0.6);
    if (const char *cl = std::getenv("CLV_CHUNK")) L = std::max(1, atoi(cl));
    e->task_capacity = (size_t)tile_taus;  // chunks of one imaginary time
    build_tiled_tasks(e, L);
    e->axis_groups = std::move(groups);
    e->speculate = !(std::getenv("CLV_NO_SPECULATE"));
    e->tiled = true;
    return CLV_OK;
}

// The windows of the tiled path: one, or, without an array for kinbar, runs of chains whose
// elements kin holds twice.  False when a chain alone is too large for that.
bool plan_windows(clv_engine *e, bool split) {
    e->windows.clear();
    const int nch = (int)e->chains_h.size();
    const long long most = split ? e->total_elems / 2 : e->total_elems;
    for (int c = 0; c < nch;) {
        clv_engine::Window w{};
        w.c0 = c;
        w.off = e->chains_h[c].off;
        for (; c < nch; ++c) {
            const ChainDev &d = e->chains_h[c];
            const long long elems = d.off + (long long)d.ncomp * d.nt * d.V - w.off;
            if (elems > most) break;
            w.elems = elems;
        }
        if (c == w.c0) {
            e->windows.clear();
            return false;
        }
        w.c1 = c;
        for (const auto &g : e->axis_groups) {  // (tasks are in the order of chains)
            int first = 0;
            while (first < g.ntasks() && g.chain_of(first) < w.c0) ++first;
            int end = first;
            while (end < g.ntasks() && g.chain_of(end) < w.c1) ++end;
            w.groups.push_back({first, end - first});
        }
        e->windows.push_back(std::move(w));
    }
    return true;
}

// Memory for a call of an engine under way; the tiled path gives kinbar's back for it where there
// is no other.
cudaError_t malloc_beside(clv_engine *e, void **p, size_t bytes) {
    const char *test = std::getenv("CLV_TEST_NO_KINBAR");
    cudaError_t ce = test && test[0] == '2' && e->kinc ? cudaErrorMemoryAllocation : cudaMalloc(p, bytes);
    if (ce != cudaErrorMemoryAllocation || !e->tiled || !e->kinc) return ce;
    cudaGetLastError();
    if (!plan_windows(e, true)) {
        plan_windows(e, false);
        return ce;
    }
    e->drop_graphs();
    if ((ce = cudaStreamSynchronize(e->stream)) != cudaSuccess) return ce;
    e->release(&e->kinc, (size_t)e->total_elems * e->elem_bytes);
    return cudaMalloc(p, bytes);
}

int check_chain(clv_engine *e, int chain) {
    if (!e) return fail(CLV_ERR_ARG, "null engine");
    if (chain < 0 || chain >= (int)e->params.size()) return fail(CLV_ERR_ARG, "chain out of range");
    return CLV_OK;
}

cudaMemcpyKind kind_of(int where, bool to_device) {
    if (where & CLV_DEVICE) return cudaMemcpyDeviceToDevice;
    return to_device ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost;
}

}  // namespace

extern "C" {

int clv_version(void) { return CLV_API_VERSION; }

const char *clv_last_error(void) { return g_last_error.c_str(); }

const char *clv_status_string(int s) {
    switch (s) {
        case CLV_OK: return "ok";
        case CLV_ERR_ARG: return "invalid argument";
        case CLV_ERR_CUDA: return "CUDA error";
        case CLV_ERR_NONFINITE: return "non-finite drift";
        case CLV_ERR_TIMEOUT: return "device wait timed out";
        case CLV_ERR_STATE: return "invalid state";
        case CLV_ERR_NOMEM: return "out of memory";
        case CLV_ERR_IO: return "i/o error";
        default: return "unknown status";
    }
}

void clv_default_chain_params(clv_chain_params *p) {
    std::memset(p, 0, sizeof *p);
    // Parameters.h
    p->nx = 256; p->ny = 1; p->nz = 1; p->nt = 32;
    p->eps = 0.01; p->a_x = 1.0; p->G = 0.1; p->Q = 0.0; p->DT = 0.002;
    // compute_new_dt (Propagator_without_cutoff.cu:391-402)
    p->dt_min = 1e-8; p->dt_max_clamp = 0.01; p->alpha = 0.9;
    // params.txt
    p->mu = -1.5; p->P = 0.0; p->seed = 7342951900870119ull;
    p->c0 = 0.5; p->c1 = -0.1; p->q = 0.05; p->K = 0.05; p->dt_max = 1e-3;
}

int clv_create(const clv_config *cfg, clv_engine **out) {
    if (!cfg || !out) return fail(CLV_ERR_ARG, "null argument");
    *out = nullptr;
    if (cfg->nchains <= 0 || !cfg->chains) return fail(CLV_ERR_ARG, "nchains must be positive");
    if (cfg->model != CLV_MODEL_REF4 && cfg->model != CLV_MODEL_SPIN1)
        return fail(CLV_ERR_ARG, "unknown model");
    if (cfg->kinetic != CLV_KIN_REF_LINEAR_PX && cfg->kinetic != CLV_KIN_EXP)
        return fail(CLV_ERR_ARG, "unknown kinetic term");
    if (cfg->dt_rule != CLV_DT_REF_MEANMAX && cfg->dt_rule != CLV_DT_K_OVER_MAX)
        return fail(CLV_ERR_ARG, "unknown step rule");
    if (cfg->noise != CLV_NOISE_EXTERNAL && cfg->noise != CLV_NOISE_PHILOX)
        return fail(CLV_ERR_ARG, "unknown noise source");
    if (cfg->precision != CLV_PREC_F64 && cfg->precision != CLV_PREC_F32)
        return fail(CLV_ERR_ARG, "unknown precision");
    long long total_sites = 0;
    for (int c = 0; c < cfg->nchains; ++c) {
        const clv_chain_params &p = cfg->chains[c];
        if (p.nx < 2 || p.ny < 1 || p.nz < 1 || p.nt < 2)
            return fail(CLV_ERR_ARG, "chain " + std::to_string(c) + ": need nx >= 2, nt >= 2");
        const long long sites = (long long)p.nx * p.ny * p.nz * p.nt;
        const int ncomp = cfg->model == CLV_MODEL_REF4 ? 4 : 3;
        if (sites * ncomp >= (1ll << 31))
            return fail(CLV_ERR_ARG, "chain " + std::to_string(c) + ": lattice too large");
        if (!(p.eps > 0) || !std::isfinite(p.eps)) return fail(CLV_ERR_ARG, "eps must be positive");
        if (cfg->model == CLV_MODEL_REF4 && !(p.a_x != 0)) return fail(CLV_ERR_ARG, "a_x must be nonzero");
        total_sites += sites;
    }
    if (total_sites >= (1ll << 40)) return fail(CLV_ERR_ARG, "batch too large");
    CK(cudaSetDevice(cfg->device));
    int nsm = 0;
    CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, cfg->device));
    clv_engine *e = new clv_engine();
    e->device = cfg->device;
    e->num_sms = nsm;
    e->model = cfg->model;
    e->kinetic = cfg->kinetic;
    e->dt_rule = cfg->dt_rule;
    e->noise = cfg->noise;
    e->precision = cfg->precision;
    e->ncomp = cfg->model == CLV_MODEL_REF4 ? 4 : 3;
    e->elem_bytes = cfg->precision == CLV_PREC_F64 ? 16 : 8;
    e->params.assign(cfg->chains, cfg->chains + cfg->nchains);
    if (const char *cap = std::getenv("CLV_SAMPLE_CAPACITY")) e->sample_cap = std::max(1, atoi(cap));
    auto bail = [&](int rc) { clv_destroy(e); return rc; };
    cudaError_t ce = cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking);
    if (ce != cudaSuccess) return bail(fail(CLV_ERR_CUDA, cudaGetErrorString(ce)));
    e->own_stream = true;
    ce = setup_line_filter();
    if (ce != cudaSuccess) return bail(fail(CLV_ERR_CUDA, cudaGetErrorString(ce)));
    int rc = build_tables(e);
    if (rc) return bail(rc);
    if ((rc = plan_fused(e))) return bail(rc);
    if ((rc = plan_tiled(e))) return bail(rc);

    if (e->model == CLV_MODEL_SPIN1 && !(std::getenv("CLV_TILED") && std::getenv("CLV_TILED")[0] == '0')) {
        bool ok = false;
        if ((rc = build_axis_groups(e, true, e->energy_groups, ok))) return bail(rc);
        e->energy_axis = ok;
        if (!ok) e->energy_groups.clear();
    }
    const size_t fb = e->total_elems * e->elem_bytes;
    const size_t fb_scratch = e->fused ? 16 : fb;  // the fused path needs no kinetic/drift arrays
    // drift arrays: the separate-kernel path, and the fused and tiled two-pass paths when they
    // store the drift
    const size_t fb_drift =
        ((e->fused && e->dt_rule != CLV_DT_REF_MEANMAX) || (e->tiled && !e->store_drift)) ? 16 : fb;
    const size_t nparts = std::max<size_t>(1, e->task_capacity);
    const int nch = cfg->nchains;
    if ((rc = e->alloc(&e->fld[0][0], fb)) || (rc = e->alloc(&e->fld[0][1], fb)) ||
        (rc = e->alloc(&e->fld[1][0], fb)) || (rc = e->alloc(&e->fld[1][1], fb)) ||
        (rc = e->alloc(&e->kin, fb)) || (!e->tiled && (rc = e->alloc(&e->kinc, fb_scratch))) ||
        (rc = e->alloc(&e->drift, fb_drift)) || (rc = e->alloc(&e->driftc, fb_drift)) ||
        (rc = e->alloc(&e->fused_tasks, (e->fused ? nparts : 1) * sizeof(FusedTask))) ||
        (rc = e->alloc(&e->fused_partials, (e->loop_per_sm > 0 ? 2 : 1) * nparts * sizeof(double2))) ||
        (rc = e->alloc(&e->tile_tasks, (e->tiled ? nparts : 1) * sizeof(TileTask))) ||
        (rc = e->alloc(&e->stage, 2 * e->max_chain_elems * sizeof(double2))) ||
        (rc = e->alloc(&e->chains_d, nch * sizeof(ChainDev))) ||
        (rc = e->alloc(&e->state_d, nch * sizeof(ChainState))) ||
        (rc = e->alloc(&e->site_tasks, e->site_tasks_h.size() * sizeof(SiteTask))) ||
        (rc = e->alloc(&e->obs_tasks, e->obs_tasks_h.size() * sizeof(SiteTask))) ||
        (rc = e->alloc(&e->partials, e->site_tasks_h.size() * sizeof(double2))) ||
        (rc = e->alloc(&e->obs_pairs, e->obs_pairs_h.size() * sizeof(ObsTask))) ||
        (rc = e->alloc(&e->obs_partials, e->obs_pairs_h.size() * 8 * sizeof(double))) ||
        (rc = e->alloc(&e->obs_scratch, e->model == CLV_MODEL_REF4 ? e->obs_scratch_n * sizeof(double) : 0)) ||
        (rc = e->alloc(&e->obs_arrive, nch * sizeof(unsigned int))) ||
        (rc = e->alloc(&e->accF, std::max(1, e->acc_F_total) * sizeof(double))) ||
        (rc = e->alloc(&e->accN, nch * 5 * sizeof(double))) ||
        (rc = e->alloc(&e->samples, (size_t)e->sample_cap * nch * 8 * sizeof(double))) ||
        (rc = e->alloc(&e->loop_sync, (e->loop_per_sm > 0 ? 2 * nparts + 1 : 1) * sizeof(unsigned int))))
        return bail(rc);
    {
        // the step loop's normals: for problems whose split tasks of one imaginary time
        // can all be resident at once (the only ones the loop takes)
        long long slices = 0;
        for (auto &d : e->chains_h) slices += d.nt;
        if (e->fused && e->fused_ln > 0 && e->loop_per_sm > 0 &&
            2 * slices <= (long long)e->loop_per_sm * e->num_sms && (rc = e->alloc(&e->loop_noise, fb)))
            return bail(rc);
    }
    for (int a = 0; a < 3; ++a)
        if (!e->line_tasks_h[a].empty() &&
            (rc = e->alloc(&e->line_tasks[a], e->line_tasks_h[a].size() * sizeof(LineTask))))
            return bail(rc);
    for (auto *gs : {&e->axis_groups, &e->energy_groups})
        for (auto &g : *gs)
            if ((rc = g.tile ? e->alloc(&g.td, g.ttasks.size() * sizeof(TileFilterTask))
                             : e->alloc(&g.d, g.tasks.size() * sizeof(AxisTask))))
                return bail(rc);
    if ((rc = e->alloc(&e->tile_plans, e->tile_plans_h.size() * sizeof(TileFilterPlan)))) return bail(rc);
    if (e->tiled) {
        // A batch that leaves no memory for kinbar steps its chains in windows, with the same bits:
        // the memory of a step that keeps no kinetic terms but the observables' (5 field arrays
        // for spin-1, 7 for the reference model at FP64).  Where one chain holds more than half of
        // the elements the stored drift gives its two arrays, also with the same bits.
        const char *test = std::getenv("CLV_TEST_NO_KINBAR");  // as if its allocation failed: 1 here, 2 later
        rc = test && test[0] == '1' ? fail(CLV_ERR_NOMEM, "kinbar withheld by a test") : e->alloc(&e->kinc, fb);
        cudaGetLastError();  // (a refused allocation is no error of a later launch)
        if (rc && !plan_windows(e, true) && e->store_drift) {
            e->release(&e->drift, fb);
            e->release(&e->driftc, fb);
            e->store_drift = e->draw_in_reduce = false;
            rc = e->alloc(&e->kinc, fb);
        }
        if (!rc) plan_windows(e, false);
        else if (e->windows.empty()) return bail(rc);
    }
    auto up = [&](void *d, const void *h, size_t b) {
        return cudaMemcpy(d, h, b, cudaMemcpyHostToDevice);
    };
    if (e->fused &&
        (ce = up(e->fused_tasks, e->fused_tasks_h.data(), e->fused_tasks_h.size() * sizeof(FusedTask))) != cudaSuccess)
        return bail(fail(CLV_ERR_CUDA, cudaGetErrorString(ce)));
    if (e->tiled &&
        (ce = up(e->tile_tasks, e->tile_tasks_h.data(), e->tile_tasks_h.size() * sizeof(TileTask))) != cudaSuccess)
        return bail(fail(CLV_ERR_CUDA, cudaGetErrorString(ce)));
    for (auto *gs : {&e->axis_groups, &e->energy_groups})
        for (auto &g : *gs)
            if ((ce = g.tile ? up(g.td, g.ttasks.data(), g.ttasks.size() * sizeof(TileFilterTask))
                             : up(g.d, g.tasks.data(), g.tasks.size() * sizeof(AxisTask))) != cudaSuccess)
                return bail(fail(CLV_ERR_CUDA, cudaGetErrorString(ce)));
    if ((ce = up(e->tile_plans, e->tile_plans_h.data(), e->tile_plans_h.size() * sizeof(TileFilterPlan))) != cudaSuccess)
        return bail(fail(CLV_ERR_CUDA, cudaGetErrorString(ce)));
    if ((ce = up(e->chains_d, e->chains_h.data(), nch * sizeof(ChainDev))) != cudaSuccess ||
        (ce = up(e->site_tasks, e->site_tasks_h.data(), e->site_tasks_h.size() * sizeof(SiteTask))) != cudaSuccess ||
        (ce = up(e->obs_tasks, e->obs_tasks_h.data(), e->obs_tasks_h.size() * sizeof(SiteTask))) != cudaSuccess ||
        (ce = up(e->obs_pairs, e->obs_pairs_h.data(), e->obs_pairs_h.size() * sizeof(ObsTask))) != cudaSuccess ||
        (ce = cudaMemset(e->obs_arrive, 0, nch * sizeof(unsigned int))) != cudaSuccess)
        return bail(fail(CLV_ERR_CUDA, cudaGetErrorString(ce)));
    for (int a = 0; a < 3; ++a)
        if (!e->line_tasks_h[a].empty() &&
            (ce = up(e->line_tasks[a], e->line_tasks_h[a].data(),
                     e->line_tasks_h[a].size() * sizeof(LineTask))) != cudaSuccess)
            return bail(fail(CLV_ERR_CUDA, cudaGetErrorString(ce)));
    std::vector<ChainState> st(nch);
    std::memset(st.data(), 0, nch * sizeof(ChainState));
    for (int c = 0; c < nch; ++c) {
        st[c].dt = e->model == CLV_MODEL_REF4 ? e->params[c].DT : e->params[c].dt_max;
    }
    if ((ce = up(e->state_d, st.data(), nch * sizeof(ChainState))) != cudaSuccess)
        return bail(fail(CLV_ERR_CUDA, cudaGetErrorString(ce)));
    const size_t fbz = e->total_elems * e->elem_bytes;
    if ((ce = cudaMemset(e->fld[0][0], 0, fbz)) != cudaSuccess || (ce = cudaMemset(e->fld[0][1], 0, fbz)) != cudaSuccess ||
        (ce = cudaMemset(e->fld[1][0], 0, fbz)) != cudaSuccess || (ce = cudaMemset(e->fld[1][1], 0, fbz)) != cudaSuccess ||
        (ce = cudaMemset(e->accF, 0, std::max(1, e->acc_F_total) * sizeof(double))) != cudaSuccess ||
        (ce = cudaMemset(e->accN, 0, nch * 5 * sizeof(double))) != cudaSuccess ||
        (ce = cudaMemset(e->samples, 0, (size_t)e->sample_cap * nch * 8 * sizeof(double))) != cudaSuccess)
        return bail(fail(CLV_ERR_CUDA, cudaGetErrorString(ce)));
    *out = e;
    return CLV_OK;
}

int clv_destroy(clv_engine *e) {
    if (!e) return CLV_OK;
    cudaSetDevice(e->device);
    if (e->stream) cudaStreamSynchronize(e->stream);
    e->drop_graphs();
    for (void *p : e->allocs) cudaFree(p);
    if (e->noise_d) cudaFree(e->noise_d);
    if (e->stage_all) cudaFree(e->stage_all);
    if (e->own_stream && e->stream) cudaStreamDestroy(e->stream);
    delete e;
    return CLV_OK;
}

int clv_set_stream(clv_engine *e, void *stream) {
    if (!e) return fail(CLV_ERR_ARG, "null engine");
    CK(cudaSetDevice(e->device));
    CK(cudaStreamSynchronize(e->stream));
    if (e->own_stream) cudaStreamDestroy(e->stream);
    e->stream = (cudaStream_t)stream;
    e->own_stream = false;
    e->drop_graphs();
    return CLV_OK;
}

int clv_synchronize(clv_engine *e) {
    if (!e) return fail(CLV_ERR_ARG, "null engine");
    CK(cudaSetDevice(e->device));
    CK(cudaStreamSynchronize(e->stream));
    return CLV_OK;
}

// Copies between the boundary layout (complex128) and the engine's buffers for
// chains [c0, c1), whose boundary arrays are concatenated in chain order.  The
// chains are contiguous in the engine's buffers too, so every field moves with
// one copy (and, at FP32, one conversion kernel) through a staging buffer sized
// for the range, allocated on first use.
static int copy_fields(clv_engine *e, int c0, int c1, const void *const src_in[2],
                       void *const dst_in[2], int where, bool to_engine) {
    const long long off = e->chains_h[c0].off;
    const ChainDev &last = e->chains_h[c1 - 1];
    const long long n = last.off + (long long)e->ncomp * last.nt * last.V - off;
    // complex64 boundary buffers (CLV_C64): moved as they are at FP32, converted
    // through the staging buffer at FP64; complex128 the other way round
    const bool c64 = (where & CLV_C64) != 0;
    const size_t ub = c64 ? 8 : 16;  // bytes per element of the caller's buffers
    const bool direct = c64 == (e->precision != CLV_PREC_F64);
    double2 *stage = e->stage;
    if (!direct && n > e->max_chain_elems) {
        if (e->stage_all_elems < n) {
            if (e->stage_all) cudaFree(e->stage_all);
            e->stage_all = nullptr;
            e->stage_all_elems = 0;
            void *q = nullptr;
            CK(malloc_beside(e, &q, n * sizeof(double2)));
            e->stage_all = (double2 *)q;
            e->stage_all_elems = n;
        }
        stage = e->stage_all;
    }
    for (int f = 0; f < 2; ++f) {
        char *eng = (char *)e->fld[e->cur][f] + off * e->elem_bytes;
        if (to_engine) {
            if (!src_in[f]) continue;
            if (direct) {
                CK(cudaMemcpyAsync(eng, src_in[f], n * ub, kind_of(where, true), e->stream));
            } else {
                CK(cudaMemcpyAsync(stage, src_in[f], n * ub, kind_of(where, true), e->stream));
                if (c64) CK(launch_export<float>((double2 *)eng, stage, n, e->stream));
                else CK(launch_import<float>(eng, stage, n, e->stream));
            }
        } else {
            if (!dst_in[f]) continue;
            if (direct) {
                CK(cudaMemcpyAsync(dst_in[f], eng, n * ub, kind_of(where, false), e->stream));
            } else {
                if (c64) CK(launch_import<float>(stage, (const double2 *)eng, n, e->stream));
                else CK(launch_export<float>(stage, eng, n, e->stream));
                CK(cudaMemcpyAsync(dst_in[f], stage, n * ub, kind_of(where, false), e->stream));
            }
        }
    }
    if (!(where & CLV_ASYNC)) CK(cudaStreamSynchronize(e->stream));
    return CLV_OK;
}

int clv_set_fields(clv_engine *e, int chain, const void *psi, const void *psic, int where) {
    if (!e) return fail(CLV_ERR_ARG, "null engine");
    if (where & ~(CLV_DEVICE | CLV_C64 | CLV_ASYNC))
        return fail(CLV_ERR_ARG, "where: CLV_HOST or CLV_DEVICE, optionally | CLV_C64 | CLV_ASYNC");
    if (chain != -1) {
        int rc = check_chain(e, chain);
        if (rc) return rc;
    }
    CK(cudaSetDevice(e->device));
    const void *src[2] = {psi, psic};
    void *const dst[2] = {nullptr, nullptr};
    return chain == -1 ? copy_fields(e, 0, (int)e->params.size(), src, dst, where, true)
                       : copy_fields(e, chain, chain + 1, src, dst, where, true);
}

int clv_get_fields(clv_engine *e, int chain, void *psi, void *psic, int where) {
    if (!e) return fail(CLV_ERR_ARG, "null engine");
    if (where & ~(CLV_DEVICE | CLV_C64 | CLV_ASYNC))
        return fail(CLV_ERR_ARG, "where: CLV_HOST or CLV_DEVICE, optionally | CLV_C64 | CLV_ASYNC");
    if (chain != -1) {
        int rc = check_chain(e, chain);
        if (rc) return rc;
    }
    CK(cudaSetDevice(e->device));
    const void *const src[2] = {nullptr, nullptr};
    void *dst[2] = {psi, psic};
    return chain == -1 ? copy_fields(e, 0, (int)e->params.size(), src, dst, where, false)
                       : copy_fields(e, chain, chain + 1, src, dst, where, false);
}

int clv_set_mean_field(clv_engine *e, int field, double re, double im) {
    if (!e) return fail(CLV_ERR_ARG, "null engine");
    if (field != 0 && field != 1) return fail(CLV_ERR_ARG, "field must be 0 or 1");
    CK(cudaSetDevice(e->device));
    LaunchSites L = e->sites();
    if (e->precision == CLV_PREC_F64) CK(launch_set_mean_field<double>(L, field, re, im, e->stream));
    else CK(launch_set_mean_field<float>(L, field, re, im, e->stream));
    CK(cudaStreamSynchronize(e->stream));
    return CLV_OK;
}

int clv_set_chemical_potential(clv_engine *e, int chain, double mu, double P) {
    if (!e) return fail(CLV_ERR_ARG, "null engine");
    if (chain != -1) {
        int rc = check_chain(e, chain);
        if (rc) return rc;
    }
    if (!std::isfinite(mu) || !std::isfinite(P)) return fail(CLV_ERR_ARG, "mu and P must be finite");
    CK(cudaSetDevice(e->device));
    const int c0 = chain == -1 ? 0 : chain, c1 = chain == -1 ? (int)e->params.size() : chain + 1;
    for (int c = c0; c < c1; ++c) {
        e->params[c].mu = mu;
        e->params[c].P = P;
        ChainDev &d = e->chains_h[c];
        d.mu = mu;
        d.P = P;
        for (int a = 0; a < kMaxComp; ++a) {
            const double m = 1.0 - a;
            d.comp_const[a] = std::exp(d.eps * (mu + d.q * m * m));
        }
    }
    // stream-ordered update of the device copies; captured graphs read them at run time
    CK(cudaMemcpyAsync(e->chains_d + c0, e->chains_h.data() + c0, (c1 - c0) * sizeof(ChainDev),
                       cudaMemcpyHostToDevice, e->stream));
    CK(cudaStreamSynchronize(e->stream));
    return CLV_OK;
}

int clv_init_spin1(clv_engine *e, double amp, double sigma) {
    if (!e) return fail(CLV_ERR_ARG, "null engine");
    CK(cudaSetDevice(e->device));
    LaunchSites L = e->sites();
    if (e->precision == CLV_PREC_F64) CK(launch_init_spin1<double>(L, amp, sigma, e->stream));
    else CK(launch_init_spin1<float>(L, amp, sigma, e->stream));
    CK(cudaStreamSynchronize(e->stream));
    return CLV_OK;
}

// Steps per block graph: long step sequences replay graphs of kStepBlock steps, so
// small lattices (the reference's own 256 x 32) pay one graph launch per block
// instead of one per step.
constexpr int kStepBlock = 16;
static_assert(kStepBlock % 2 == 0, "a block must return to its starting buffer set");

static int capture_steps(clv_engine *e, int from, int n, cudaGraph_t *g_out, cudaGraphExec_t *x_out) {
    CK(cudaStreamBeginCapture(e->stream, cudaStreamCaptureModeThreadLocal));
    int rc = CLV_OK;
    for (int i = 0; i < n && rc == CLV_OK; ++i) rc = enqueue_step_any(e, false, nullptr, from ^ (i & 1));
    cudaGraph_t g = nullptr;
    cudaError_t ce = cudaStreamEndCapture(e->stream, &g);
    if (rc) { if (g) cudaGraphDestroy(g); return rc; }
    if (ce != cudaSuccess) return fail(CLV_ERR_CUDA, std::string("capture: ") + cudaGetErrorString(ce));
    *g_out = g;
    CK(cudaGraphInstantiate(x_out, g, 0));
    return CLV_OK;
}

int clv_step(clv_engine *e, int nsteps) {
    if (!e) return fail(CLV_ERR_ARG, "null engine");
    if (nsteps < 0) return fail(CLV_ERR_ARG, "nsteps must be >= 0");
    CK(cudaSetDevice(e->device));
    if (nsteps == 0) return CLV_OK;
    if (use_loop(e)) {
        int done = 0;
        const int rc = enqueue_loop_any(e, nsteps, nullptr, &done);
        if (rc != kLoopRefused) return rc;
        nsteps -= done;  // the graphs take the rest
    }
    // graphs need a capturable stream (not the legacy default stream)
    if (nsteps == 1 || e->stream == nullptr || std::getenv("CLV_NO_GRAPH")) {
        for (int i = 0; i < nsteps; ++i) {
            int rc = enqueue_step_any(e, false, nullptr, e->cur);
            if (rc) return rc;
            e->cur ^= 1;
        }
        return CLV_OK;
    }
    while (nsteps >= kStepBlock) {
        const int from = e->cur;
        if (!e->block_exec[from]) {
            int rc = capture_steps(e, from, kStepBlock, &e->block_graph[from], &e->block_exec[from]);
            if (rc) return rc;
        }
        CK(cudaGraphLaunch(e->block_exec[from], e->stream));
        nsteps -= kStepBlock;
    }
    for (int i = 0; i < nsteps; ++i) {
        const int from = e->cur;
        if (!e->graph_exec[from]) {
            int rc = capture_steps(e, from, 1, &e->graph[from], &e->graph_exec[from]);
            if (rc) return rc;
        }
        CK(cudaGraphLaunch(e->graph_exec[from], e->stream));
        e->cur ^= 1;
    }
    return CLV_OK;
}

int clv_step_timed(clv_engine *e, float *phase_ms, int capacity, int *nphases) {
    if (!e) return fail(CLV_ERR_ARG, "null engine");
    CK(cudaSetDevice(e->device));
    EventTrail trail;
    int rc;
    if (use_loop(e) && (rc = enqueue_loop_any(e, 1, &trail)) != kLoopRefused) {
        if (rc) return rc;  // (two marks, bracketing the launch)
    } else {
        CK(trail.mark(e->stream));
        rc = enqueue_step_any(e, false, &trail, e->cur);
        if (rc) return rc;
        e->cur ^= 1;
    }
    CK(cudaStreamSynchronize(e->stream));
    // (the windows of a tiled step go through the same phases one after the other)
    const int all = (int)trail.ev.size() - 1, n = e->tiled ? all / (int)e->windows.size() : all;
    for (int i = 0; i < all; ++i) {
        float ms = 0.f;
        CK(cudaEventElapsedTime(&ms, trail.ev[i], trail.ev[i + 1]));
        if (phase_ms && i % n < capacity) phase_ms[i % n] = i < n ? ms : phase_ms[i % n] + ms;
    }
    if (nphases) *nphases = n;
    return CLV_OK;
}

int clv_step_with_noise(clv_engine *e, const double *noise, int where) {
    if (!e) return fail(CLV_ERR_ARG, "null engine");
    if (!noise) return fail(CLV_ERR_ARG, "null noise");
    if (where != CLV_HOST && where != CLV_DEVICE) return fail(CLV_ERR_ARG, "where: CLV_HOST or CLV_DEVICE");
    CK(cudaSetDevice(e->device));
    if (!e->noise_d) {
        void *p = nullptr;
        CK(malloc_beside(e, &p, e->noise_total * sizeof(double)));
        e->noise_d = (double *)p;
    }
    CK(cudaMemcpyAsync(e->noise_d, noise, e->noise_total * sizeof(double), kind_of(where, true),
                       e->stream));
    int rc = enqueue_step_any(e, true, nullptr, e->cur);
    if (rc) return rc;
    e->cur ^= 1;
    if (where == CLV_HOST) CK(cudaStreamSynchronize(e->stream));
    return CLV_OK;
}

int clv_get_step_info(clv_engine *e, double *dt, double *max_drift, double *mean_drift,
                      double *langevin_time, uint64_t *steps) {
    if (!e) return fail(CLV_ERR_ARG, "null engine");
    CK(cudaSetDevice(e->device));
    const int nch = (int)e->params.size();
    std::vector<ChainState> st(nch);
    CK(cudaMemcpyAsync(st.data(), e->state_d, nch * sizeof(ChainState), cudaMemcpyDeviceToHost,
                       e->stream));
    CK(cudaStreamSynchronize(e->stream));
    for (int c = 0; c < nch; ++c) {
        if (dt) dt[c] = st[c].dt;
        if (max_drift) max_drift[c] = st[c].max;
        if (mean_drift) mean_drift[c] = st[c].mean;
        if (langevin_time) langevin_time[c] = st[c].t;
        if (steps) steps[c] = st[c].step;
    }
    return CLV_OK;
}

int clv_get_chain_flags(clv_engine *e, int *flags) {
    if (!e || !flags) return fail(CLV_ERR_ARG, "null argument");
    CK(cudaSetDevice(e->device));
    const int nch = (int)e->params.size();
    std::vector<ChainState> st(nch);
    CK(cudaMemcpyAsync(st.data(), e->state_d, nch * sizeof(ChainState), cudaMemcpyDeviceToHost,
                       e->stream));
    CK(cudaStreamSynchronize(e->stream));
    int any = 0;
    for (int c = 0; c < nch; ++c) {
        flags[c] = st[c].flags;
        any |= st[c].flags;
    }
    if (any & CLV_FLAG_TIMEOUT)
        return fail(CLV_ERR_TIMEOUT, "a bounded device-side wait gave up (a chain's step is incomplete)");
    return (any & CLV_FLAG_NONFINITE) ? fail(CLV_ERR_NONFINITE, "a chain's drift became non-finite") : CLV_OK;
}

int clv_evaluate(clv_engine *e) {
    if (!e) return fail(CLV_ERR_ARG, "null engine");
    CK(cudaSetDevice(e->device));
    const int nch = (int)e->params.size();
    if (e->model == CLV_MODEL_REF4) {
        LaunchObs L = e->obs();
        L.sites = e->obs_tasks;
        L.nsites = (int)e->obs_tasks_h.size();
        L.scratch = e->obs_scratch;
        L.accF = e->accF;
        L.accN = e->accN;
        if (e->precision == CLV_PREC_F64) CK(launch_obs_ref<double>(L, e->stream));
        else CK(launch_obs_ref<float>(L, e->stream));
    } else {
        if (e->sample_count == e->sample_cap) {
            // move the full sample buffer to the host and start over
            const size_t n = (size_t)e->sample_cap * nch * 8;
            const size_t old = e->sample_spill.size();
            e->sample_spill.resize(old + n);
            CK(cudaMemcpyAsync(e->sample_spill.data() + old, e->samples, n * sizeof(double),
                               cudaMemcpyDeviceToHost, e->stream));
            CK(cudaMemsetAsync(e->samples, 0, n * sizeof(double), e->stream));
            CK(cudaStreamSynchronize(e->stream));
            e->sample_spilled += e->sample_cap;
            e->sample_count = 0;
        }
        if (e->energy_axis) {
            // kinetic energy sum_a (k_a^2/2) psi
            const int rc = e->precision == CLV_PREC_F64 ? run_groups<double>(e, e->energy_groups, e->psi(), nullptr)
                                                        : run_groups<float>(e, e->energy_groups, e->psi(), nullptr);
            if (rc) return rc;
        } else {
            int rc = e->precision == CLV_PREC_F64
                         ? run_kinetic<double>(e, e->psi(), nullptr, e->kin, nullptr, 1, 1)
                         : run_kinetic<float>(e, e->psi(), nullptr, e->kin, nullptr, 1, 1);
            if (rc) return rc;
        }
        LaunchObs L = e->obs();
        L.tpsi = e->kin;
        L.group = e->obs_group;
        L.arrive = e->obs_arrive;
        L.samples = e->samples;
        L.slot = e->sample_count;
        L.nchains = nch;
        if (e->precision == CLV_PREC_F64) CK(launch_obs_spin1<double>(L, e->stream));
        else CK(launch_obs_spin1<float>(L, e->stream));
        e->sample_count++;
    }
    e->counter++;
    return CLV_OK;
}

int clv_get_counter(clv_engine *e) { return e ? e->counter : 0; }

int clv_read_ref_observables(clv_engine *e, int chain, double *n, double *F_x, double *F_y,
                             double *F_z) {
    int rc = check_chain(e, chain);
    if (rc) return rc;
    if (e->model != CLV_MODEL_REF4) return fail(CLV_ERR_STATE, "reference observables need the REF4 model");
    if (e->counter == 0) return fail(CLV_ERR_STATE, "evaluate() has not been called");
    CK(cudaSetDevice(e->device));
    const ChainDev &d = e->chains_h[chain];
    std::vector<double> F(3 * d.V), N(5);
    CK(cudaMemcpyAsync(F.data(), e->accF + d.obs_off, 3 * d.V * sizeof(double),
                       cudaMemcpyDeviceToHost, e->stream));
    CK(cudaMemcpyAsync(N.data(), e->accN + chain * 5, 5 * sizeof(double), cudaMemcpyDeviceToHost,
                       e->stream));
    CK(cudaStreamSynchronize(e->stream));
    // Observables::write_n_* (:1527-1547): /T /counter /V ; write_F_* (:1614-1634): /T /counter
    const double T = d.nt, cnt = e->counter, V = d.V;
    if (n)
        for (int i = 0; i < 5; ++i) n[i] = N[i] / T / cnt / V;
    double *outs[3] = {F_x, F_y, F_z};
    for (int k = 0; k < 3; ++k)
        if (outs[k])
            for (int s = 0; s < d.V; ++s) outs[k][s] = F[k * d.V + s] / T / cnt;
    return CLV_OK;
}

int clv_read_spin1_samples(clv_engine *e, int chain, double *samples, int capacity, int *count) {
    int rc = check_chain(e, chain);
    if (rc) return rc;
    if (e->model != CLV_MODEL_SPIN1) return fail(CLV_ERR_STATE, "spin-1 samples need the SPIN1 model");
    CK(cudaSetDevice(e->device));
    const int nch = (int)e->params.size();
    const int total = e->sample_spilled + e->sample_count;
    // only this chain's rows of the device buffer ([k][chain][8]), and only what fits
    const int want = samples ? std::min(capacity, total) : 0;
    const int ndev = std::max(0, want - e->sample_spilled);
    std::vector<double> dev((size_t)ndev * 8);
    if (ndev > 0) {
        CK(cudaMemcpy2DAsync(dev.data(), 8 * sizeof(double), e->samples + (size_t)chain * 8,
                             (size_t)nch * 8 * sizeof(double), 8 * sizeof(double), ndev,
                             cudaMemcpyDeviceToHost, e->stream));
        CK(cudaStreamSynchronize(e->stream));
    }
    for (int k = 0; k < want; ++k) {
        const double *src = k < e->sample_spilled ? &e->sample_spill[((size_t)k * nch + chain) * 8]
                                                  : &dev[(size_t)(k - e->sample_spilled) * 8];
        std::memcpy(samples + (size_t)k * 8, src, 8 * sizeof(double));
    }
    if (count) *count = samples ? want : total;
    return CLV_OK;
}

// Re-plan with explicit knobs (chunk length; fused path: bulk copies, compile-time
// line length) and upload the new task tables; the captured graphs are dropped.
static int apply_plan(clv_engine *e, int L, int tma, int ln, int sd) {
    auto up = [&](void *d, const void *h, size_t b) {
        return cudaMemcpyAsync(d, h, b, cudaMemcpyHostToDevice, e->stream);
    };
    if (e->fused) {
        build_fused_tasks(e, L);
        e->use_tma = tma && e->fused_aligned;
        e->store_drift = sd && e->dt_rule == CLV_DT_REF_MEANMAX;
        if (ln != e->fused_ln) {
            LaunchFused probe{};
            probe.model = e->model;
            probe.ln = ln;
            probe.smem_bytes = e->fused_smem;
            probe.slot_stride = e->slot_stride;
            int per_sm = 0;
            if (e->precision == CLV_PREC_F64) CK(setup_fused<double>(probe, &per_sm));
            else CK(setup_fused<float>(probe, &per_sm));
            if (per_sm < 1) return fail(CLV_ERR_ARG, "fused plan variant does not fit");
            e->fused_ln = ln;
        }
        CK(up(e->fused_tasks, e->fused_tasks_h.data(), e->fused_tasks_h.size() * sizeof(FusedTask)));
    } else if (e->tiled) {
        build_tiled_tasks(e, L);
        CK(up(e->tile_tasks, e->tile_tasks_h.data(), e->tile_tasks_h.size() * sizeof(TileTask)));
    }
    CK(up(e->chains_d, e->chains_h.data(), e->chains_h.size() * sizeof(ChainDev)));
    CK(cudaStreamSynchronize(e->stream));
    e->drop_graphs();
    return CLV_OK;
}

int clv_autotune(clv_engine *e, int trial_steps, char *report, int capacity) {
    if (!e) return fail(CLV_ERR_ARG, "null engine");
    CK(cudaSetDevice(e->device));
    trial_steps = std::max(1, trial_steps);
    std::string rep;
    if (!e->fused && !e->tiled) {
        rep = "no tunable plan (separate line-filter, drift and update kernels)";
    } else {
        struct Cand { int L, tma, ln, sd; float ms; };
        std::vector<Cand> cands;
        int tmax = 0;
        for (auto &d : e->chains_h) tmax = std::max(tmax, d.nt);
        std::vector<int> Ls = {e->chunk};
        for (int L : {1, 2, 4, 8, 16, 32, 64})
            if (L <= tmax && L != e->chunk) Ls.push_back(L);
        for (int L : Ls) {
            if (e->fused) {
                for (int tma : {1, 0}) {
                    if (tma && !e->fused_aligned) continue;
                    for (int ln : {e->fused_ln_static, 0}) {
                        for (int sd : {0, 1}) {
                            if (sd && e->dt_rule != CLV_DT_REF_MEANMAX) continue;
                            cands.push_back({L, tma, ln, sd, 0.f});
                        }
                        if (e->fused_ln_static == 0) break;
                    }
                }
            } else {
                cands.push_back({L, 0, 0, e->store_drift, 0.f});
            }
        }
        // the trials run real steps: keep the state and restore it after each
        const size_t fb = (size_t)e->total_elems * e->elem_bytes;
        const int nch = (int)e->params.size();
        void *save[2] = {nullptr, nullptr};
        std::vector<ChainState> st(nch);
        const int cur0 = e->cur;
        cudaEvent_t ev0 = nullptr, ev1 = nullptr;
        auto cleanup = [&]() {
            for (void *p : save) if (p) cudaFree(p);
            if (ev0) cudaEventDestroy(ev0);
            if (ev1) cudaEventDestroy(ev1);
        };
        auto restore = [&]() -> cudaError_t {
            cudaError_t r;
            for (int f = 0; f < 2; ++f)
                if ((r = cudaMemcpyAsync(e->fld[cur0][f], save[f], fb, cudaMemcpyDeviceToDevice, e->stream)) != cudaSuccess)
                    return r;
            if ((r = cudaMemcpyAsync(e->state_d, st.data(), nch * sizeof(ChainState), cudaMemcpyHostToDevice,
                                     e->stream)) != cudaSuccess)
                return r;
            e->cur = cur0;
            return cudaStreamSynchronize(e->stream);
        };
        cudaError_t ce = cudaSuccess;
        for (int f = 0; f < 2 && ce == cudaSuccess; ++f) {
            ce = malloc_beside(e, &save[f], fb);
            if (ce == cudaSuccess)
                ce = cudaMemcpyAsync(save[f], e->fld[cur0][f], fb, cudaMemcpyDeviceToDevice, e->stream);
        }
        if (ce == cudaSuccess)
            ce = cudaMemcpyAsync(st.data(), e->state_d, nch * sizeof(ChainState), cudaMemcpyDeviceToHost, e->stream);
        if (ce == cudaSuccess) ce = cudaStreamSynchronize(e->stream);
        if (ce == cudaSuccess) ce = cudaEventCreate(&ev0);
        if (ce == cudaSuccess) ce = cudaEventCreate(&ev1);
        if (ce != cudaSuccess) {
            cleanup();
            return fail(CLV_ERR_NOMEM, std::string("autotune state copy: ") + cudaGetErrorString(ce));
        }
        int best = -1;
        for (int i = 0; i < (int)cands.size(); ++i) {
            Cand &c = cands[i];
            int rc = apply_plan(e, c.L, c.tma, c.ln, c.sd);
            if (rc == CLV_OK && (ce = restore()) != cudaSuccess) rc = fail(CLV_ERR_CUDA, cudaGetErrorString(ce));
            if (rc == CLV_OK) rc = clv_step(e, 2);  // captures the graphs of both parities
            if (rc == CLV_OK) {
                cudaEventRecord(ev0, e->stream);
                rc = clv_step(e, trial_steps);
                cudaEventRecord(ev1, e->stream);
                if ((ce = cudaEventSynchronize(ev1)) != cudaSuccess) rc = fail(CLV_ERR_CUDA, cudaGetErrorString(ce));
            }
            if (rc != CLV_OK) {
                cleanup();
                return rc;
            }
            cudaEventElapsedTime(&c.ms, ev0, ev1);
            c.ms /= trial_steps;
            if (best < 0 || c.ms < cands[best].ms) best = i;
            char line[128];
            std::snprintf(line, sizeof line, "chunk=%d tma=%d static_line=%d stored_drift=%d: %.4f ms/step\n",
                          c.L, c.tma, c.ln, c.sd, c.ms);
            rep += line;
        }
        const Cand &b = cands[best];
        int rc = apply_plan(e, b.L, b.tma, b.ln, b.sd);
        if (rc == CLV_OK && (ce = restore()) != cudaSuccess) rc = fail(CLV_ERR_CUDA, cudaGetErrorString(ce));
        cleanup();
        if (rc) return rc;
        char line[128];
        std::snprintf(line, sizeof line, "chosen: chunk=%d tma=%d static_line=%d stored_drift=%d", b.L, b.tma,
                      b.ln, b.sd);
        rep += line;
    }
    e->tune_report = rep;
    if (report && capacity > 0) {
        const size_t n = std::min(rep.size(), (size_t)capacity - 1);
        std::memcpy(report, rep.data(), n);
        report[n] = 0;
    }
    return CLV_OK;
}

// Name of a filter launch: planes and axes with their length, tile launches over whole slices
// or over lines of several lengths without one.
static std::string group_name(const clv_engine::AxisGroup &g) {
    if (g.tile && (g.whole || !g.n))
        return (g.whole ? "slices" : "lines" + std::to_string(g.axis)) + (g.threads > 128 ? "_wide" : "");
    return (g.plane ? "plane" + std::to_string(g.axis) + std::to_string(g.axis + 1) : "axis" + std::to_string(g.axis)) +
           "_n" + std::to_string(g.n);
}

int clv_get_plan(clv_engine *e, char *buf, int capacity) {
    if (!e || !buf || capacity < 1) return fail(CLV_ERR_ARG, "null argument");
    std::string p;
    if (e->fused) {
        if (use_loop(e)) p = "fused:loop_step";
        else if (e->speculate && e->dt_rule == CLV_DT_K_OVER_MAX) p = "fused:fused_step,fused_redo";
        else if (e->store_drift) p = "fused:fused_reduce,stored_drift_update";
        else p = "fused:fused_reduce,fused_apply";
    } else if (e->tiled) {
        p = "tiled:";
        for (const auto &g : e->axis_groups) p += group_name(g) + ",";
        p += (e->speculate && e->dt_rule == CLV_DT_K_OVER_MAX) ? "tiled_step,tiled_redo"
             : e->store_drift ? "tiled_reduce,stored_drift_update" : "tiled_reduce,tiled_apply";
    } else {
        p = "unfused:";
        for (const auto &g : e->axis_groups) p += group_name(g) + ",";
        for (int a = 0; a < 3 && e->axis_groups.empty(); ++a) {
            if (e->line_tasks_h[a].empty()) continue;
            if (e->kinetic == CLV_KIN_REF_LINEAR_PX && a > 0) break;
            p += "kinetic_axis" + std::to_string(a) + ",";
        }
        p += "drift,update";
    }
    if ((int)p.size() >= capacity) return fail(CLV_ERR_ARG, "buffer too small for the plan");
    std::memcpy(buf, p.c_str(), p.size() + 1);
    return CLV_OK;
}

int clv_device_bytes(clv_engine *e, size_t *bytes) {
    if (!e || !bytes) return fail(CLV_ERR_ARG, "null argument");
    *bytes = e->dev_bytes + (e->noise_d ? e->noise_total * sizeof(double) : 0);
    return CLV_OK;
}

// ------------------------------------------------------------- checkpoint
// File: magic "CLVCKPT1", int32 header {version, model, precision, ncomp, nchains},
// per chain {nx, ny, nz, nt}, ChainState[nchains], int32 counter, sample state,
// then per chain psi, psibar (complex128, boundary layout), F accumulators,
// N accumulators and the spin-1 samples.
int clv_save_checkpoint(clv_engine *e, const char *path) {
    if (!e || !path) return fail(CLV_ERR_ARG, "null argument");
    CK(cudaSetDevice(e->device));
    const int nch = (int)e->params.size();
    FILE *f = std::fopen(path, "wb");
    if (!f) return fail(CLV_ERR_IO, std::string("cannot open ") + path);
    bool ok = true;
    auto W = [&](const void *p, size_t b) { ok = ok && std::fwrite(p, 1, b, f) == b; };
    W("CLVCKPT1", 8);
    const int hdr[5] = {CLV_API_VERSION, e->model, e->precision, e->ncomp, nch};
    W(hdr, sizeof hdr);
    for (auto &p : e->params) { const int dims[4] = {p.nx, p.ny, p.nz, p.nt}; W(dims, sizeof dims); }
    std::vector<ChainState> st(nch);
    cudaError_t ce = cudaMemcpyAsync(st.data(), e->state_d, nch * sizeof(ChainState),
                                     cudaMemcpyDeviceToHost, e->stream);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(e->stream);
    if (ce != cudaSuccess) { std::fclose(f); return fail(CLV_ERR_CUDA, cudaGetErrorString(ce)); }
    W(st.data(), nch * sizeof(ChainState));
    const int counters[3] = {e->counter, e->sample_count, e->sample_spilled};
    W(counters, sizeof counters);
    std::vector<double2> a(e->max_chain_elems), b(e->max_chain_elems);
    for (int c = 0; c < nch && ok; ++c) {
        int rc = clv_get_fields(e, c, a.data(), b.data(), CLV_HOST);
        if (rc) { std::fclose(f); return rc; }
        const long long n = (long long)e->ncomp * e->chains_h[c].nt * e->chains_h[c].V;
        W(a.data(), n * 16);
        W(b.data(), n * 16);
    }
    std::vector<double> F(std::max(1, e->acc_F_total)), N(nch * 5);
    std::vector<double> S((size_t)e->sample_count * nch * 8);
    ce = cudaMemcpy(F.data(), e->accF, F.size() * sizeof(double), cudaMemcpyDeviceToHost);
    if (ce == cudaSuccess) ce = cudaMemcpy(N.data(), e->accN, N.size() * sizeof(double), cudaMemcpyDeviceToHost);
    if (ce == cudaSuccess && !S.empty())
        ce = cudaMemcpy(S.data(), e->samples, S.size() * sizeof(double), cudaMemcpyDeviceToHost);
    if (ce != cudaSuccess) { std::fclose(f); return fail(CLV_ERR_CUDA, cudaGetErrorString(ce)); }
    W(F.data(), F.size() * sizeof(double));
    W(N.data(), N.size() * sizeof(double));
    W(S.data(), S.size() * sizeof(double));
    W(e->sample_spill.data(), e->sample_spill.size() * sizeof(double));
    if (std::fclose(f) != 0) ok = false;
    return ok ? CLV_OK : fail(CLV_ERR_IO, std::string("short write to ") + path);
}

int clv_load_checkpoint(clv_engine *e, const char *path) {
    if (!e || !path) return fail(CLV_ERR_ARG, "null argument");
    CK(cudaSetDevice(e->device));
    const int nch = (int)e->params.size();
    FILE *f = std::fopen(path, "rb");
    if (!f) return fail(CLV_ERR_IO, std::string("cannot open ") + path);
    bool ok = true;
    auto R = [&](void *p, size_t b) { ok = ok && std::fread(p, 1, b, f) == b; };
    char magic[8];
    int hdr[5];
    R(magic, 8);
    R(hdr, sizeof hdr);
    if (!ok || std::memcmp(magic, "CLVCKPT1", 8) != 0 || hdr[1] != e->model ||
        hdr[2] != e->precision || hdr[3] != e->ncomp || hdr[4] != nch) {
        std::fclose(f);
        return fail(CLV_ERR_IO, "checkpoint does not match this engine");
    }
    for (auto &p : e->params) {
        int dims[4];
        R(dims, sizeof dims);
        if (!ok || dims[0] != p.nx || dims[1] != p.ny || dims[2] != p.nz || dims[3] != p.nt) {
            std::fclose(f);
            return fail(CLV_ERR_IO, "checkpoint lattice sizes do not match");
        }
    }
    std::vector<ChainState> st(nch);
    R(st.data(), nch * sizeof(ChainState));
    int counters[3];
    R(counters, sizeof counters);
    if (!ok || counters[1] < 0 || counters[1] > e->sample_cap || counters[2] < 0) {
        std::fclose(f);
        return fail(CLV_ERR_IO, "truncated checkpoint");
    }
    std::vector<double2> a(e->max_chain_elems), b(e->max_chain_elems);
    for (int c = 0; c < nch && ok; ++c) {
        const long long n = (long long)e->ncomp * e->chains_h[c].nt * e->chains_h[c].V;
        R(a.data(), n * 16);
        R(b.data(), n * 16);
        if (!ok) break;
        int rc = clv_set_fields(e, c, a.data(), b.data(), CLV_HOST);
        if (rc) { std::fclose(f); return rc; }
    }
    std::vector<double> F(std::max(1, e->acc_F_total)), N(nch * 5);
    std::vector<double> S((size_t)counters[1] * nch * 8);
    std::vector<double> spill((size_t)counters[2] * nch * 8);
    R(F.data(), F.size() * sizeof(double));
    R(N.data(), N.size() * sizeof(double));
    R(S.data(), S.size() * sizeof(double));
    R(spill.data(), spill.size() * sizeof(double));
    std::fclose(f);
    if (!ok) return fail(CLV_ERR_IO, "truncated checkpoint");
    for (auto &s : st) s.arrive = 0;
    CK(cudaMemcpy(e->state_d, st.data(), nch * sizeof(ChainState), cudaMemcpyHostToDevice));
    CK(cudaMemcpy(e->accF, F.data(), F.size() * sizeof(double), cudaMemcpyHostToDevice));
    CK(cudaMemcpy(e->accN, N.data(), N.size() * sizeof(double), cudaMemcpyHostToDevice));
    CK(cudaMemset(e->samples, 0, (size_t)e->sample_cap * nch * 8 * sizeof(double)));
    if (!S.empty()) CK(cudaMemcpy(e->samples, S.data(), S.size() * sizeof(double), cudaMemcpyHostToDevice));
    e->counter = counters[0];
    e->sample_count = counters[1];
    e->sample_spilled = counters[2];
    e->sample_spill = std::move(spill);
    return CLV_OK;
}

}  // extern "C"
