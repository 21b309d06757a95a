// Host build of the tile filter (csrc/k_tile.cuh) at FP64: whole slices with the plans of
// csrc/tile_plan.h, and the same lines by FP64 butterflies for comparison.
#include "host_cuda.h"

namespace clv { alignas(128) unsigned char smem[1 << 19]; }

#include "../cl_var_dt_gb300/csrc/k_tile.cuh"
#include "../cl_var_dt_gb300/csrc/tile_plan.h"

using namespace clv;

extern "C" int tile_plan(int n, int most, int *fac) {
    int nf = 0;
    return tile_factors(n, most, fac, nf) ? nf : 0;
}
extern "C" int tile_pitch_of(int elem_bytes, int n, int lines) { return tile_pitch(elem_bytes, n, lines); }
extern "C" void tile_frequencies(int n, int most, int *out) {
    int fac[kMaxTileFactors], nf;
    if (!tile_factors(n, most, fac, nf)) return;
    const std::vector<int> o = tile_order(n, fac, nf);
    std::copy(o.begin(), o.end(), out);
}

extern "C" void fixed_twiddle_table(int n, long long *out) {
    for (const WCplx &w : fixed_twiddles(n)) {
        *out++ = (long long)w.x.h * 4294967296ll + w.x.l;
        *out++ = (long long)w.y.h * 4294967296ll + w.y.l;
    }
}

static std::vector<double2> twiddles(int n) {
    std::vector<double2> tw(n);
    for (int k = 0; k < n; ++k) {
        const long double a = -2.0L * acosl(-1.0L) * (long double)k / (long double)n;
        tw[k] = make_double2((double)cosl(a), (double)sinl(a));
    }
    return tw;
}

// ns slices of dims, filters of the axes (n values each, 1/n folded in) one after the other; axes:
// how many of the leading axes are filtered; energy: the filters are summed.  cst: a constant
// factor.  0 when the tile does not fit.
extern "C" int tile_filter(const int *dims, int axes, int ns, int energy, double cst, const double *filt,
                           const double *in, double *out) {
    ChainDev ch{};
    ch.nx = dims[0]; ch.ny = dims[1]; ch.nz = dims[2];
    ch.V = dims[0] * dims[1] * dims[2];
    ch.nt = ns;
    ch.ncomp = 1;
    ch.comp_const[0] = cst;
    TileFilterPlan P{};
    std::vector<WCplx> tw[3];
    std::vector<double> f[3];
    int last = 0, nsum = 0;
    for (int a = 0, o = 0; a < 3; ++a) {
        AxisDev &ax = ch.axis[a];
        ax.n = dims[a];
        ax.inner = a == 0 ? dims[1] * dims[2] : (a == 1 ? dims[2] : 1);
        if (dims[a] > 1) last = a;
        if (dims[a] <= 1 || a >= axes) continue;
        if (!tile_factors(ax.n, tile_radix_max<double>(), ax.tfac, ax.tnf)) return 0;
        tw[a] = fixed_twiddles(ax.n);
        const std::vector<int> order = tile_order(ax.n, ax.tfac, ax.tnf);
        f[a].resize(ax.n);
        double most = 0;
        for (int i = 0; i < ax.n; ++i) {
            f[a][i] = filt[o + order[i]];
            most = std::max(most, std::fabs(f[a][i]));
        }
        o += ax.n;
        ax.tw62 = tw[a].data();
        ax.tfilt64 = ax.tefilt64 = f[a].data();
        ax.fmax = ax.efmax = most;
        P.axis[P.naxes] = a;
        P.inner[P.naxes++] = ax.inner;
        nsum += ax.n;
    }
    const int cols = dims[last], rows = ns * ch.V / cols;
    P.with_const = !energy;
    // a filter that vanishes at zero frequency, long lines (large slices of a sum)
    P.based = (P.naxes == 1 ? ch.axis[P.axis[0]].n : ch.V) > kBasedSites && (energy || filt[0] == 0.0);
    P.pitch = tile_pitch(16, cols, rows);
    P.tile_elems = (rows * P.pitch + 1) / 2 * 2;
    if ((size_t)P.tile_elems * 16 + nsum * 24 + rows * 8 + 36 * (size_t)rows * cols > sizeof smem) return 0;
    const TileFilterTask task{0, 0, 0, 0, rows, cols};
    LaunchTileFilter A{};
    A.chains = &ch;
    A.plans = &P;
    A.tasks = &task;
    A.ntasks = 1;
    A.src0 = in;
    A.dst0 = out;
    A.nfields = 1;
    A.filter = energy;
    tile_filter_kernel<double, 128>(A);
    return 1;
}

extern "C" int line_path(int fp64, int ref_rule, int ln, int ncomp, int chains, int nt, long long device_bytes) {
    LineBatch b{};
    b.fp64 = fp64; b.ref_rule = ref_rule; b.ln = ln;
    b.largest = (long long)ln * nt;
    b.sites = chains * b.largest;
    b.slices = (long long)chains * nt;
    b.field_bytes = b.sites * ncomp * (fp64 ? 16 : 8);
    b.device_bytes = device_bytes;
    b.num_sms = 152;
    b.loop_ctas = 152;
    return lines_on_the_tiled_path(b);
}

// One line of n sites by FP64 butterflies of 8, 4, 2, 3 and 5 (Stockham passes), filter f
// in the order of frequencies.
template <int R, int S>
static void pass64(int n, int NS, const double2 *s, double2 *d, const double2 *tw) {
    for (int j = 0; j < n / R; ++j) {
        const int k = j % NS;
        double2 v[R];
        for (int r = 0; r < R; ++r) {
            double2 w = tw[k * r * (n / (NS * R))];
            if (S > 0) w.y = -w.y;
            v[r] = s[j + r * (n / R)];
            if (NS > 1 && r > 0) v[r] = vmul(v[r], w);
        }
        Radix<double2, R>::template run<S>(v);
        for (int q = 0; q < R; ++q) d[j / NS * NS * R + k + q * NS] = v[q];
    }
}
template <int S>
static void transform64(int n, double2 *x, double2 *y, const double2 *tw) {
    int NS = 1;
    for (int m = n; m > 1;) {
        const int R = m % 8 == 0 ? 8 : m % 4 == 0 ? 4 : m % 2 == 0 ? 2 : m % 3 == 0 ? 3 : 5;
        switch (R) {
            case 8: pass64<8, S>(n, NS, x, y, tw); break;
            case 4: pass64<4, S>(n, NS, x, y, tw); break;
            case 2: pass64<2, S>(n, NS, x, y, tw); break;
            case 3: pass64<3, S>(n, NS, x, y, tw); break;
            default: pass64<5, S>(n, NS, x, y, tw);
        }
        std::copy(y, y + n, x);
        NS *= R;
        m /= R;
    }
}
extern "C" void line_filter64(int n, int lines, const double *f, double *io) {
    const std::vector<double2> tw = twiddles(n);
    std::vector<double2> y(n);
    for (int l = 0; l < lines; ++l) {
        double2 *x = reinterpret_cast<double2 *>(io) + (size_t)l * n;
        transform64<-1>(n, x, y.data(), tw.data());
        for (int k = 0; k < n; ++k) x[k] = vscale(f[k], x[k]);
        transform64<1>(n, x, y.data(), tw.data());
    }
}
