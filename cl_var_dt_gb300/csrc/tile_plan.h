// tile_plan.h -- host side of the tile filter's plans (k_tile.cuh): radices, the order of
// frequencies that they leave, the tile's pitch; the twiddles of the integer lines.
#pragma once

#include <algorithm>
#include <vector>

#include "clv_internal.cuh"
#include "fft_int.cuh"

namespace clv {

// In-place plan of the tile filter: as few radices of 2 .. most as the length allows, the most
// even such split, larger ones first.
inline bool tile_factors(int n, int most, int *fac, int &nf) {
    static const int radices[] = {16, 15, 12, 10, 9, 8, 6, 5, 4, 3, 2};
    if (n <= 1) return false;
    for (int want = 1; want <= kMaxTileFactors; ++want) {
        int best[kMaxTileFactors], cur[kMaxTileFactors], sum = 1 << 30;
        auto search = [&](auto &&self, int rest, int depth, int top) -> void {
            if (depth == want) {
                int s = 0;
                for (int i = 0; i < want; ++i) s += cur[i];
                if (rest == 1 && s < sum) {
                    sum = s;
                    std::copy(cur, cur + want, best);
                }
                return;
            }
            for (int r : radices)
                if (r <= top && rest % r == 0) {
                    cur[depth] = r;
                    self(self, rest / r, depth + 1, r);
                }
        };
        search(search, n, 0, most);
        if (sum < (1 << 30)) {
            nf = want;
            std::copy(best, best + want, fac);
            return true;
        }
    }
    return false;
}

// Frequency at every position after the forward passes: position sum_p q_p (L_p / R_p) holds
// sum_p q_p (R_0 ... R_{p-1}).
inline std::vector<int> tile_order(int n, const int *fac, int nf) {
    std::vector<int> order(n);
    for (int i = 0; i < n; ++i) {
        int rest = i, L = n, w = 1, k = 0;
        for (int p = 0; p < nf; ++p) {
            L /= fac[p];
            k += rest / L * w;
            rest %= L;
            w *= fac[p];
        }
        order[i] = k;
    }
    return order;
}

// exp(-2 pi i k / n), k < n, with 62 fraction bits.  Rounded doubles would carry 2^-54 of an
// element into every product, which is the whole error of a line with one site far above the
// others.  Taylor series in 96 fraction bits of the angle from the nearest multiple of pi / 4
// (integers: the same table on every host).
inline std::vector<WCplx> fixed_twiddles(int n) {
    using u128 = unsigned __int128;
    using i128 = __int128;
    auto mul = [](i128 a, i128 b) {  // |a|, |b| <= 2^96
        const u128 x = a < 0 ? -(u128)a : (u128)a, y = b < 0 ? -(u128)b : (u128)b, m = ((u128)1 << 48) - 1;
        const u128 p = (x >> 48) * (y >> 48) + (((x >> 48) * (y & m) + (x & m) * (y >> 48)) >> 48);
        return (a < 0) != (b < 0) ? -(i128)p : (i128)p;
    };
    const i128 one = (i128)1 << 96, twopi = ((i128)0x6487ED511ull << 64) | 0x0B4611A62633145Cull;
    const i128 h = ((i128)0xB504F333ull << 64) | 0xF9DE6484597D89B3ull;  // sqrt(1/2)
    constexpr int kTerms = 22;                                     // (pi / 8)^22 / 22! < 2^-99
    i128 inv[kTerms + 1] = {one};                                  // 1 / j!
    for (int j = 1; j <= kTerms; ++j) inv[j] = inv[j - 1] / j;
    std::vector<WCplx> tw(n);
    for (int k = 0; 2 * k <= n; ++k) {
        const int o = (8 * k + n / 2) / n;                         // nearest multiple of pi / 4
        const i128 t = twopi * (8 * k - o * n) / (8 * n), t2 = mul(t, t);
        i128 c = inv[kTerms], s = inv[kTerms - 1];                 // cos, sin of t, |t| <= pi / 8
        for (int j = kTerms - 2; j >= 0; j -= 2) {
            c = inv[j] - mul(c, t2);
            if (j > 0) s = inv[j - 1] - mul(s, t2);
        }
        s = mul(s, t);
        const i128 d = mul(h, c - s), e = mul(h, c + s);
        // angle o pi / 4 + t
        const i128 x[8] = {c, d, -s, -e, -c, -d, s, e}, y[8] = {s, e, c, d, -s, -e, -c, -d};
        auto round = [](i128 v) { return (long long)((v + ((i128)1 << 33)) >> 34); };
        const long long wx = round(x[o & 7]), wy = round(y[o & 7]);
        tw[k] = WCplx{wsplit(wx), wsplit(-wy)};
        tw[(n - k) % n] = WCplx{wsplit(wx), wsplit(k ? wy : 0)};
    }
    return tw;
}

// Shared elements between the rows of a tile with `lines` lines along rows of n.  A phase of a
// warp's access (16 elements at FP32, 8 at FP64) takes the lines of the tile at as many
// neighbouring positions as fit: an odd pitch keeps it free of conflicts when one position of
// that many lines does, else an odd multiple of the positions does.
inline int tile_pitch(int elem_bytes, int n, int lines) {
    int g = elem_bytes == 8 ? 16 : 8;
    for (int l = 1; l < lines && g > 1; l *= 2) g /= 2;
    return g == 1 ? n | 1 : (n + g - 1) / g * g + ((n + g - 1) / g % 2 ? 0 : g);
}

// Lines (slices of a sum) of more sites than this are taken relative to their first site under a
// filter that vanishes at zero frequency, the reference's k^2 and kinetic energies, where a
// condensate costs precision: up to 256 sites at most 0.8 of the FP64 butterflies' error is left
// (128 sites: 0.2), from 270 to 2048 up to 2.2 times it, and relative to the first site 0.8.
constexpr int kBasedSites = 256;

// A batch of 1D lines that both the fused and the tiled path can step.
struct LineBatch {
    bool fp64, ref_rule;
    int ln;                        // sites of a line: 64, 128, 256
    long long sites, largest;      // of all chains and imaginary times, of the largest chain
    long long slices;              // imaginary times of all chains
    long long field_bytes, device_bytes;
    int num_sms, loop_ctas;        // the step loop's resident CTAs
};

// 1D batches of ln-site lines that the tiled path steps faster than the fused one (us a step,
// fused / tiled; chains x sites x imaginary times).  The fused step saves the kinetic term's way
// through HBM, but filters with a warp per line; the tile filter fills its warps whatever
// the lines, and the tiled step overlaps noise and drift over more of them.
//   * FP32 under the reference's rule, whose second pass filters once more (the step loop's
//     small problems aside): 3 x 64 x 32 27 / 23, 8 x 256 x 64 47 / 38, 120 x 128 x 100 275 / 177.
//   * FP64 from three blocks of sites an SM on, lines of 64 and, under the reference's rule,
//     of 256: reference model 40 x 64 x 64 212 / 158, 120 x 256 x 100 2669 / 2172; spin-1 40 x 64
//     x 64 159 / 122.  Others stay: reference model 120 x 128 x 100 1056 / 1113; 8 x 64 x 64
//     64 / 64; spin-1 40 x 128 x 64 201 / 219, 40 x 256 x 64 328 / 384.
//   * FP32, K/max rule: lines of 64 from 16 blocks an SM on (120 x 64 x 100 84 / 69; 40 x 64 x 64
//     28 / 28; 120 x 128 x 100 104 / 113).
// The two paths round differently, so sizes alone decide, not the memory that other engines leave:
// that would change a chain's trajectory.  The tiled path steps in windows where kinbar does not
// fit, which takes chains of at most half of the sites; batches of one large chain, a field of
// over a 64th of the device's memory, stay fused, except for the reference model at FP64, which
// can do without its stored drift.
inline bool lines_on_the_tiled_path(const LineBatch &b) {
    if (2 * b.largest > b.sites && !(b.ref_rule && b.fp64) && b.field_bytes > b.device_bytes / 64) return false;
    const long long per_sm = b.sites / (256LL * b.num_sms);
    if (b.fp64) return per_sm >= 3 && (b.ln == 64 || (b.ln == 256 && b.ref_rule));
    if (!b.ref_rule) return b.ln == 64 && per_sm >= 16;
    return 2 * b.slices > b.loop_ctas;
}

}  // namespace clv
