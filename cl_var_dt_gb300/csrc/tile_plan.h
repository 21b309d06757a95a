// tile_plan.h -- host side of the tile filter's plans (k_tile.cuh): radices, the order of
// frequencies that they leave, the tile's pitch.
#pragma once

#include <algorithm>
#include <vector>

#include "clv_internal.cuh"

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

// Shared elements between the rows of a tile with `lines` lines along rows of n.  A phase of a
// warp's access (16 elements at FP32, 8 at FP64) takes the lines of the tile at as many
// neighbouring positions as fit: an odd pitch keeps it free of conflicts when one position of
// that many lines does, else an odd multiple of the positions does.
inline int tile_pitch(int elem_bytes, int n, int lines) {
    int g = elem_bytes == 8 ? 16 : 8;
    for (int l = 1; l < lines && g > 1; l *= 2) g /= 2;
    return g == 1 ? n | 1 : (n + g - 1) / g * g + ((n + g - 1) / g % 2 ? 0 : g);
}

}  // namespace clv
