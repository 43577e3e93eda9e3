// x3 chunk lengths of the sweeps: planes per block (host arithmetic only).
#pragma once
#include <algorithm>
#include <utility>
#include <vector>

namespace sph {

// x3 chunk length of a batch's sweeps: the time model (k + 2) * max(2.15, 1.1 n + 0.5), n = blocks on the fullest SM
// (two are resident, and two together are hardly slower than one), over 1..24 planes.  us per sweep of 256 grids of
// 31 .. 47 cells a side, chunks of 8 / 16 (its pick) / 24 planes: 580 / 515 / 530; of 64: 221 / 201 / 207.
// tiles: (tiles in x1 and x2, planes) of each grid of the launch
inline int chunk_rule(const std::vector<std::pair<long long, int>>& tiles, int sms) {
    int best = 1, planes = 0;
    for (const auto& t : tiles) planes = std::max(planes, t.second);
    double best_t = 1e300;
    for (int k : {1, 2, 3, 4, 6, 8, 12, 16, 24}) {
        long long blocks = 0;
        for (const auto& t : tiles) blocks += t.first * ((t.second + k - 1) / k);
        const int n = (int)((blocks + sms - 1) / sms);
        const double t = (k + 2.0) * std::max(2.15, 1.1 * n + 0.5);
        if (t < best_t) { best_t = t; best = k; }
        if (k >= planes) break;
    }
    return best;
}

// x3 chunk length of the sweep of one grid: the end of its last block, in planes.  A block takes its planes and one more
// (the halo plane below), two blocks are resident on an SM, and the blocks start in order of x3, so that the short
// last chunks of a column (the rest of n3 / k) come last, on the slots that the others leave free.  A last wave on
// half the SMs' slots or fewer runs an eighth faster.  Chunks above 24 planes are not considered: 32 are better at
// 255^3 (298 us) but worse at 511 x 255 x 255 (620).
// Measured on a GB300, us per sweep with the rule above and with this one: 38 x 172 x 248 77.7 and 62.0, 200 x 16 x 200
// 34.4 and 28.8, 127 x 32 x 244 35.2 and 28.9, 96 x 85 x 180 39.6 and 32.2, 127^3 58.0 and 50.1, 221 x 116 x 80 53.7 and 45.6,
// 131 x 117 x 101 44.5 and 44.1; the same length, or the same time, at 47 x 31 x 39, 63^3, 255^3 and 511 x 255 x 255.
// Of 15 lengths tried at ten sizes its pick is the best or within 1 %.
// sph_autotune measures instead.
inline int grid_chunk(long long tiles, int planes, int sms) {
    const long long slots = 2LL * sms;
    int best = 1;
    double best_t = 1e300;
    for (int k = 1; k <= 24 && k <= planes; k += k < 16 ? 1 : 4) {
        const long long full = tiles * (planes / k), q = full / slots, r = full % slots;
        const int rem = planes % k, u = k + 1;
        double t = (double)(q + (r > 0)) * u;
        if (rem) {
            const long long fit = (slots - r) * (u / (rem + 1));  // short blocks that end before the last full ones
            if (r == 0 || tiles > fit) {
                const long long late = r == 0 ? tiles : tiles - fit;
                t += (double)((late + slots - 1) / slots) * (rem + 1);
            }
        } else if (r > 0 && r <= sms) {
            t -= 0.125 * u;
        }
        if (t < best_t) { best_t = t; best = k; }
    }
    return best;
}

// x3 chunk length of k_fused: tiles of 32 x 8 cells, three blocks on an SM, and about two and a half planes of fill and halo
// a block: (k + 2.5) max(1, n / 3 + 0.3), n = blocks on the fullest SM.  us per sweep with grid_chunk (whose tiles, residency and halo are
// those of k_sweep) and with this: 47 x 31 x 39 14.3 and 12.8, 63^3 23.2 and 20.8, 23 x 40 x 200 22.2 and 20.0, 127 x 32 x 244 50.7 and
// 47.2, 28 x 29 x 158 19.3 and 18.0, 255^3 574 and 571; 131 x 117 x 101 79.3 and 81.0, 127^3 86.9 and 88.9, 200 x 16 x 200 35.4 and 37.6.
inline int fallback_chunk(long long tiles, int planes, int sms) {
    int best = 1;
    double best_t = 1e300;
    for (int k = 1; k <= 24 && k <= planes; k += k < 16 ? 1 : 4) {
        const long long n = (tiles * ((planes + k - 1) / k) + sms - 1) / sms;
        const double t = (k + 2.5) * std::max(1.0, n / 3.0 + 0.3);
        if (t < best_t) { best_t = t; best = k; }
    }
    return best;
}

}  // namespace sph
