// How a filter pass of the exact k-NN is split over the GPU. Host code.
#pragma once

#include <algorithm>
#include <cstdint>

// A CTA takes tps tiles of rows for one query tile; splits CTAs cover a query tile's rows.
struct Split {
    int tps, splits;
};

// What a CTA's start and end cost, in tiles. Its value matters little: with 0, 1, 3 and 6 nineteen searches (1 to
// 10K queries, 3K to 1M rows, bytes and floats) took the same time within what repeats differ (10K x 60K x 784 bytes
// 1.13, 1.13, 1.12, 1.13 ms), with 12 that one took 1.15 ms.
constexpr int FIXED_TILES = 3;

// The split of `tiles` tiles for qt query tiles whose waves of CTAs (one an SM) end soonest, of at most about
// eight waves; of equal ones the fewest CTAs. In a given number of waves the most CTAs have the fewest tiles
// each, so one split a wave is looked at (trying every number of CTAs took the host 4.8 us for one query tile
// of 3,907 tiles, several times a call; this takes 0.1 us).
inline Split split_tiles(int qt, int tiles, int sms) {
    const int most = std::min(tiles, std::max(1, (8 * sms + qt - 1) / qt));
    Split best{tiles, 1};
    int64_t least = INT64_MAX;
    for (int64_t w = (int64_t(qt) + sms - 1) / sms;; w++) {
        const int s = int(std::min<int64_t>(most, w * sms / qt));
        const int tps = (tiles + s - 1) / s, splits = (tiles + tps - 1) / tps;
        const int64_t waves = (int64_t(qt) * splits + sms - 1) / sms, cost = waves * (tps + FIXED_TILES);
        if (cost < least) {
            least = cost;
            best = Split{tps, splits};
        }
        if (s == most) return best;
    }
}
