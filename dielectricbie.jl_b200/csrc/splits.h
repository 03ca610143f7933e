// Source splits of a direct sum (host side).
#pragma once
#include <algorithm>
#include <cstdint>

namespace bie {

constexpr int kTS = 128;  // sources per shared-memory tile; splits are whole tiles

// Splits of n sources for `tiles` target tiles on `slots` resident CTAs. The CTAs run in waves, so the
// sum takes waves x sources per split; one wave at most leaves up to half of the slots empty when the
// tiles are more than half of them, so up to eight waves are considered. A CTA's start costs about 64
// sources, a split's partials (written, and read by the reduction) about 60 per wave of tiles.
inline int wave_splits(int64_t n, int64_t tiles, int64_t slots) {
    const int64_t chunks = (n + kTS - 1) / kTS;
    const int64_t most = std::max<int64_t>(1, std::min(chunks, 8 * slots / std::max<int64_t>(tiles, 1)));
    int64_t best = 1;
    double cost = -1.0;
    for (int64_t ns = 1; ns <= most; ++ns) {
        const int64_t cps = (chunks + ns - 1) / ns, used = (chunks + cps - 1) / cps;  // splits that get sources
        const int64_t waves = (tiles * used + slots - 1) / slots;
        const double c = (double)waves * (double)(kTS * cps + 64) + 60.0 * (double)(used * tiles) / (double)slots;
        if (cost < 0.0 || c < cost) {
            cost = c;
            best = used;
        }
    }
    return (int)best;
}

}  // namespace bie
