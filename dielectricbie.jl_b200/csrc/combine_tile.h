// Column tile of the block-row correction apply (k_combine_dmma) and its shared memory (host side).
#pragma once
#include <algorithm>
#include <cstddef>

namespace bie {

// Slab row stride for a kt-column tile: kt rounded up to 8, plus 4 (stride = 4 or 12
// mod 16 doubles, so a half-warp's fragment loads hit distinct banks).
constexpr int comb_ldx(int kt) { return ((kt + 7) / 8) * 8 + 4; }

// Shared memory of the block-row combine for nb-row panels, kt-column tiles and
// `stages` pipeline stages (reused for the warps' final reduction).
inline size_t combine_smem_bytes(int nb, int kt, int stages, int warps) {
    const int mt = (nb + 7) / 8, kp = ((nb + 3) / 4) * 4;
    const int ldc = mt * 8 + 4;
    const size_t pipe = (size_t)stages * kp * (ldc + comb_ldx(kt) + 1);
    const size_t red = (size_t)warps * mt * 2 * 32;  // cross-warp reduction of the accumulators
    return sizeof(double) * std::max(pipe, red);
}

// Warps of ct-column tiles that an SM holds (228 KB of shared memory, 1 KB of it reserved per CTA).
inline int combine_warps(int nb, int ct) {
    const size_t per = combine_smem_bytes(nb, ct, 2, ct / 8) + 1024;
    return (int)std::min<size_t>(228 * 1024 / per, 2048 / (4 * ct)) * (ct / 8);
}

// Columns a CTA takes: 64 read the blocks half as often as 32, but need more shared memory. us with
// tiles of 32 and of 64 columns:
//   half as many tiles: 128 columns, 1,168 panels of 36 nodes 223 and 197, 728 panels of 64 408 and 382;
//     64 columns: 121 and 126 on 1,168 panels of 36, 331 and 272 on 2,632, so at this width only on many;
//   two tiles instead of three, the last at most half full (80 columns, 728 panels): worth it where an SM
//     then holds more warps: 36 nodes 112 and 105, 49 nodes 306 and 226; but 9 nodes 454 and 491, 64 nodes
//     (one CTA per SM) 277 and 315.
inline int combine_tile(int nb, int k, int npanels, int sms) {
    if (k < 64 || (k == 64 && npanels < 12 * sms)) return 32;
    if (2 * ((k + 63) / 64) == (k + 31) / 32) return 64;
    return combine_warps(nb, 64) > combine_warps(nb, 32) ? 64 : 32;
}

}  // namespace bie
