// rc_tileplan.h -- how the tile kernels (rc_tile.cu) divide their columns of tiles into units. Plain C++.
#pragma once
#include <algorithm>
#include <cstdint>

namespace rcb {

// Planes per unit for `columns` columns of tiles of nz planes on `ctas` CTAs that take units in turn: the fewest turns x
// planes read (two more of x per unit, about the cost of one plane), down to four planes. Of the numbers of units per
// column that fill the same turns only the largest can be the best, and turns x 1.2 more than the planes per CTA is the
// least that any larger number costs, so few are tried (76 at most over 60,000 random sizes; 10^6 planes: 18). One by
// one, a step on 8 x 8 x 100,000 points spent 0.1 ms here.
inline int tile_planes(int64_t nz, int64_t columns, int64_t ctas, double* cost_out = nullptr, int* tries = nullptr) {
    const int64_t most = std::max<int64_t>(1, (nz + 3) / 4);
    double best = 1e300;
    int planes = (int)nz, n = 0;
    for (int64_t k = 1; k <= most; ++k) {
        const int64_t turns = (columns * k + ctas - 1) / ctas;
        if ((double)columns * nz / ctas + 1.2 * turns > best * (1.0 + 1e-12)) break;  // (ties are decided by rounding)
        k = std::max(k, std::min(most, turns * ctas / columns));
        const int64_t ml = (nz + k - 1) / k, units = columns * ((nz + ml - 1) / ml);
        const double cost = (double)((units + ctas - 1) / ctas) * (ml + 1.2);
        if (cost < best) {
            best = cost;
            planes = (int)ml;
        }
        ++n;
    }
    if (tries) *tries = n;
    if (cost_out) *cost_out = best;
    return planes;
}

// Whether 27-point tiles that read `planes` planes one after the other (turns x planes per unit) are faster than the
// gather runs on an FP64 block, or a bfloat16 one, of `bytes`. A plane takes a CTA 0.5 to 0.75 us whatever share of its
// tile lies in the grid, and the gather runs of 64 rows at least 50 to 110 us (bfloat16 75 to 250) and 1.1 to 2 us per MB
// (bfloat16 1.5 to 3.4). Narrow grids waste most of a tile. Filters of 10 steps, gather -> tiles, us: FP64
// 2 x 2 x 50,000 x 96 1892 -> 14,600, 2 x 2 x 2000 x 96 489 -> 649 and x 48 490 -> 349, 3 x 5 x 60,000 x 8 1886 -> 2317,
// 4 x 8 x 20,000 x 96 5850 -> 6771, 64 x 1 x 4000 x 96 2134 -> 2728 and x 24 924 -> 695, 6 x 6 x 6000 x 96 3406 -> 2131;
// bfloat16 steps and the residual block 2 x 2 x 50,000 x 48 874 -> 3098, 3 x 5 x 60,000 x 24 3086 -> 3470,
// 4 x 4 x 20,000 x 3 1544 -> 1103.
inline bool tile27_pays(bool bf16, double planes, double bytes) {
    const double mb = bytes / 1048576.0;
    return 0.58 * planes <= (bf16 ? std::max(100.0, 2.0 * mb) : std::max(65.0, 1.25 * mb));
}

}  // namespace rcb
