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
inline int tile_planes(int64_t nz, int64_t columns, int64_t ctas, int* tries = nullptr) {
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
    return planes;
}

}  // namespace rcb
