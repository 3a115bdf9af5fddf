// Which kernel and tile the expert GEMMs take: rules on sizes that the host knows, without a look at the device.
#pragma once
#include <algorithm>
#include <cmath>

#include "gemm_api.h"

namespace dx {

inline long long tiles_up(long long a, long long b) { return (a + b - 1) / b; }

// Whether FP8 with fp32 scales takes tiles of 256 columns instead of 128 (n % 256 == 0). Half as many tiles, each of which takes less than twice as
// long: it pays unless the narrow ones fill the SMs that much better. With q = rounds of wide tiles / rounds of narrow ones (0.5 with many, 1
// where both are dealt out at once), time wide / narrow over 9300 products of random sizes and routings, geometric mean and in brackets the worst tenth:
//
//   K blocks                                             1 to 3      4-7         8-15        16-31       32 on
//   whole groups, plain,  q 0.5                       1.04 (1.08) 0.98 (1.02) 0.93 (1.00) 0.87 (0.96) 0.80 (0.89)
//                         q 0.56 to 0.61              1.16        1.11        1.07        1.02        0.92
//                         q 1                         1.27        1.41        1.39        1.32        1.25
//   whole groups, SwiGLU, q 0.5                       1.01 (1.02) 1.00 (1.03) 0.96 (1.03) 0.91 (0.98) 0.86 (0.94)
//   ends given,   plain,  q 0.5, tiles full           1.04 (1.10) 0.97 (1.00) 0.89 (0.95) 0.83 (0.88) 0.75 (0.85)
//                         q 0.51 to 0.56, tiles full  1.06        1.01        0.93        0.88        0.78
//                         q 0.56 to 0.61, tiles full  1.14        1.08        1.01        0.94        0.86
//                         q 0.56 to 0.61, up to 24    0.92        0.89        0.91        0.93        0.89      rows in a tile
//                         q 0.61 to 0.68, up to 24    1.02        0.98        0.94        0.99        0.95
//   ends given,   SwiGLU, q 0.56 to 0.61              0.69        0.76        0.84        0.88        0.91
//                         q 0.61 to 0.68              0.77        0.84        0.87        0.96        0.99
//
// (With the ends of the groups given, warps without rows promote nothing.) A layout that has room for more rows than come (m_ends without
// rows_hint) says nothing about the tiles: where two of 32 experts are in use, 1.2 to 1.36, where all are, 0.5 to 1; it keeps the narrow ones.
inline bool wide_promotion(const GroupedGemmArgs& a) {
    const bool ends = a.m_ends != nullptr;
    if (a.cta_pairs || a.n % 256 != 0 || (ends && a.rows_hint <= 0)) return false;
    long long row_tiles = tiles_up(a.m_total, 128);
    if (a.rows_hint > 0) {
        // groups that get a row, each with half a tile to spare, but one tile at least
        const double groups = a.num_groups, used = groups * (1.0 - std::exp(-a.rows_hint / groups));
        row_tiles = std::min<long long>(row_tiles, std::max<long long>(1, (long long)(std::max(used, a.rows_hint / 128.0 + used / 2) + 0.5)));
    }
    const int kb = a.k / 128;
    double most;
    if (!ends) most = kb < 8 ? 0.0 : kb < 16 ? 0.53 : kb < 32 ? 0.56 : 0.6;
    else if (a.swiglu) most = 0.625;
    else if (a.rows_hint <= 48 * row_tiles) most = kb < 4 ? 0.58 : 0.625;
    else most = kb < 4 ? 0.0 : kb < 8 ? 0.51 : kb < 16 ? 0.56 : 0.6;
    auto pays = [&](long long rt) {
        const long long tiles = rt * (a.n / 256);
        return (double)tiles_up(tiles, a.num_sms) <= most * (double)tiles_up(2 * tiles, a.num_sms);
    };
    if (ends) return pays(row_tiles);
    // Without the ends nothing says whether every group is a whole number of tiles, fills a part of one (32 of 100 rows, K 1024: 32 tiles, not 25;
    // 38.9 / 46.5) or has half a tile to spare: it has to pay for each of them.
    return pays(row_tiles) && pays(std::max<long long>(row_tiles, std::min(a.num_groups, a.m_total))) && pays(row_tiles + a.num_groups / 2);
}

}  // namespace dx
