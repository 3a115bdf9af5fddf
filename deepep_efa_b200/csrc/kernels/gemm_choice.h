// Which kernel and tile the expert GEMMs take: rules on sizes that the host knows, without a look at the device.
#pragma once
#include <algorithm>
#include <cmath>

#include "gemm_api.h"

namespace dx {

inline long long tiles_up(long long a, long long b) { return (a + b - 1) / b; }

// Whether FP8 with fp32 scales takes tiles of 256 columns instead of 128 (n % 256 == 0). Half as many tiles, each of which takes less than twice as
// long: it pays unless the narrow ones fill the SMs that much better. With q = rounds of wide tiles / rounds of narrow ones (0.5 with many, 1
// where both are dealt out at once):
//
// Whole groups, time of the product wide / narrow over 3400 of random sizes, geometric mean and in brackets the worst tenth
//   K blocks                          1 to 3      4-7         8-15        16-31       32 on
//   plain,  q 0.5                   1.04 (1.08) 0.98 (1.02) 0.93 (1.00) 0.87 (0.96) 0.80 (0.89)
//           q 0.56 to 0.61          1.16        1.11        1.07        1.02        0.92
//           q 1                     1.27        1.41        1.39        1.32        1.25
//   SwiGLU, q 0.5                   1.01 (1.02) 1.00 (1.03) 0.96 (1.03) 0.91 (0.98) 0.86 (0.94)
//
// Ends given, change of a whole layer's time in per cent (1700 decode steps, fused and step-by-step layers of random sizes and routings)
//   q                               to 0.53   0.53-0.56   0.56-0.6   0.6-0.63   0.63-0.7   1
//   SwiGLU,  8 to 15 K blocks        -2.7      +0.1        +3.1       +5.0       +6.9     +13.8
//           16 to 31                 -3.4      -0.4        +2.3       +4.9       +8.5     +20.4
//           32 on                    -6.5      -2.8        -0.2       +2.7       +7.4     +20.0
//   plain,   4 to 7                  -4.0      -3.7        -2.3       -0.7       -0.1      +2.1
//            8 on                    -4.6      -3.7        -2.1       -1.6       -0.1      +3.7
//
// Alone, with plain tiles of one to three K blocks: 1.04 where they are full of rows, 0.9 with up to 24 rows in one. SwiGLU alone gains more than in
// a layer where the rows of the padding are not zero. A layout that has room for more rows than come (m_ends without rows_hint) says nothing about
// the tiles: where two of 32 experts are in use, 1.2 to 1.36, where all are, 0.5 to 1; it keeps the narrow ones.
inline bool wide_promotion(const GroupedGemmArgs& a) {
    const bool ends = a.m_ends != nullptr;
    if (a.narrow_promotion || a.cta_pairs || a.n % 256 != 0 || (ends && a.rows_hint <= 0)) return false;
    long long row_tiles = tiles_up(a.m_total, 128);
    if (a.rows_hint > 0) {
        // groups that get a row, each with half a tile to spare, but one tile at least
        const double groups = a.num_groups, used = groups * (1.0 - std::exp(-a.rows_hint / groups));
        row_tiles = std::min<long long>(row_tiles, std::max<long long>(1, (long long)(std::max(used, a.rows_hint / 128.0 + used / 2) + 0.5)));
    }
    const int kb = a.k / 128;
    double most;
    if (!ends) most = kb < 8 ? 0.0 : kb < 16 ? 0.53 : kb < 32 ? 0.56 : 0.6;
    else if (a.swiglu) most = kb < 16 ? 0.55 : kb < 32 ? 0.56 : 0.6;
    else if (a.rows_hint <= 48 * row_tiles) most = kb < 4 ? 0.58 : 0.67;
    else most = kb < 4 ? 0.0 : kb < 8 ? 0.58 : 0.625;
    auto pays = [&](long long rt) {
        const long long tiles = rt * (a.n / 256);
        return (double)tiles_up(tiles, a.num_sms) <= most * (double)tiles_up(2 * tiles, a.num_sms);
    };
    if (ends) return pays(row_tiles);
    // Without the ends nothing says whether every group is a whole number of tiles, fills a part of one (32 of 100 rows, K 1024: 32 tiles, not 25;
    // 38.9 / 46.5) or has half a tile to spare: it has to pay for each of them.
    return pays(row_tiles) && pays(std::max<long long>(row_tiles, std::min(a.num_groups, a.m_total))) && pays(row_tiles + a.num_groups / 2);
}

// BF16 products with tokens as rows: whether a CTA pair shares a tile of 256 of them. For weight gradients all but those that read their operands in
// place, which take pairs from 480 padded rows per expert on (with fewer the output is the work; both of 64 experts of 4096 -> 1408 in a loop, single / pair, us:
// 242 rows 779 / 818, 384 rows 1025 / 963, 512 rows 1266 / 1131; of 160 products of random sizes pairs take 1.04 to 1.4 of the time up to 370 padded rows, 0.94 to 1.1 from 390 to
// 470, 0.86 to 1.1 and 0.97 on average from 490 on); else where a pair's tile has little padding (first product of the same layer, 128 rows 255 / 316,
// 242 rows 346 / 329, 512 rows 689 / 565; in whole steps at the power limit 270 to 430 rows lose 2 to 8 %). With ends and no zeros behind them
// the number of rows is not known.
inline bool rows_on_pairs(const GroupedGemmArgs& a) {
    if (a.fp8 || a.num_sms < 2) return false;
    const double rows = (double)a.m_total / a.num_groups;
    if (a.mode == 1) return !a.a_mn || rows >= 480;
    return (a.m_ends == nullptr || a.zero_tail) && ((rows >= 224 && rows <= 270) || rows >= 430);
}

// BF16 forward products and input gradients: tokens of a tile where gemm_pairs.cu takes them as columns, 0 where they stay rows. Below about a
// tile of rows per expert tiles have 128 of them, which leaves room for eight stages instead of six.
//
// What decides is the K blocks (the columns' epilogue turns its output over, and few of them do not hide that), how the work of a round compares, and
// how many rounds there are. With s = rounds x tokens of the columns' tiles / rounds x features of the rows' tiles (1: the same number of
// products per SM), time columns / rows over 7250 products of random sizes and routings, geometric mean and in brackets the middle eight tenths:
//
//   K                                     320 to 512        576 to 704        768 to 960        1024 to 1216      1280 to 1728      1792 to 2496      2560 on
//   to 128 rows,  s < 0.8, one round   0.94 (.89 .99)    0.90 (.85 .95)    0.89 (.84 .94)    0.85 (.82 .89)    0.84 (.80 .88)    0.79 (.75 .84)    0.73 (.64 .80)
//                 s to 1.1, one        1.06 (1.0 1.1)    1.01 (.95 1.1)    1.00 (.93 1.0)    0.95 (.89 .99)    0.90 (.86 .95)    0.86 (.82 .90)    0.80 (.74 .86)
//                           two        1.09 (.91 1.2)    1.11 (.94 1.3)    1.05 (.88 1.2)    0.98 (.77 1.2)    0.92 (.81 1.1)    0.87 (.66 1.0)    0.91 (.70 1.1)
//                           more       1.13 (1.0 1.2)    1.01 (.91 1.1)    0.98 (.91 1.0)    0.98 (.91 1.1)    0.95 (.86 1.0)    0.94 (.87 1.0)    0.93 (.86 1.0)
//                 s above, one or two  1.26              1.20              -                 -                 -                 -                 0.99 (.86 1.3)
//                          more        1.20              1.10              1.02              1.06              0.99              0.98              0.92 (.87 1.1)
//   more rows,    s < 0.8              1.08 (.95 1.2)    0.99 (.90 1.1)    0.98 (.80 1.1)    1.00 (.89 1.1)    0.96 (.80 1.1)    0.91 (.82 1.0)    0.87 (.74 1.0)
//                 s to 1.1, one        1.03 (.92 1.1)    1.06 (.97 1.1)    1.01 (.95 1.1)    1.04 (.96 1.1)    1.02 (.95 1.1)    0.96 (.84 1.1)    0.94 (.83 1.0)
//                           two to 5   1.07 (.99 1.2)    0.98 (.87 1.1)    0.97 (.85 1.1)    0.98 (.89 1.0)    0.95 (.80 1.0)    0.92 (.75 1.0)    0.92 (.82 1.0)
//                           more       1.01 (.84 1.2)    0.92 (.79 1.0)    0.93 (.79 1.0)    0.92 (.80 1.0)    0.89 (.75 1.0)    0.86 (.70 1.0)    0.87 (.67 1.0)
//                 s above, one or two  1.25              1.19              1.19              1.12              1.12              1.07              1.03 (.89 1.2)
//                          more        1.12              0.97              -                 -                 -                 0.97              0.89 (.76 1.0)
//
// K below 320: 1.1 to 1.3 everywhere. In loops of 0.4 s at the power limit (94 products of more than 60 us) the rule takes 0.92 of the rows' time.
// Where ends are given without zeros behind them (a low-latency layout), how many rows come is not known: 0.70 to 0.95 from K 1280 on, but 1.2
// where tiles are many and an odd number of 128 features leaves half of one empty, and 1.1 at K 1024 with more than a round (64 groups, N 512: 16.1 / 17.9).
inline int token_columns(const GroupedGemmArgs& a) {
    if (a.mode != 0 || a.fp8 || a.swiglu || a.num_sms < 2 || a.n % 128 != 0 || a.k % 64 != 0 || a.m_total <= 0) return 0;
    const bool few = a.m_total <= 128ll * a.num_groups, unknown = a.m_ends != nullptr && !a.zero_tail;
    const int cap = few ? 128 : 256, pairs = a.num_sms / 2;
    // groups with rows: with zeros behind the ends every group is a whole number of 128
    const long long groups = unknown ? a.num_groups : std::max(1, std::min(a.num_groups, a.zero_tail ? a.m_total / 128 : a.m_total));
    const long long units = tiles_up(a.m_total, 32 * groups), per_group = tiles_up(units, cap / 32), feature_tiles = tiles_up(a.n, 256);
    const long long rounds = tiles_up(groups * per_group * feature_tiles, pairs);
    if (unknown) return (rounds == 1 ? a.k >= 1024 : a.k >= 1280 && (a.n % 256 == 0 || a.n >= 896)) ? cap : 0;
    const bool wide = a.n % 256 == 0 || (a.b_mn && a.n > 256);
    const long long row_cols = wide ? feature_tiles : a.n / 128, row_tiles = tiles_up(a.m_total, (rows_on_pairs(a) ? 256 : 128) * groups);
    const long long row_rounds = tiles_up(groups * row_tiles * row_cols, rows_on_pairs(a) ? pairs : a.num_sms);
    const double s = (double)(rounds * std::max(128ll, 32 * tiles_up(units, per_group))) / (double)(row_rounds * (wide ? 256 : 128));
    bool columns;
    if (s < 0.8) columns = a.k >= 1024;
    else if (s <= 1.1) columns = a.k >= 1792 || (few ? a.k >= 1024 && rounds != 2 : (a.k >= 1024 && rounds >= 2) || (a.k >= 576 && rounds >= 6));
    else columns = a.k >= 2560 && rounds >= 3;
    return columns ? cap : 0;
}

}  // namespace dx
