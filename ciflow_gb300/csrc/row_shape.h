// Lanes and chunks of the row-per-group CRS matvecs (spmv.cu).
#pragma once

#include <cstdint>

namespace cigpu {

// Rows of a CRS: a determinant list's can differ by orders of magnitude (the reference
// determinant of a CISD list meets the whole list); a DOCI or FCI space's all have one
// length, but for the elements that vanish.
enum class RowKind { kList, kDoci, kFci };

struct RowShape {
    int lanes;   // lanes per row
    int chunks;  // chunks of four elements per lane and round
};

// FP64 products are bound by the FP64 pipe as much as by memory: a lane without an element
// in a round, and every step of a row's final sum, costs the pipe a full warp.
//   * mean rows of 48 chunks and more: 32 lanes, four chunks each; FCI rows two in FP64
//     (fewer registers: L=9 4a3b, 504 elements, 22.7 -> 18.6 us, L=8 4a4b 12.4 -> 11.3;
//     lists' uneven rows lose by it: 20.6 and 24.5 at 595);
//   * DOCI rows (18-36 chunks) in FP64 from 12,000 rows: 4 lanes. 8 | 4 lanes, among
//     others: L=16 8 pairs (12,870 rows) 8.3 | 8.2 us, L=17 8 pairs (24,310) 13.7 | 10.3,
//     L=18 9 pairs (48,620) 20.8 | 16.5, L=20 8 pairs (125,970) 52.9 | 41.1, L=40 4 pairs
//     (91,390) 55.4 | 42.7; L=14 (3,432), too few warps, 5.2 | 6.2;
//   * else 8 lanes, five chunks each (one round covers a DOCI row's 36). Lists too: the few
//     long rows of a list are chains of rounds, and 4 lanes would make each a chain five
//     times as long.
constexpr int64_t kFourLaneRows = 12000;

inline RowShape row_shape(int64_t n, int64_t nnz, bool fp64, RowKind kind) {
    const double chunks = n > 0 ? (double)nnz / n / 4.0 : 0;
    if (chunks >= 48) return {32, fp64 && kind == RowKind::kFci ? 2 : 4};
    if (fp64 && kind != RowKind::kList && n >= kFourLaneRows) return {4, 2};
    return {8, 5};
}

}  // namespace cigpu
