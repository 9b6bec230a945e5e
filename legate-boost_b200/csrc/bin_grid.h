// How many blocks share the rows of a table of the binning kernels (proposals.cu).
//
// A block fills the table of its features once and then walks over its share of the rows; the shares are equal.  So
// the kernel takes as many shares as there are waves of blocks, and a wave of a few blocks takes as long as a full one:
// 150 blocks on 148 SMs (three tables of 50 blocks) take twice the time of 147.  With the resident blocks divided by
// the tables and rounded up, and now: float32, 256 proposals: 10M x 96 1977 -> 1068 us, 10M x 160 3404 -> 1934, 10M x 256
// 5362 -> 2914, 2M x 512 2032 -> 1178, 200k x 75 54 -> 32; float64, 2M x 75 622 -> 425, 2M x 160 1032 -> 668.
#pragma once
#include <cstdint>

namespace lbk {

// Blocks per table.  resident: blocks that the device holds at once; fill_rows: rows that take a block as long as
// filling its table.  Of one to eight waves that are as full as whole blocks per table make them, the ones whose shares and tables
// come to the least: one wave as a rule; more where a wave of whole blocks per table leaves many places empty (15
// tables on 148 places: 135), and where the tables alone are more than one.
inline int64_t BinGridBlocks(int64_t rows, int64_t tables, int64_t resident, int64_t fill_rows)
{
  const int64_t most = rows > 64 ? (rows + 63) / 64 : 1;
  int64_t best = 1;
  double best_cost = 0.0;
  for (int w = 1; w <= 8; ++w) {
    int64_t blocks = w * resident / tables;
    if (blocks > most) blocks = most;
    if (blocks < 1) blocks = 1;
    const double waves = static_cast<double>((blocks * tables + resident - 1) / resident);
    const double cost  = waves * (static_cast<double>(rows) / static_cast<double>(blocks) + static_cast<double>(fill_rows));
    if (w == 1 || cost < 0.98 * best_cost) {
      best      = blocks;
      best_cost = cost;
    }
  }
  return best;
}

}  // namespace lbk
