// Which kernel a product runs on, and its blocks: rules on sizes alone, so that
// they can be checked without a GPU.
#pragma once

#include <cstdint>
#include <initializer_list>

namespace hmc {

// Rows per thread of gemm_f32_kernel for more than four columns (a block owns
// sixteen times as many, and 32 columns), the choice with the least padding; 0:
// gemm_kernel, whose offsets have 64 bits.  A block of gemm_f32_kernel keeps 32-bit
// offsets from its first row of A, so its rows times k have to stay below 2^32; a
// grid has at most 65535 blocks of rows.
// Two rows per thread spend 6 loads on 32 multiply-adds where four spend 8 on 64,
// so they pay where blocks are what is missing, or where they save more than a
// tenth of the rows: with two blocks of 64 rows for every SM, 20 000 rows, 1024
// columns, k = 60 take 129 us with two rows per thread, 115 us in the 64 x 64 tiles
// of gemm_kernel and 87 us with nine; below, 2080 rows, 200 columns 6.2 us with two
// and 8.2 us with six.  (Of 396 products of 33 to 100 000 rows none is slower by this
// rule than by padding alone, the mean is 5 % faster.)
constexpr int F32_FEW_COLUMNS = 4, F32_FEW_ROWS = 64;  // up to four columns: 64 rows, a thread each
constexpr int64_t GRID_ROWS = 65535;
inline bool f32_offsets_fit(int64_t rows, int64_t k) { return k < (int64_t)0xffffffff / rows; }
inline int f32_rows_per_thread(int64_t m, int64_t n, int64_t k) {
  int rpt = 0;
  int64_t least = 0;
  for (int r : {9, 8, 6, 4, 2}) {
    const int64_t blocks = (m + 16 * r - 1) / (16 * r), padded = blocks * (16 * r);
    if (!f32_offsets_fit(16 * r, k) || blocks > GRID_ROWS) continue;
    if (r == 2 && rpt != 0 && (m + 63) / 64 * ((n + 31) / 32) >= 2 * 152 && 10 * least <= 11 * padded) continue;
    if (rpt == 0 || padded < least) rpt = r, least = padded;
  }
  return rpt;
}

}  // namespace hmc
