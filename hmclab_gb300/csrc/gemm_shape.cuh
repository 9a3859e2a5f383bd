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

// FP64 products of up to 64 columns and 9664 rows (a tile of 64 x 64 for each SM at
// most): gemv_kernel (true) or gemm_kernel.  Both are bound by FP64 lanes.  A tile
// costs its SM 64 x 64 of them for each k, however few columns are real; the row
// kernel, over all SMs, one for each product of groups of eight columns, and for
// each such group of a row 5 x 8 adds of 32 lanes that sum over the warp.  Its factors were
// measured over 1000 .. 9700 rows, 5 .. 64 columns, k of 16 .. 4000: 1.2, and 1.7 where
// the rows of B are whole 128-byte lines and B exceeds an SM's L1 (a warp's loads
// of a column, one per row of B, then fall into few of its sets).  9000 rows, k = 60:
// 32 columns 137 us by rows and 76 us in tiles, 8 columns 37 and 76; 9000 x 1000, 64
// columns 1901 and 1203; 1000 x 1000, 64 columns 241 and 1134.  Up to four columns
// the row kernel was faster at every size.
inline bool f64_by_rows(int64_t m, int64_t n, int64_t k) {
  if (n > 64 || (m + 63) / 64 >= 152) return false;
  if (n <= 4) return true;
  const double factor = n % 16 == 0 && n * k > 16384 ? 1.7 : 1.2;
  const double lanes = factor * (double)m * (double)((n + 7) / 8 * 8) * 32.0 * (double)((k + 31) / 32 + 5);
  return lanes <= 152.0 * 64.0 * 64.0 * (double)((k + 15) / 16 * 16);
}

}  // namespace hmc
