// Which tiles a tensor-core contraction takes (dense_tc.cu): a rule on sizes alone, so
// that it can be checked without a GPU.
#pragma once

#include <cstdint>

namespace hmc {
namespace tc {

constexpr int BM = 128;     // chains per tile (UMMA M)
constexpr int BN = 256;     // matrix rows per tile (UMMA N), many tiles
constexpr int BN_FEW = 32;  // the same where 256 would leave most SMs idle

// Tiles of 256 matrix rows read the operands least often; where they are so few
// that most SMs would idle, eight times as many of 32 rows (512 x 256 outputs,
// 512 products: 37 us with 4 wide tiles, 8.6 us with 32).  As long as every narrow
// tile has an SM of its own they are faster whatever the length of the products;
// when they need a second wave, only while latency is most of a tile's time (1024 x
// 1000 outputs, hi/lo split: 600 products 21.5 us wide and 18.8 narrow, 1000 products 26.7
// and 27.4, 4000 products 62.9 and 88.7; plain BF16, 4000 products at worst 48.7 and 62.8).
inline bool narrow_tiles(int64_t C, int64_t rows, int64_t K, int products) {
  const int64_t m = (C + BM - 1) / BM;
  if (m * ((rows + BN - 1) / BN) > 38) return false;
  return m * ((rows + BN_FEW - 1) / BN_FEW) <= 152 || K <= (products == 3 ? 768 : 2000);
}

}  // namespace tc
}  // namespace hmc
