// How the per-chain sums of columns.cuh are laid out over the chip: rules on sizes
// alone, so that they can be checked without a GPU.
#pragma once

#include <cstdint>

namespace hmc {

constexpr int COL_THREADS = 512;  // of a block at most

struct ColumnShape {
  int log_x;    // a tile holds 1 << log_x chains
  int cluster;  // blocks that share a tile's rows
  int threads;  // of a block
};

// Tile width: 32 chains (one 128-byte FP32 row segment per warp), or the next
// power of two for fewer chains, whose idle lanes then take rows instead.
// Threads: 512 where every lane gets two rows, fewer below, as idle warps only add
// to a block's barriers.  More tiles than two for every SM fill the chip by
// themselves, and 128 threads serve them best until their lanes' rows add
// up (d = 4, 100 000 chains: accept kernel 16 us against 52 with 512 threads and
// 24 in 8-warp blocks of 32 chains; d = 600, 20 000 chains: prior misfit 51 us with
// 128, 35 with 512).  narrow_until: the rows up to which that holds for a kernel (the
// accept kernel, which moves rows too, d = 300, 100 000 chains: 196 against 227 us).
// Cluster: doubled while the grid stays within one resident wave (two blocks on
// an SM) and every lane keeps four rows: a block sums, waits for the cluster and
// then moves rows, and a second wave pays these latencies again (a pass of two
// proposals of 20 steps, d = 1000, 4096 chains: 2052 us at up to 256 blocks, 2063
// at 512, 2113 at 1024, 2116 at 128); fewer than 32 chains of 64 rows and more spread
// over eight SMs, because a warp alone on its scheduler issues FP64 at half the SM's
// rate (d = 1000, one chain: momenta in 13 us on eight SMs,
// 418 us in one lane of one block's warps); below, one block is faster (d = 16, one
// FP64 chain: momenta 9.1 us, 11.0 on two SMs).
inline ColumnShape column_shape(int64_t C, int64_t rows, int64_t narrow_until = 64) {
  ColumnShape s{0, 1, 128};
  while (s.log_x < 5 && (1ll << s.log_x) < C) ++s.log_x;
  const int64_t tiles = (C + (1 << s.log_x) - 1) >> s.log_x;
  if (tiles > 2 * 152) {
    s.threads = rows <= narrow_until ? 128 : (rows <= 256 ? 256 : 512);
    return s;
  }
  while (s.threads < COL_THREADS && rows > 2 * (s.threads >> s.log_x)) s.threads *= 2;
  if (s.log_x < 5) {
    if (rows < 64) return s;
    s.threads = COL_THREADS;
    while (s.cluster < 8 && rows >= 16 * s.cluster) s.cluster *= 2;
  } else if (s.threads == COL_THREADS) {
    const int64_t lanes = COL_THREADS >> s.log_x;
    while (s.cluster < 8 && 2 * s.cluster * tiles <= 256 && rows >= 4 * lanes * 2 * s.cluster) s.cluster *= 2;
  }
  return s;
}

// How a thread of the kernels that update every element of a [d][C] array (kick and
// drift, prior gradients) takes them: 16 bytes of chains in one access or one chain,
// and up to `most` rows loaded together.  Both save accesses and repeated work per
// chain where the array fills the chip with threads, and leave it idle where it
// does not; FP64, whose instructions a scheduler issues every 64 cycles, wants more
// threads for as long as memory does not bound it.  40 rows, 512 FP64 chains: prior
// gradient 1.8 us with an element per thread, 3.0 with two chains and four rows; 1500 rows,
// 20 000 FP64 chains 148 us by chain and 131 by 16 bytes; 600 rows, 1024 FP32
// chains: kick and drift 5.8 us with an element, 2.7 with four chains and two rows.
struct ElementShape {
  bool vec;  // 16-byte accesses (only where every row allows them)
  int rows;
};
inline ElementShape element_shape(int64_t d, int64_t C, int element_bytes, bool aligned, int most) {
  const int per = 16 / element_bytes;
  const bool wide = element_bytes == 8;
  ElementShape s{aligned && C % per == 0 && d * C >= (wide ? 2000000 : 64000), wide && most > 2 ? 2 : most};
  const int64_t threads = d * C / (s.vec ? per : 1);
  while (s.rows > 1 && threads / s.rows < 40000) s.rows /= 2;
  return s;
}

}  // namespace hmc
