// FP64 sums over the rows of a [d][C] array, one per chain, for the kernels
// that draw, accept and weigh (momenta and K0, accept test, priors, residual
// norms).  A tile of 1 .. 32 chains belongs to a thread-block cluster: its
// blocks share the rows, reduce their part in shared memory and block 0 adds
// the parts through distributed shared memory, always in the same order, so
// results are bit-reproducible and no workspace is needed.
//
// With one block of 8 warps per 32 chains (before) a batch of 1024 chains
// occupied 32 SMs, and one chain a single lane per warp: at d = 4096 and 1024
// chains the accept kernel took 565 us for 67 MB of traffic.
#pragma once

#include <cooperative_groups.h>

#include "column_shape.cuh"
#include "common.cuh"

namespace hmc {

struct ColumnTile {
  int64_t c;   // this thread's chain
  int x;       // its place in the tile
  bool live;   // c < C
  bool first;  // the one thread per chain that holds the total
  int64_t row, rows;  // this thread's first row and the stride
};

__device__ __forceinline__ ColumnTile column_tile(const ColumnShape& s, int64_t C) {
  ColumnTile t;
  const int rank = (int)(blockIdx.x % (unsigned)s.cluster);
  t.x = threadIdx.x & ((1 << s.log_x) - 1);
  t.c = ((int64_t)(blockIdx.x / (unsigned)s.cluster) << s.log_x) + t.x;
  t.live = t.c < C;
  t.first = rank == 0 && (int)threadIdx.x < (1 << s.log_x);
  // consecutive rows go to different blocks, so few rows still use every SM
  t.row = (int64_t)(threadIdx.x >> s.log_x) * s.cluster + rank;
  t.rows = (int64_t)(s.threads >> s.log_x) * s.cluster;
  return t;
}

struct ColumnShared {
  double warp[COL_THREADS / 32][32];
  double block[32];
  int flag[32];
};

// Wait for all blocks of the tile (and order their shared-memory accesses).
__device__ __forceinline__ void column_sync(const ColumnShape& s) {
  if (s.cluster > 1)
    cooperative_groups::this_cluster().sync();
  else
    __syncthreads();
}

// Total of v over the rows of each chain; valid in the `first` threads.  The
// blocks' shared memory is read remotely: a column_sync has to follow before
// any block of the cluster exits.
__device__ __forceinline__ double column_total(const ColumnShape& s, double v, ColumnShared& sh) {
  const int X = 1 << s.log_x;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int o = 16; o >= X; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane < X) sh.warp[w][lane] = v;
  __syncthreads();
  double total = 0.0;
  if ((int)threadIdx.x < X) {
    for (int k = 0; k < s.threads / 32; ++k) total += sh.warp[k][threadIdx.x];
    sh.block[threadIdx.x] = total;
  }
  column_sync(s);
  if (s.cluster > 1 && blockIdx.x % (unsigned)s.cluster == 0 && (int)threadIdx.x < X) {
    for (int r = 1; r < s.cluster; ++r)
      total += *cooperative_groups::this_cluster().map_shared_rank(&sh.block[threadIdx.x], r);
  }
  return total;
}

// flag[x] of the tile's block `rank`.
__device__ __forceinline__ int column_flag(const ColumnShape& s, ColumnShared& sh, int x, int rank) {
  return s.cluster > 1 ? *cooperative_groups::this_cluster().map_shared_rank(&sh.flag[x], rank) : sh.flag[x];
}

template <typename... P, typename... A>
int launch_columns(const char* who, void (*kernel)(P...), const ColumnShape& s, int64_t C, cudaStream_t st, A... args) {
  const int64_t tiles = (C + (1 << s.log_x) - 1) >> s.log_x;
  HMC_REQUIRE(tiles * s.cluster <= 0x7FFFFFFF, "%s: too many chains", who);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * s.cluster));
  cfg.blockDim = dim3((unsigned)s.threads);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim = {(unsigned)s.cluster, 1, 1};
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
  if (e != cudaSuccess) return cuda_fail(e, who);
  return check_launch(who);
}

}  // namespace hmc
