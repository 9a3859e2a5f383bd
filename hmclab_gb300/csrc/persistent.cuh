// What the persistent kernels of small dense linear-Gaussian targets share: the
// views of a target and of its chains, and the launchers (persistent.cu tells
// which kernel runs when).
#pragma once

#include "common.cuh"

namespace hmc {
namespace pers {

constexpr int MAX_D = 128;
enum PriorKind { PRIOR_NONE = 0, PRIOR_NORMAL = 1, PRIOR_LAPLACE = 2 };

template <typename T>
struct Target {
  int d, ld;  // dimension, odd row stride of GtG in shared memory
  int prior;  // PriorKind
  const T* GtG;
  const T* Gtd0;
  double dtd;
  const T* pmean;
  const T* pw;
};

template <typename T>
struct State {
  int64_t C;
  int mass;  // HMC_MASS_*
  T* q_cur;
  double* x_cur;
  const T* eps;
  int64_t* accepted;
  const int64_t* control;
  uint64_t seed;
  int randomize;
  const T* mdiag;
  const T* minv;
  const T* mchol;      // FULL: lower Cholesky factor of M, [d][d]
  const T* mfull_inv;  // FULL: M^-1, [d][d]
  const T* sz;
  const T* seps;
  const double* su;
  int64_t slen;
  T* ring_q;
  double* ring_x;
  int64_t ring_slots, thin;
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <typename T>
__device__ __forceinline__ T sign_of(T x) {
  return x > (T)0 ? (T)1 : (x < (T)0 ? (T)-1 : (T)0);
}

// Standard normal for row i of chain c at proposal n: the injected stream or
// the Philox quad (i / 4) that the launch-per-step path draws.
template <typename T>
__device__ __forceinline__ T momentum_draw(const State<T>& s, int d, int i, int64_t c, int64_t n) {
  if (s.sz) return s.sz[((n % s.slen) * d + i) * s.C + c];
  T z[4];
  philox_normal4<T>(s.seed, (uint32_t)(i >> 2), (uint32_t)c, (uint64_t)n, PURPOSE_MOMENTUM, z);
  const int j = i & 3;  // select without a local-memory array index
  return j == 0 ? z[0] : (j == 1 ? z[1] : (j == 2 ? z[2] : z[3]));
}

// Copies a [d][d] matrix into shared memory with row stride ld.
template <typename T>
__device__ __forceinline__ void load_matrix(T* dst, const T* src, int d, int ld) {
  for (int e = threadIdx.x; e < d * d; e += blockDim.x) {
    const int r = e / d;
    dst[r * ld + (e - r * d)] = src[e];
  }
}

// The kernels for unit and diagonal mass.  single: every kick and drift
// coefficient is an FP32 value (scaled_step).
template <typename T>
int launch_lanes(const State<T>& st, const Target<T>& tg, const hmc_schedule& sch, int64_t nprop, int dry, bool single,
                 int chains, int groups, cudaStream_t stream);
template <typename T>
int launch_rows(const State<T>& st, const Target<T>& tg, const hmc_schedule& sch, int64_t nprop, int dry, bool single,
                int cluster, cudaStream_t stream);
}  // namespace pers
}  // namespace hmc
