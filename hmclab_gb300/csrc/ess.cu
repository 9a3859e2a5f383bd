// Multi-chain effective sample size of every parameter, on the device.
//
// The reference has no ESS estimator (its only mixing diagnostic is
// Helpers/Processing.py:6-13, a numpy autocorrelation).  This follows the
// split-chain multi-chain estimator of Gelman et al., Bayesian Data Analysis
// (3rd ed., section 11.5) as used by Stan: every chain is split into two
// halves (M = 2C half-chains of n = N/2 draws), the lag-t autocorrelation is
//   rho_t = 1 - (W - mean_m gamma_{m,t}) / var+,
// with W the mean within-half-chain variance, var+ = (n-1)/n W + B/n, and the
// sum of rho is truncated by Geyer's initial monotone sequence (pairs
// rho_{2k} + rho_{2k+1} summed while positive, made non-increasing):
//   ESS = M n / (-1 + 2 sum_k P_k).
// Samples are laid out [N][d][C] (the sampler's ring), chain fastest.
#include "common.cuh"

namespace hmc {
namespace {

constexpr int ESS_CH = 32;    // half-chains per block (one per lane)
constexpr int ESS_LAGS = 8;    // lags a warp accumulates together
constexpr int ESS_WARPS = 8;   // warps per block at most
constexpr int ESS_FIRST = 8;   // lags of the first round

// Sum over the warp of eight values per lane, the eight totals left one per
// group of four lanes (lane 4 j holds the total of value j): 4 + 2 + 1 + 2 adds
// instead of 5 per value, as an FP64 add of a warp takes 16 cycles of its SM.
__device__ __forceinline__ double warp_sum8(const double v[ESS_LAGS], int lane) {
  double a[4], b[2], c;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const bool up = lane & 16;
    a[j] = (up ? v[j + 4] : v[j]) + __shfl_xor_sync(0xffffffffu, up ? v[j] : v[j + 4], 16);
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const bool up = lane & 8;
    b[j] = (up ? a[j + 2] : a[j]) + __shfl_xor_sync(0xffffffffu, up ? a[j] : a[j + 2], 8);
  }
  const bool up = lane & 4;
  c = (up ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, up ? b[0] : b[1], 4);
  c += __shfl_xor_sync(0xffffffffu, c, 2);
  c += __shfl_xor_sync(0xffffffffu, c, 1);
  return c;  // lane 4 j: total of value j = 4 (lane bit 16) + 2 (bit 8) + (bit 4)
}

// Per (parameter, block of half-chains), for the lags lag0 <= t < lag1:
// part[(i*nblk + b)*(lags+2) + ...] receives
//   [0] sum of half-chain means, [1] sum of squared means (round 0), [2 + t]
//   sum over half-chains of gamma_{m,t} (with 1/n normalisation).
// Parameters whose autocorrelation sum was truncated by an earlier round
// (done[i] > 0) are skipped: Geyer's sequence ends there, so no later lag
// enters their result.
//
// Bound by the FP64 pipe (1.7 lanes per cycle and SM measured), so the
// kernel spends it on the products alone: draws are converted and centred
// once (MODE 2: FP64 deviations in shared memory, up to ESS_DEV_MAX draws; MODE 1:
// FP32 draws staged, centred when read; MODE 0: read in place), a warp keeps
// eight lags of every half-chain in registers and slides one window of
// deviations past them, and lags are computed in rounds (8, 16, 32, ...)
// until every parameter has truncated.  600 parameters x 128 half-chains of
// 50 draws, 50 lags: 237 us in rounds of 8, 16 and 26 lags against 1242 us
// with one warp per block that converts and centres both factors of every
// product; the 98 M products of all lags alone would take 185 us.
template <typename T, int MODE>
__global__ void ess_lags_kernel(const T* __restrict__ x, int64_t d, int64_t C, int n, int lag0, int lag1, int lags,
                                double* __restrict__ part, const double* __restrict__ done) {
  extern __shared__ __align__(16) unsigned char ess_smem[];
  __shared__ double red[ESS_WARPS][ESS_CH];
  const int64_t i = blockIdx.y;
  if (lag0 > 0 && done[i] > 0.0) return;  // uniform over the block
  const int lane = threadIdx.x, w = threadIdx.y, W = blockDim.y;
  const int64_t M = 2 * C;
  const int64_t m = (int64_t)blockIdx.x * ESS_CH + lane;
  const bool live = m < M;
  const int64_t c = m % C, half = m / C;
  const T* __restrict__ src = x + (half * n * d + i) * C + c;
  const int64_t step = d * C;
  float* sf = (float*)ess_smem;    // MODE 1: [n][32]
  double* sd = (double*)ess_smem;  // MODE 2: [n][32]
  double sum = 0.0;
  for (int k = w; k < n; k += W) {
    const float v = live ? (float)src[k * step] : 0.f;
    const double v64 = f64_of(v);
    sum += v64;
    if (MODE == 1) sf[k * ESS_CH + lane] = v;
    if (MODE == 2) sd[k * ESS_CH + lane] = v64;
  }
  red[w][lane] = sum;
  __syncthreads();
  double mean = 0.0;
  for (int j = 0; j < W; ++j) mean += red[j][lane];
  mean /= n;
  if (MODE == 2) {
    for (int k = w; k < n; k += W) sd[k * ESS_CH + lane] -= mean;
    __syncthreads();
  }
  double* out = part + ((int64_t)i * gridDim.x + blockIdx.x) * (lags + 2);
  if (lag0 == 0 && w == 0) {
    double s1 = live ? mean : 0.0, s2 = s1 * s1;
    for (int o = 16; o > 0; o >>= 1) {
      s1 += __shfl_xor_sync(0xffffffffu, s1, o);
      s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    }
    if (lane == 0) {
      out[0] = s1;
      out[1] = s2;
    }
  }
  // the k-th deviation from the mean; zero past the end and for idle lanes
  auto dev = [&](int k) -> double {
    if (MODE == 2) return k < n ? sd[k * ESS_CH + lane] : 0.0;
    if (k >= n || !live) return 0.0;
    return f64_of(MODE == 1 ? sf[k * ESS_CH + lane] : (float)src[k * step]) - mean;
  };
  for (int t0 = lag0 + ESS_LAGS * w; t0 < lag1; t0 += ESS_LAGS * W) {
    double acc[ESS_LAGS], win[ESS_LAGS];
#pragma unroll
    for (int j = 0; j < ESS_LAGS; ++j) {
      acc[j] = 0.0;
      win[j] = dev(t0 + j);  // win[(k + j) % 8] = deviation k + t0 + j
    }
    for (int k0 = 0; k0 < n - t0; k0 += ESS_LAGS) {
#pragma unroll
      for (int u = 0; u < ESS_LAGS; ++u) {
        const double a = dev(k0 + u);
#pragma unroll
        for (int j = 0; j < ESS_LAGS; ++j) acc[j] = fma(a, win[(u + j) % ESS_LAGS], acc[j]);
        win[u] = dev(k0 + u + t0 + ESS_LAGS);
      }
    }
    const double total = warp_sum8(acc, lane);
    const int t = t0 + (lane >> 2);
    if ((lane & 3) == 0 && t < lag1) out[2 + t] = total / n;
  }
}

// One warp per parameter: combine the block partials of the lags computed so
// far and apply Geyer's truncation.  `last`: no round follows, so a window
// that did not truncate is reported (negative).
__global__ void ess_final_kernel(const double* __restrict__ part, int64_t d, int nblk, int64_t M, int n, int first,
                                 int known, int lags, int last, double* __restrict__ ess, double* __restrict__ rhat) {
  const int64_t i = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i >= d) return;
  if (!first && ess[i] > 0.0) return;  // truncated in an earlier round
  const int lane = threadIdx.x & 31;
  const double* p = part + i * nblk * (lags + 2);
  double smean = 0.0, smean2 = 0.0, W = 0.0;
  for (int b = lane; b < nblk; b += 32) {
    smean += p[b * (int64_t)(lags + 2)];
    smean2 += p[b * (int64_t)(lags + 2) + 1];
    W += p[b * (int64_t)(lags + 2) + 2];
  }
  for (int o = 16; o > 0; o >>= 1) {
    smean += __shfl_xor_sync(0xffffffffu, smean, o);
    smean2 += __shfl_xor_sync(0xffffffffu, smean2, o);
    W += __shfl_xor_sync(0xffffffffu, W, o);
  }
  W = W * n / (n - 1) / M;  // mean of the unbiased within-half-chain variances
  const double mu = smean / M;
  const double B = (double)n / (M - 1) * (smean2 - M * mu * mu);  // n * var of half-chain means
  const double varp = (n - 1.0) / n * W + B / n;
  if (rhat && lane == 0) rhat[i] = sqrt(varp / W);
  double tau_sum = 0.0, prev = INFINITY;
  bool truncated = false;
  for (int t0 = 0; t0 + 1 < known && !truncated; t0 += 32) {
    const int t = t0 + lane;
    double g = 0.0;
    if (t < known)
      for (int b = 0; b < nblk; ++b) g += p[b * (int64_t)(lags + 2) + 2 + t];
    const double rho = 1.0 - (W - g / M) / varp;
    const double pair = rho + __shfl_down_sync(0xffffffffu, rho, 1);
    for (int u = 0; u < 32 && t0 + u + 1 < known; u += 2) {
      double P = __shfl_sync(0xffffffffu, pair, u);
      if (P < 0.0) {
        truncated = true;
        break;
      }
      if (P > prev) P = prev;  // initial monotone sequence
      prev = P;
      tau_sum += P;
    }
  }
  if (lane != 0) return;
  if (!truncated && !last) {
    ess[i] = -1.0;  // another round follows
    return;
  }
  const double tau = -1.0 + 2.0 * tau_sum;
  double e = M * (double)n / tau;
  if (!truncated) e = -e;  // flag: lag window too short for this parameter
  ess[i] = e;
}

// Shared memory of the staged modes: FP64 deviations while two blocks fit an
// SM, FP32 draws up to the 1024 of the largest staged window, else in place.
constexpr int ESS_DEV_MAX = 384, ESS_DRAW_MAX = 1024;

template <typename T>
int ess_rounds(const T* x, int64_t N, int64_t d, int64_t C, int n, int lags, double* part, double* ess, double* rhat,
               cudaStream_t st) {
  const int nblk = (int)((2 * C + ESS_CH - 1) / ESS_CH);
  const int mode = n <= ESS_DEV_MAX ? 2 : (n <= ESS_DRAW_MAX ? 1 : 0);
  const size_t smem = mode == 2 ? (size_t)n * ESS_CH * 8 : (mode == 1 ? (size_t)n * ESS_CH * 4 : 0);
  auto kern = mode == 2 ? ess_lags_kernel<T, 2> : (mode == 1 ? ess_lags_kernel<T, 1> : ess_lags_kernel<T, 0>);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(ess_lags_kernel)");
  }
  for (int lag0 = 0, size = ESS_FIRST; lag0 < lags; size *= 2) {
    const int lag1 = lags - lag0 < 2 * size ? lags : lag0 + size;
    const int groups = (lag1 - lag0 + ESS_LAGS - 1) / ESS_LAGS;
    const dim3 block(ESS_CH, (unsigned)(groups < ESS_WARPS ? groups : ESS_WARPS));
    kern<<<dim3(nblk, (unsigned)d), block, smem, st>>>(x, d, C, n, lag0, lag1, lags, part, ess);
    HMC_TRY(check_launch("ess_lags_kernel"));
    ess_final_kernel<<<blocks_for(d, 4), 128, 0, st>>>(part, d, nblk, 2 * C, n, lag0 == 0, lag1, lags, lag1 == lags,
                                                     ess, rhat);
    HMC_TRY(check_launch("ess_final_kernel"));
    lag0 = lag1;
  }
  return HMC_OK;
}

}  // namespace
}  // namespace hmc

using namespace hmc;

extern "C" HMC_API int hmc_ess(int dtype, int64_t N, int64_t d, int64_t C, const void* samples, int lags,
                               double* work, double* ess, double* rhat, void* stream) {
  HMC_REQUIRE(N >= 4 && d > 0 && C > 0, "hmc_ess: need at least 4 draws, 1 parameter, 1 chain");
  HMC_REQUIRE(samples && work && ess, "hmc_ess: null argument");
  HMC_REQUIRE(N / 2 <= (1ll << 30), "hmc_ess: too many draws");
  const int n = (int)(N / 2);
  HMC_REQUIRE(lags >= 2 && lags <= n, "hmc_ess: lags must be in [2, N/2]");
  HMC_REQUIRE(d <= 65535, "hmc_ess: too many parameters for one call");
  HMC_REQUIRE((2 * C + ESS_CH - 1) / ESS_CH <= 0x7FFFFFFF, "hmc_ess: too many chains");
  return HMC_DISPATCH(dtype, T, [&] {
    return ess_rounds<T>((const T*)samples, N, d, C, n, lags, work, ess, rhat, as_stream(stream));
  });
}

namespace hmc {
namespace {
// Mean and variance over all draws and chains of every parameter: one block
// per parameter, fixed-order FP64 reduction.
template <typename T>
__global__ void moments_kernel(const T* __restrict__ x, int64_t N, int64_t d, int64_t C, double* mean, double* var) {
  __shared__ double s1[256], s2[256];
  const int64_t i = blockIdx.x;
  double a = 0.0, b = 0.0;
  const int64_t total = N * C;
  for (int64_t t = threadIdx.x; t < total; t += blockDim.x) {
    const int64_t n = t / C, c = t % C;
    const double v = f64_of(x[(n * d + i) * C + c]);
    a += v;
    b += v * v;
  }
  s1[threadIdx.x] = a;
  s2[threadIdx.x] = b;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      s1[threadIdx.x] += s1[threadIdx.x + w];
      s2[threadIdx.x] += s2[threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double m = s1[0] / total;
    mean[i] = m;
    var[i] = s2[0] / total - m * m;
  }
}
}  // namespace
}  // namespace hmc

extern "C" HMC_API int hmc_moments(int dtype, int64_t N, int64_t d, int64_t C, const void* samples, double* mean,
                                   double* var, void* stream) {
  HMC_REQUIRE(N > 0 && d > 0 && C > 0 && d <= 0x7FFFFFFF, "hmc_moments: bad sizes");
  HMC_REQUIRE(samples && mean && var, "hmc_moments: null argument");
  return HMC_DISPATCH(dtype, T, [&] {
    moments_kernel<T><<<(unsigned)d, 256, 0, as_stream(stream)>>>((const T*)samples, N, d, C, mean, var);
    return check_launch("moments_kernel");
  });
}

extern "C" HMC_API int64_t hmc_ess_work_size(int64_t d, int64_t C, int lags) {
  const int64_t nblk = (2 * C + ESS_CH - 1) / ESS_CH;
  return d * nblk * (lags + 2) + d * nblk;
}

// ---- rank normalisation (Vehtari, Gelman, Simpson, Carpenter & Buerkner
// 2021, "Rank-normalization, folding, and localization: an improved R-hat",
// section 4.1): every draw of a parameter is replaced by the normal score of
// its rank among all N x C draws of that parameter,
//   z = Phi^-1((r - 3/8) / (S + 1/4)),  S = N C,
// with tied draws given their average rank.  The split-R-hat and ESS of z are
// the bulk diagnostics of that paper.
namespace hmc {
namespace {
constexpr int RANK_V = 8;  // keys per thread of the sort (tiles of up to 1024 threads x 8)

// Draws as unsigned keys of the same order (-0 equals +0).  NaN compares with
// nothing: it takes the largest key, the padding's, which no draw is counted
// against.
template <typename T>
struct RankKey;
template <>
struct RankKey<float> {
  using K = uint32_t;
  static constexpr K top = 0xffffffffu;
  static __device__ __forceinline__ K of(float v) {
    if (isnan(v)) return top;
    const uint32_t b = __float_as_uint(v + 0.f);
    return b & 0x80000000u ? ~b : b | 0x80000000u;
  }
};
template <>
struct RankKey<double> {
  using K = unsigned long long;
  static constexpr K top = 0xffffffffffffffffull;
  static __device__ __forceinline__ K of(double v) {
    if (isnan(v)) return top;
    const unsigned long long b = (unsigned long long)__double_as_longlong(v + 0.0);
    return b >> 63 ? ~b : b | 0x8000000000000000ull;
  }
};

template <typename K>
__device__ __forceinline__ void rank_order(K& a, K& b, bool up) {
  if ((a > b) == up) {
    const K t = a;
    a = b;
    b = t;
  }
}

// Bitonic sort (Batcher 1968) of the block's RANK_V * blockDim.x keys, thread
// t holding the keys 8 t .. 8 t + 7: exchanges at distance < 8 stay in the
// thread's registers, < 256 in the warp's shuffles, and the rest go through
// shared memory.  blockDim.x is a power of two.
template <typename K>
__device__ __forceinline__ void rank_sort(K r[RANK_V], K* s) {
  const int t = threadIdx.x, T = blockDim.x;
  const int P = RANK_V * T;
  for (int size = 2; size <= P; size *= 2) {
    for (int dist = size / 2; dist >= RANK_V; dist /= 2) {
      const int td = dist / RANK_V;
      const bool keep_min = ((t & td) == 0) == ((RANK_V * t & size) == 0);
      if (td < 32) {
#pragma unroll
        for (int j = 0; j < RANK_V; ++j) {
          const K o = __shfl_xor_sync(0xffffffffu, r[j], td);
          r[j] = (o < r[j]) == keep_min ? o : r[j];
        }
      } else {
        __syncthreads();  // the previous exchange's reads are done
#pragma unroll
        for (int j = 0; j < RANK_V; ++j) s[j * T + t] = r[j];
        __syncthreads();
#pragma unroll
        for (int j = 0; j < RANK_V; ++j) {
          const K o = s[j * T + (t ^ td)];
          r[j] = (o < r[j]) == keep_min ? o : r[j];
        }
      }
    }
#pragma unroll
    for (int dist = RANK_V / 2; dist > 0; dist /= 2) {
      if (dist >= size) continue;
#pragma unroll
      for (int j = 0; j < RANK_V; ++j)
        if ((j & dist) == 0) rank_order(r[j], r[j | dist], ((RANK_V * t + j) & size) == 0);
    }
  }
}

// Number of sorted keys below k (upper: not above k); P a power of two.
template <typename K>
__device__ __forceinline__ int rank_bound(const K* s, int P, K k, bool upper) {
  int lo = 0;
  for (int w = P / 2; w > 0; w /= 2)
    if (upper ? s[lo + w - 1] <= k : s[lo + w - 1] < k) lo += w;
  return lo + (upper ? s[lo] <= k : s[lo] < k);
}

// Normal score of the rank r = r2 / 2 among S draws.
__device__ __forceinline__ double rank_score(uint32_t r2, double S) {
  return normcdfinv((0.5 * (double)r2 - 0.375) / (S + 0.25));
}

// Block (tile, parameter): sorts one tile of the parameter's draws and finds
// every draw of the parameter in it by binary search.  ONE tile holds all the
// draws of a run of up to 8192: the scores are written at once.  Otherwise the
// counts (draws below, low word; equal, high word) are added into the 64-bit
// words of z, exactly in any order, and rank_scores_kernel turns them into
// scores.  `scores` (nullable) holds the score of rank r at entry 2 r: the
// inverse normal distribution costs about a hundred FP64 instructions, and
// every parameter has the same S (or with ties 2 S) ranks.
template <typename T, bool ONE>
__global__ void __launch_bounds__(1024) rank_tiles_kernel(const T* __restrict__ x, int64_t d, uint32_t C, uint32_t S,
                                                          int64_t i0, const double* __restrict__ scores,
                                                          double* z) {
  using Key = RankKey<T>;
  using K = typename Key::K;
  extern __shared__ __align__(16) unsigned char rank_smem[];
  K* s = (K*)rank_smem;
  const int64_t i = i0 + blockIdx.y;
  const int t = threadIdx.x, nt = blockDim.x, P = RANK_V * nt;
  auto at = [&](uint32_t u) -> int64_t {
    const uint32_t n = u / C;
    return ((int64_t)n * d + i) * C + (u - n * C);
  };
  const uint32_t base = blockIdx.x * (uint32_t)P;
  K r[RANK_V];
#pragma unroll
  for (int j = 0; j < RANK_V; ++j) {
    const uint32_t u = base + (uint32_t)(j * nt + t);
    r[j] = u < S ? Key::of(x[at(u)]) : Key::top;
  }
  rank_sort(r, s);
  __syncthreads();
#pragma unroll
  for (int j = 0; j < RANK_V; ++j) s[RANK_V * t + j] = r[j];
  __syncthreads();
  for (uint32_t u = t; u < S; u += nt) {
    const int64_t o = at(u);
    const K k = Key::of(x[o]);
    int less = 0, equal = 0;
    if (k != Key::top) {
      less = rank_bound(s, P, k, false);
      if (less < P && s[less] == k)
        equal = less + 1 < P && s[less + 1] == k ? rank_bound(s, P, k, true) - less : 1;
    }
    if (ONE) {
      const uint32_t r2 = 2u * (uint32_t)less + (uint32_t)equal + 1u;
      z[o] = scores ? scores[r2] : rank_score(r2, (double)S);
    } else if (less | equal) {
      atomicAdd((unsigned long long*)z + o, (unsigned long long)less | ((unsigned long long)equal << 32));
    }
  }
}

__global__ void rank_scores_kernel(int64_t total, double S, const double* __restrict__ scores, double* z) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const unsigned long long w = ((const unsigned long long*)z)[e];
    const uint32_t r2 = 2u * (uint32_t)w + (uint32_t)(w >> 32) + 1u;
    z[e] = scores ? scores[r2] : rank_score(r2, S);
  }
}

__global__ void rank_table_kernel(int64_t entries, double S, double* scores) {
  const int64_t r2 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r2 < entries) scores[r2] = rank_score((uint32_t)r2, S);
}

// S draws per parameter cost S log^2 of a tile, where comparing each with each
// other cost S^2 FP64 comparisons: 600 parameters of 6400 draws take 156 us
// against 93.8 ms (535 us with every score computed from its rank).  The table
// pays from three parameters on (2 S scores against S d).
template <typename T>
int rank_normalize(int64_t N, int64_t d, int64_t C, const T* x, double* scores, double* z, cudaStream_t st) {
  const int64_t S = N * C;
  if (d <= 2) scores = nullptr;
  if (scores) {
    const int64_t entries = hmc_rank_scores_size(N, C);
    rank_table_kernel<<<blocks_for(entries, 128), 128, 0, st>>>(entries, (double)S, scores);
    HMC_TRY(check_launch("rank_table_kernel"));
  }
  int threads = 32;  // the smallest power of two whose tile holds the draws
  while (threads < 1024 && (int64_t)threads * RANK_V < S) threads *= 2;
  const int64_t tiles = (S + threads * RANK_V - 1) / (threads * RANK_V);
  const size_t smem = (size_t)threads * RANK_V * sizeof(typename RankKey<T>::K);
  auto kern = tiles == 1 ? rank_tiles_kernel<T, true> : rank_tiles_kernel<T, false>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(rank_tiles_kernel)");
  }
  if (tiles > 1) {
    cudaError_t e = cudaMemsetAsync(z, 0, (size_t)(S * d) * sizeof(double), st);
    if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync(rank counts)");
  }
  for (int64_t i0 = 0; i0 < d; i0 += 65535) {
    const unsigned dy = (unsigned)(d - i0 < 65535 ? d - i0 : 65535);
    kern<<<dim3((unsigned)tiles, dy), threads, smem, st>>>(x, d, (uint32_t)C, (uint32_t)S, i0, scores, z);
    HMC_TRY(check_launch("rank_tiles_kernel"));
  }
  if (tiles == 1) return HMC_OK;
  const unsigned g = blocks_for(S * d, 256) < 152u * 16u ? blocks_for(S * d, 256) : 152u * 16u;
  rank_scores_kernel<<<g, 256, 0, st>>>(S * d, (double)S, scores, z);
  return check_launch("rank_scores_kernel");
}
}  // namespace
}  // namespace hmc

extern "C" HMC_API int hmc_rank_normalize_table(int dtype, int64_t N, int64_t d, int64_t C, const void* samples,
                                                double* scores, double* z, void* stream) {
  HMC_REQUIRE(N > 0 && d > 0 && C > 0, "hmc_rank_normalize: bad sizes");
  HMC_REQUIRE(samples && z, "hmc_rank_normalize: null argument");
  const int64_t S = N * C;
  HMC_REQUIRE(S < (1ll << 31) / 2, "hmc_rank_normalize: too many draws per parameter");
  // the documented size limit of the entry point
  HMC_REQUIRE((double)S * (double)S * (double)d <= 1.1e12,
              "hmc_rank_normalize: S^2 d = %.3g is beyond this estimator's budget (1.1e12)",
              (double)S * (double)S * (double)d);
  return HMC_DISPATCH(dtype, T, [&] {
    return rank_normalize<T>(N, d, C, (const T*)samples, scores, z, as_stream(stream));
  });
}

extern "C" HMC_API int hmc_rank_normalize(int dtype, int64_t N, int64_t d, int64_t C, const void* samples, double* z,
                                          void* stream) {
  return hmc_rank_normalize_table(dtype, N, d, C, samples, nullptr, z, stream);
}

extern "C" HMC_API int64_t hmc_rank_scores_size(int64_t N, int64_t C) { return 2 * N * C + 2; }
