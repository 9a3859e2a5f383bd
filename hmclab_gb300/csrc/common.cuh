// Shared helpers of the hmclab_gb300 CUDA library: status handling, dtype
// dispatch, Philox4x32-10 and per-chain FP64 reductions over the [d][C]
// (dimension-major, chain-fastest) layout.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "hmclab_gb300.h"

namespace hmc {

// Records `msg` as the calling thread's last error and returns `code`.
int fail(int code, const char* fmt, ...);
// Maps a CUDA error to HMC_ERR_CUDA with the call site in the message.
int cuda_fail(cudaError_t e, const char* where);
// Counts launches issued by this library (reported to callers for audits).
void count_launch(int n = 1);

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// Limits of the bounded device waits, read by the launchers of the kernels
// that wait on tensor-copy barriers.  Production: 2 s, nothing withheld.
// hmc_set_wait_limits shortens the limit and makes block 0 of those kernels
// withhold its first barrier arrival, so a test can make a wait run out and
// check the status path without faulting or hanging the GPU.
struct WaitLimits {
  uint64_t ns;
  int withhold;
};
WaitLimits wait_limits();

// Check the launch that was just issued.
inline int check_launch(const char* where) {
  count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, where);
  return HMC_OK;
}

#define HMC_REQUIRE(cond, ...)                                   \
  do {                                                           \
    if (!(cond)) return ::hmc::fail(HMC_ERR_INVALID_ARG, __VA_ARGS__); \
  } while (0)

#define HMC_TRY(expr)            \
  do {                           \
    int _rc = (expr);            \
    if (_rc != HMC_OK) return _rc; \
  } while (0)

// Dispatch a templated launcher on the dtype code.
#define HMC_DISPATCH(dtype, T, ...)                                   \
  [&]() -> int {                                                      \
    if ((dtype) == HMC_F32) { using T = float; return __VA_ARGS__(); }  \
    if ((dtype) == HMC_F64) { using T = double; return __VA_ARGS__(); } \
    return ::hmc::fail(HMC_ERR_INVALID_ARG, "unknown dtype code %d", (int)(dtype)); \
  }()

// ---------------------------------------------------------------------------
// Philox4x32-10 (Salmon, Moraes, Dror, Shaw, "Parallel random numbers: as easy
// as 1, 2, 3", SC 2011): 10 rounds of the 4x32 multiply-xorshift round with
// the Weyl key schedule.
// ---------------------------------------------------------------------------
__host__ __device__ inline uint32_t mulhi32(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * (uint64_t)b) >> 32);
#endif
}

__host__ __device__ inline uint4 philox4x32_10(uint4 ctr, uint2 key) {
  const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u;
  const uint32_t W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    if (r > 0) {
      key.x += W0;
      key.y += W1;
    }
    const uint32_t hi0 = mulhi32(M0, ctr.x), lo0 = M0 * ctr.x;
    const uint32_t hi1 = mulhi32(M1, ctr.z), lo1 = M1 * ctr.z;
    ctr = make_uint4(hi1 ^ ctr.y ^ key.x, lo1, hi0 ^ ctr.w ^ key.y, lo0);
  }
  return ctr;
}

// Counter purposes: keep the momentum and scalar streams disjoint.
enum : uint32_t { PURPOSE_MOMENTUM = 0u, PURPOSE_SCALARS = 1u };

// Uniform in (0, 1) from 32 bits (never 0, never 1).
__device__ inline float u01f(uint32_t x) { return ((float)(x >> 8) + 0.5f) * (1.0f / 16777216.0f); }
// Uniform in (0, 1) with 53 bits from two words.
__device__ inline double u01d(uint32_t a, uint32_t b) {
  const uint64_t v = ((uint64_t)a << 21) ^ (uint64_t)(b >> 11);  // 53 bits
  return ((double)v + 0.5) * (1.0 / 9007199254740992.0);
}

// Four uniforms for (row quad, chain, proposal), and the two halves of
// Box-Muller: z = radius(u0) (cos, sin)(angle(u1)), radius(u2) (cos, sin)(angle(u3)).
template <typename T>
__device__ inline void philox_uniforms4(uint64_t seed, uint32_t quad, uint32_t chain, uint64_t proposal,
                                        uint32_t purpose, T u[4]);

template <>
__device__ inline void philox_uniforms4<float>(uint64_t seed, uint32_t quad, uint32_t chain, uint64_t proposal,
                                               uint32_t purpose, float u[4]) {
  const uint4 r = philox4x32_10(
      make_uint4(quad, chain, (uint32_t)proposal, ((uint32_t)(proposal >> 32) & 0x0FFFFFFFu) | (purpose << 28)),
      make_uint2((uint32_t)seed, (uint32_t)(seed >> 32)));
  u[0] = u01f(r.x);
  u[1] = u01f(r.y);
  u[2] = u01f(r.z);
  u[3] = u01f(r.w);
}

template <>
__device__ inline void philox_uniforms4<double>(uint64_t seed, uint32_t quad, uint32_t chain, uint64_t proposal,
                                                uint32_t purpose, double u[4]) {
  // Two Philox blocks give 53-bit uniforms for the FP64 verification mode.
  const uint2 key = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
  const uint32_t w = ((uint32_t)(proposal >> 32) & 0x07FFFFFFu) | (purpose << 28);
  const uint4 r0 = philox4x32_10(make_uint4(quad, chain, (uint32_t)proposal, w), key);
  const uint4 r1 = philox4x32_10(make_uint4(quad, chain, (uint32_t)proposal, w | 0x08000000u), key);
  u[0] = u01d(r0.x, r0.y);
  u[1] = u01d(r0.z, r0.w);
  u[2] = u01d(r1.x, r1.y);
  u[3] = u01d(r1.z, r1.w);
}

__device__ __forceinline__ float normal_radius(float u) { return sqrtf(-2.0f * logf(u)); }
__device__ __forceinline__ double normal_radius(double u) { return sqrt(-2.0 * log(u)); }
__device__ __forceinline__ void normal_angle(float u, float& c, float& s) {
  const float t = 6.283185307179586f * u;
  c = cosf(t);
  s = sinf(t);
}
__device__ __forceinline__ void normal_angle(double u, double& c, double& s) {
  const double t = 6.283185307179586 * u;
  c = cos(t);
  s = sin(t);
}

// Four standard normals for (row quad, chain, proposal) by Box-Muller.
template <typename T>
__device__ inline void philox_normal4(uint64_t seed, uint32_t quad, uint32_t chain, uint64_t proposal,
                                      uint32_t purpose, T out[4]) {
  T u[4], c, s;
  philox_uniforms4<T>(seed, quad, chain, proposal, purpose, u);
  const T a = normal_radius(u[0]), b = normal_radius(u[2]);
  normal_angle(u[1], c, s);
  out[0] = a * c;
  out[1] = a * s;
  normal_angle(u[3], c, s);
  out[2] = b * c;
  out[3] = b * s;
}

// Per-chain scalar uniforms for proposal n: step factor and accept uniform.
__device__ inline void philox_scalars(uint64_t seed, uint32_t chain, uint64_t proposal, double* u_eps,
                                      double* u_acc) {
  const uint4 r = philox4x32_10(
      make_uint4(0u, chain, (uint32_t)proposal,
                 ((uint32_t)(proposal >> 32) & 0x0FFFFFFFu) | (PURPOSE_SCALARS << 28)),
      make_uint2((uint32_t)seed, (uint32_t)(seed >> 32)));
  *u_eps = u01d(r.x, r.y);
  *u_acc = u01d(r.z, r.w);
}

// FP32 to FP64, exact.  The conversion instruction occupies the FP64 pipe (2
// lanes per cycle and SM measured, and for its full time when its predicate is
// false), so FP64 sums of FP32 terms spent most of their time converting.  The
// words are built with integer instructions at 64 lanes per cycle instead:
// exponent rebased by 1023 - 127, fraction shifted into the high word and the
// low; subnormals are scaled by 2^64 first, and zero, infinity and NaN keep
// their meaning.
__device__ __forceinline__ double f64_of(float v) {
  uint32_t b = __float_as_uint(v), add = 0x38000000u;
  if ((b & 0x7f800000u) - 0x00800000u >= 0x7f000000u) {
    if (b & 0x7f800000u) {
      add = 0x70000000u;  // infinity, NaN: exponent 255 becomes 2047
    } else {
      b = __float_as_uint(v * 18446744073709551616.f);
      add = (b & 0x7fffffffu) ? 0x34000000u : 0u;  // 2^64 less, or zero
    }
  }
  return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + add)), (int)(b << 29));
}
__device__ __forceinline__ double f64_of(double v) { return v; }

// (T)(coeff * (double)e).  An FP32 coefficient (1 and 1/2 of the leapfrog) makes
// the FP64 product exact, so its rounding to FP32 is the FP32 product.
template <typename T>
__device__ __forceinline__ T scaled_step(double coeff, bool single, T e) {
  return single ? (T)coeff * e : (T)(coeff * (double)e);
}
inline bool is_single(double coeff) { return (double)(float)coeff == coeff; }

// Short kernels that follow one another on a stream (the surrogates' training
// steps) overlap their launch latencies: each is launched with programmatic
// stream serialisation, lets its successor be set up at once, and touches memory
// only after its predecessors have completed.
__device__ __forceinline__ void chain_begin() {
  asm volatile("griddepcontrol.launch_dependents;" :::);
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <typename... P, typename... A>
int launch_chained(const char* who, void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
  if (e != cudaSuccess) return cuda_fail(e, who);
  return check_launch(who);
}

// sqrt of a mass: FP32 through the correctly rounded single-precision root,
// which equals the FP64 root rounded to FP32.
__device__ __forceinline__ float mass_root(float m) { return sqrtf(m); }
__device__ __forceinline__ double mass_root(double m) { return sqrt(m); }

// exp(dh) > u, the accept test, for dh = H0 - H1 (strict; NaN compares false).
// An FP64 exponential is some forty FP64 instructions at 64 cycles each; the
// FP32 one, within 1e-5 of the exact value for -80 < dh < 0 (its argument is
// rounded by up to 5e-6 and its own error is 2 ulp), settles every test whose
// sides differ by more than 1e-4.  The rest takes the FP64 test.
__device__ __forceinline__ bool accept_test(double dh, double u) {
  const float x = (float)dh, v = (float)u;
  if (x > -80.f && x < 80.f && v > 1e-30f && v < 0.999f) {
    const float a = expf(x);
    if (a * 0.9999f > v) return true;
    if (a * 1.0001f < v) return false;
  }
  return exp(dh) > u;
}

// ---------------------------------------------------------------------------
// Per-chain reductions over the [d][C] layout: a block owns 32 consecutive
// chains (threadIdx.x) and RY row lanes (threadIdx.y); rows are strided by RY
// and partial sums are combined in a fixed order, so results are
// bit-reproducible run to run.
// ---------------------------------------------------------------------------
constexpr int RED_X = 32;
constexpr int RED_Y = 8;

__device__ inline double block_chain_sum(double v, double (*sh)[RED_X + 1]) {
  sh[threadIdx.y][threadIdx.x] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.y == 0) {
#pragma unroll
    for (int y = 0; y < RED_Y; ++y) s += sh[y][threadIdx.x];
  }
  __syncthreads();
  return s;  // valid in row lane 0
}

inline dim3 red_grid(int64_t C) { return dim3((unsigned)((C + RED_X - 1) / RED_X)); }
inline dim3 red_block() { return dim3(RED_X, RED_Y); }

inline unsigned blocks_for(int64_t n, int threads) {
  int64_t b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > 0x7FFFFFFF) b = 0x7FFFFFFF;
  return (unsigned)b;
}

}  // namespace hmc
