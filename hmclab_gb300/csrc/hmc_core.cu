// Batched HMC trajectory kernels: momentum draw + first drift, kick/drift
// steps, and the FP64 Metropolis accept with thinned sample recording.
//
// Semantics follow the reference sampler (larsgeb/hmclab):
//   momentum   MassMatrices.py:135-142 (Unit), 220-227 (Diagonal), 307-314 (Full)
//   K, dK/dp   MassMatrices.py:100-133, 185-218, 270-305
//   leapfrog   Samplers.py:1524-1584 (position Verlet: drift-kick-drift)
//   corrector  Distributions/base.py:239-270 (reflect at bounds, flip p)
//   accept     Samplers.py:1471-1492 (exp(H0 - H1) > u, strict, NaN rejects)
//   autotune   Samplers.py:1494-1522
//   append     Samplers.py:675-678 (thinned vstack([q, x]))
#include <math.h>

#include <type_traits>

#include "columns.cuh"

namespace hmc {
int gemm_dispatch(int dtype, int64_t m, int64_t n, int64_t k, double alpha, const void* A, const void* B,
                  const void* bias, void* out, int accumulate, cudaStream_t stream);
}

namespace hmc {
namespace {

template <typename T>
struct ChainView {
  int64_t d, C;
  T* q_cur;
  T* q;
  T* p;
  const T* g;
  T* v;
  const T* mdiag;
  const T* minv;
  const T* lo;
  const T* hi;
  T* eps;
  T* eps_local;
  double* x_cur;
  double* x_prop;
  double* k_cur;
  double* k_prop;
  int64_t* accepted;
  int32_t* flags;
  int64_t* control;  // [0] proposal counter, [1] block arrival counter
  uint64_t seed;
  int randomize;
  int autotune;
  double target, kappa, min_eps;
  const T* sz;
  const T* seps;
  const double* su;
  int64_t slen;
  T* ring_q;
  double* ring_x;
  int64_t ring_slots, thin;
  double* rec_eps;
  double* rec_acc;
  int64_t rec_len;
  const double* beta;  // per-chain inverse temperature, nullptr = 1
};

template <typename T>
ChainView<T> view(const hmc_chains* s) {
  ChainView<T> v;
  v.d = s->dims;
  v.C = s->chains;
  v.q_cur = (T*)s->q_cur;
  v.q = (T*)s->q;
  v.p = (T*)s->p;
  v.g = (const T*)s->g;
  v.v = (T*)s->v;
  v.mdiag = (const T*)s->mass_diag;
  v.minv = (const T*)s->mass_inv_diag;
  v.lo = (const T*)s->lower;
  v.hi = (const T*)s->upper;
  v.eps = (T*)s->eps;
  v.eps_local = (T*)s->eps_local;
  v.x_cur = s->x_cur;
  v.x_prop = s->x_prop;
  v.k_cur = s->k_cur;
  v.k_prop = s->k_prop;
  v.accepted = s->accepted;
  v.flags = s->flags;
  v.control = s->proposal;
  v.seed = s->seed;
  v.randomize = s->randomize_stepsize;
  v.autotune = s->autotune;
  v.target = s->target_acceptance;
  v.kappa = s->learning_rate;
  v.min_eps = s->minimal_stepsize;
  v.sz = (const T*)s->stream_z;
  v.seps = (const T*)s->stream_eps;
  v.su = s->stream_u;
  v.slen = s->stream_len;
  v.ring_q = (T*)s->ring_q;
  v.ring_x = s->ring_x;
  v.ring_slots = s->ring_slots;
  v.thin = s->thinning;
  v.rec_eps = s->rec_stepsize;
  v.rec_acc = s->rec_acceptance;
  v.rec_len = s->rec_len;
  v.beta = s->beta;
  return v;
}

// M^-1 p for one element; FULL reads the precomputed product from v.
template <typename T, int MASS>
__device__ __forceinline__ T minv_p(const ChainView<T>& s, int64_t i, int64_t idx, T p) {
  if (MASS == HMC_MASS_UNIT) return p;
  if (MASS == HMC_MASS_DIAG) return s.minv[i] * p;
  return s.v[idx];
}

// Reflection of base.py:239-270 (lower bound first, then upper); returns
// true when the position is still outside after the reflection.
template <typename T>
__device__ __forceinline__ bool reflect(const ChainView<T>& s, int64_t i, T& q, T& p) {
  bool out = false;
  if (s.lo) {
    const T lb = s.lo[i];
    if (q < lb) {
      q += (T)2 * (lb - q);
      p = -p;
    }
  }
  if (s.hi) {
    const T ub = s.hi[i];
    if (q > ub) {
      q += (T)2 * (ub - q);
      p = -p;
    }
  }
  if (s.lo && q < s.lo[i]) out = true;
  if (s.hi && q > s.hi[i]) out = true;
  return out;
}

template <typename T>
__device__ __forceinline__ T step_factor(const ChainView<T>& s, int64_t c, int64_t n) {
  if (s.seps) return s.seps[(n % s.slen) * s.C + c];
  double ue, ua;
  philox_scalars(s.seed, (uint32_t)c, (uint64_t)n, &ue, &ua);
  return (T)(0.5 + ue);
}

template <typename T>
__device__ __forceinline__ void draw_z4(const ChainView<T>& s, int64_t quad, int64_t c, int64_t n, T z[4]) {
  if (s.sz) {
    const T* base = s.sz + (n % s.slen) * s.d * s.C;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t i = 4 * quad + j;
      z[j] = i < s.d ? base[i * s.C + c] : (T)0;
    }
  } else {
    philox_normal4<T>(s.seed, (uint32_t)quad, (uint32_t)c, (uint64_t)n, PURPOSE_MOMENTUM, z);
  }
}

// FULL mass, step 1: z -> v (the host then forms p = L z and v = M^-1 p).
template <typename T>
__global__ void draw_z_kernel(ChainView<T> s) {
  const int64_t n = s.control[0];
  const int64_t quads = (s.d + 3) / 4;
  const int64_t total = quads * s.C;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = t % s.C, qd = t / s.C;
    T z[4];
    draw_z4(s, qd, c, n, z);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t i = 4 * qd + j;
      if (i < s.d) s.v[i * s.C + c] = z[j];
    }
  }
}

// Momentum (UNIT/DIAG; FULL has p and v = M^-1 p already), K0 in FP64, step
// size of this trajectory, first drift and reflection.  Bound by issue (Philox
// and Box-Muller, 43 % ALU) once the step size is formed once per chain and
// block and the mass's root in FP32: d = 4096, 1024 chains, diagonal mass,
// cold cache: 36 us against 561 us with one 8-warp block per 32 chains and an
// FP64 root and three conversions per element.
template <typename T, int MASS>
__global__ void __launch_bounds__(COL_THREADS) begin_kernel(ChainView<T> s, double drift, bool single,
                                                            ColumnShape shape) {
  __shared__ ColumnShared sh;
  __shared__ T step[32], first_drift[32];
  const ColumnTile t = column_tile(shape, s.C);
  const int64_t n = s.control[0], c = t.c;
  if ((int)threadIdx.x < (1 << shape.log_x)) {
    T e = (T)0;
    if (t.live) {
      e = s.eps[c];
      if (s.randomize) e *= step_factor(s, c, n);  // the FP64 product of two T rounds to the product in T
    }
    step[t.x] = e;
    first_drift[t.x] = scaled_step(drift, single, e);  // (drift * eps), then times M^-1 p
    sh.flag[t.x] = 0;
  }
  __syncthreads();
  const T e = step[t.x], ce = first_drift[t.x];
  double k = 0.0;
  bool oob = false;
  if (t.live) {
    if (MASS == HMC_MASS_FULL) {
      for (int64_t i = t.row; i < s.d; i += t.rows) {
        const int64_t idx = i * s.C + c;
        T p = s.p[idx];
        const T mp = s.v[idx];
        k += f64_of(p) * f64_of(mp);
        T q = s.q_cur[idx] + ce * mp;
        oob |= reflect(s, i, q, p);
        s.q[idx] = q;
        s.p[idx] = p;
      }
    } else {
      const int64_t quads = (s.d + 3) / 4;
      for (int64_t qd = t.row; qd < quads; qd += t.rows) {
        const int64_t i0 = 4 * qd, k0 = i0 * s.C + c;
        T qc[4], z[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) qc[j] = i0 + j < s.d ? s.q_cur[k0 + j * s.C] : (T)0;
        draw_z4(s, qd, c, n, z);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int64_t i = i0 + j;
          if (i < s.d) {
            const int64_t idx = k0 + j * s.C;
            T p = MASS == HMC_MASS_DIAG ? mass_root(s.mdiag[i]) * z[j] : z[j];
            const T mp = minv_p<T, MASS>(s, i, idx, p);
            k += f64_of(p) * f64_of(mp);
            T q = qc[j] + ce * mp;
            oob |= reflect(s, i, q, p);
            s.q[idx] = q;
            s.p[idx] = p;
          }
        }
      }
    }
  }
  if (oob) atomicOr(&sh.flag[t.x], 1);
  const double ksum = column_total(shape, k, sh);  // orders the flags too
  if (t.first && t.live) {
    int out = 0;
    for (int r = 0; r < shape.cluster; ++r) out |= column_flag(shape, sh, t.x, r);
    s.k_cur[c] = 0.5 * ksum;
    s.eps_local[c] = e;
    s.flags[c] = out ? HMC_FLAG_OUT_OF_BOUNDS : 0;
  }
  if (shape.cluster > 1) column_sync(shape);
}

// VEC consecutive chains in one access of 16 bytes.
template <typename T, int VEC>
struct alignas(sizeof(T) * VEC) Pack {
  T v[VEC];
};
constexpr int KICK_ROWS = 2;  // rows of a thread loaded together

// p -= kick * eps * g; q += drift * eps * M^-1 p; reflect.  For FULL the kick
// and the drift are split around the host-issued v = M^-1 p product.  A thread
// owns VEC chains and walks rows, so the step sizes and the index arithmetic
// are paid per chain instead of per element (where FP64 products and 64-bit
// divisions bounded it); d = 4096, 1024 chains, cold
// cache: 15 us for 84 MB (5.6 TB/s) against 41 us.
template <typename T, int MASS, int DO_KICK, int DO_DRIFT, int VEC>
__global__ void __launch_bounds__(256, 4) kick_drift_kernel(ChainView<T> s, double kick, double drift, bool single) {
  using V = Pack<T, VEC>;
  const int64_t c = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) * VEC;
  if (c >= s.C) return;
  T ck[VEC], cd[VEC];
#pragma unroll
  for (int v = 0; v < VEC; ++v) {
    const T e = s.eps_local[c + v];
    if (DO_KICK) ck[v] = s.beta ? (T)(kick * (double)e * s.beta[c + v]) : scaled_step(kick, single, e);
    if (DO_DRIFT) cd[v] = scaled_step(drift, single, e);
  }
  const int64_t stride = (int64_t)gridDim.y * blockDim.y;
  for (int64_t r0 = blockIdx.y * (int64_t)blockDim.y + threadIdx.y; r0 < s.d; r0 += KICK_ROWS * stride) {
    V p[KICK_ROWS], q[KICK_ROWS], w[KICK_ROWS];  // w: the gradient, or v = M^-1 p of a full mass
#pragma unroll
    for (int u = 0; u < KICK_ROWS; ++u) {
      const int64_t i = r0 + u * stride;
      if (i >= s.d) break;
      const int64_t idx = i * s.C + c;
      p[u] = *(const V*)(s.p + idx);
      if (DO_KICK) w[u] = *(const V*)(s.g + idx);
      if (DO_DRIFT) q[u] = *(const V*)(s.q + idx);
      if (DO_DRIFT && MASS == HMC_MASS_FULL) w[u] = *(const V*)(s.v + idx);
    }
#pragma unroll
    for (int u = 0; u < KICK_ROWS; ++u) {
      const int64_t i = r0 + u * stride;
      if (i >= s.d) break;
      const int64_t idx = i * s.C + c;
      const T mi = DO_DRIFT && MASS == HMC_MASS_DIAG ? s.minv[i] : (T)1;
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        if (DO_KICK) p[u].v[v] -= ck[v] * w[u].v[v];
        if (DO_DRIFT) {
          const T mp = MASS == HMC_MASS_FULL ? w[u].v[v] : (MASS == HMC_MASS_DIAG ? mi * p[u].v[v] : p[u].v[v]);
          q[u].v[v] = q[u].v[v] + cd[v] * mp;
          if (s.lo || s.hi) {
            if (reflect(s, i, q[u].v[v], p[u].v[v])) atomicOr(&s.flags[c + v], HMC_FLAG_OUT_OF_BOUNDS);
          }
        }
      }
      if (DO_DRIFT) *(V*)(s.q + idx) = q[u];
      if (DO_KICK || s.lo || s.hi) *(V*)(s.p + idx) = p[u];
    }
  }
}

// FP64 kinetic energy of p (MASS != FULL) or of (p, v = M^-1 p) (FULL).
template <typename T, int MASS>
__device__ __forceinline__ double kinetic_partial(const ChainView<T>& s, const T* __restrict__ p,
                                                  const T* __restrict__ mp_full, const ColumnTile& t) {
  double k = 0.0;
#pragma unroll 8
  for (int64_t i = t.row; i < s.d; i += t.rows) {
    const int64_t idx = i * s.C + t.c;
    const T pi = p[idx];
    const T mp = MASS == HMC_MASS_UNIT ? pi : (MASS == HMC_MASS_DIAG ? s.minv[i] * pi : mp_full[idx]);
    k += f64_of(pi) * f64_of(mp);
  }
  return k;
}

template <typename T, int MASS>
__global__ void __launch_bounds__(COL_THREADS) kinetic_kernel(ChainView<T> s, const T* p, const T* mp_full, double* out,
                                                              ColumnShape shape) {
  __shared__ ColumnShared sh;
  const ColumnTile t = column_tile(shape, s.C);
  const double ks = column_total(shape, t.live ? kinetic_partial<T, MASS>(s, p, mp_full, t) : 0.0, sh);
  if (t.first && t.live) out[t.c] = 0.5 * ks;
  if (shape.cluster > 1) column_sync(shape);
}

// K1, the accept test (FP64, one thread per chain), and the accepted or kept
// position into q_cur and the sample ring.  Bound by memory latency; d = 4096,
// 1024 chains, cold cache: 37 us against 565 us.  The test's operands are loaded
// while the rows are summed, and without step-size adaptation it needs alpha only
// to the side of u it falls on (accept_test).
template <typename T, int MASS>
__global__ void __launch_bounds__(COL_THREADS) end_kernel(ChainView<T> s, ColumnShape shape) {
  __shared__ ColumnShared sh;
  const ColumnTile t = column_tile(shape, s.C);
  const int64_t c = t.c;
  const int64_t n = s.control[0];
  // what the accept test needs besides K1, loaded while the rows are summed
  double x0 = 0.0, x1 = 0.0, k0 = 0.0, b = 1.0, u = 0.0;
  if (t.first && t.live) {
    x0 = s.x_cur[c];
    x1 = s.x_prop[c];
    k0 = s.k_cur[c];
    if (s.beta) b = s.beta[c];
    if (s.flags[c] & HMC_FLAG_OUT_OF_BOUNDS) {
      x1 = INFINITY;
      s.x_prop[c] = x1;
    }
    if (s.su) {
      u = s.su[(n % s.slen) * s.C + c];
    } else {
      double ue;
      philox_scalars(s.seed, (uint32_t)c, (uint64_t)n, &ue, &u);
    }
  }
  const double ks = column_total(shape, t.live ? kinetic_partial<T, MASS>(s, s.p, s.v, t) : 0.0, sh);
  if (t.first) {
    int accept = 0;
    if (t.live) {
      const double k1 = 0.5 * ks;
      s.k_prop[c] = k1;
      const double h0 = (s.beta ? b * x0 : x0) + k0;
      const double h1 = (s.beta ? b * x1 : x1) + k1;
      if (s.autotune) {
        const double alpha = exp(h0 - h1);
        const T eps_now = s.eps[c];
        if (s.rec_eps && n < s.rec_len) {
          s.rec_eps[n * s.C + c] = (double)eps_now;
          s.rec_acc[n * s.C + c] = alpha;
        }
        const double w = pow((double)(n + 1), -s.kappa);
        const double a = isnan(alpha) ? 0.0 : alpha;
        double e = (double)eps_now - w * (s.target - fmin(a, 1.0));
        if (e <= 0.0) e = fmax(e, s.min_eps);
        s.eps[c] = (T)e;
        accept = alpha > u ? 1 : 0;  // strict; NaN compares false
      } else {
        accept = accept_test(h0 - h1, u) ? 1 : 0;
      }
      if (accept) {
        s.x_cur[c] = x1;
        s.accepted[c] += 1;
      }
    }
    sh.flag[t.x] = accept;
  }
  column_sync(shape);
  const bool record = s.ring_q != nullptr && (n % s.thin) == 0;
  const int64_t slot = record ? (n / s.thin) % s.ring_slots : 0;
  const bool acc = column_flag(shape, sh, t.x, 0) != 0;
  if (t.live && (acc || record)) {
    const T* __restrict__ from = acc ? s.q : s.q_cur;
    T* ring = record ? s.ring_q + slot * s.d * s.C : nullptr;
    constexpr int U = 8;  // rows loaded together
    for (int64_t i0 = t.row; i0 < s.d; i0 += U * t.rows) {
      T qv[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t i = i0 + u * t.rows;
        if (i < s.d) qv[u] = from[i * s.C + c];
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t i = i0 + u * t.rows;
        if (i >= s.d) break;
        if (acc) s.q_cur[i * s.C + c] = qv[u];
        if (record) ring[i * s.C + c] = qv[u];
      }
    }
  }
  if (record && t.first && t.live) s.ring_x[slot * s.C + c] = s.beta ? s.beta[c] * s.x_cur[c] : s.x_cur[c];
  // The last block to finish advances the proposal counter.
  __threadfence();
  column_sync(shape);  // and no block of the tile leaves while its flags are read
  if (threadIdx.x == 0) {
    const unsigned long long prev = atomicAdd((unsigned long long*)&s.control[1], 1ull);
    if (prev == (unsigned long long)(gridDim.x - 1)) {
      s.control[0] = n + 1;
      s.control[1] = 0;
      __threadfence();
    }
  }
}

template <typename T>
int check_state(const hmc_chains* s, const char* who) {
  HMC_REQUIRE(s != nullptr, "%s: null state", who);
  HMC_REQUIRE(s->dims > 0 && s->chains > 0, "%s: dims and chains must be positive", who);
  HMC_REQUIRE(s->chains <= 0xFFFFFFFFll, "%s: too many chains", who);
  HMC_REQUIRE(s->q_cur && s->q && s->p && s->eps && s->eps_local && s->x_cur && s->x_prop && s->k_cur &&
                  s->k_prop && s->accepted && s->flags && s->proposal,
              "%s: missing state buffer", who);
  HMC_REQUIRE(s->mass_kind >= HMC_MASS_UNIT && s->mass_kind <= HMC_MASS_FULL, "%s: bad mass kind", who);
  if (s->mass_kind == HMC_MASS_DIAG)
    HMC_REQUIRE(s->mass_diag && s->mass_inv_diag, "%s: diagonal mass needs diag and inverse", who);
  if (s->mass_kind == HMC_MASS_FULL)
    HMC_REQUIRE(s->mass_chol && s->mass_inv && s->v, "%s: full mass needs cholesky, inverse and v", who);
  if (s->stream_z || s->stream_eps || s->stream_u)
    HMC_REQUIRE(s->stream_z && s->stream_u && s->stream_len > 0 && (s->stream_eps || !s->randomize_stepsize),
                "%s: incomplete injected streams", who);
  if (s->ring_q) HMC_REQUIRE(s->ring_x && s->ring_slots > 0 && s->thinning > 0, "%s: bad sample ring", who);
  return HMC_OK;
}

inline unsigned ew_grid(int64_t n) {
  const unsigned b = blocks_for(n, 256);
  return b > 152u * 32u ? 152u * 32u : b;
}

template <typename T>
int begin_impl(const hmc_chains* s, double drift, cudaStream_t st) {
  HMC_TRY(check_state<T>(s, "hmc_begin_trajectory"));
  ChainView<T> v = view<T>(s);
  const ColumnShape shape = column_shape(s->chains, s->dims);
  const char* who = "begin_kernel";
  switch (s->mass_kind) {
    case HMC_MASS_UNIT:
      return launch_columns(who, begin_kernel<T, HMC_MASS_UNIT>, shape, s->chains, st, v, drift, is_single(drift), shape);
    case HMC_MASS_DIAG:
      return launch_columns(who, begin_kernel<T, HMC_MASS_DIAG>, shape, s->chains, st, v, drift, is_single(drift), shape);
    default: {
      const int64_t quads = (s->dims + 3) / 4;
      draw_z_kernel<T><<<ew_grid(quads * s->chains), 256, 0, st>>>(v);
      HMC_TRY(check_launch("draw_z_kernel"));
      const int dt = std::is_same<T, double>::value ? HMC_F64 : HMC_F32;
      // p = L z, then v = M^-1 p.
      HMC_TRY(gemm_dispatch(dt, s->dims, s->chains, s->dims, 1.0, s->mass_chol, s->v, nullptr, s->p, 0, st));
      HMC_TRY(gemm_dispatch(dt, s->dims, s->chains, s->dims, 1.0, s->mass_inv, s->p, nullptr, s->v, 0, st));
      return launch_columns(who, begin_kernel<T, HMC_MASS_FULL>, shape, s->chains, st, v, drift, is_single(drift), shape);
    }
  }
}

// Threads (x over chains, y over rows) and grid of the kick: `rows` at least per
// thread (element_shape), KICK_ROWS of them loaded together.
template <typename T, int MASS, int VEC>
int kick_drift_launch(const ChainView<T>& v, int rows, bool do_kick, bool do_drift, double kick, double drift,
                      cudaStream_t st) {
  const int64_t cols = (v.C + VEC - 1) / VEC;
  unsigned bx = 1;
  while (bx < 256 && bx < cols) bx *= 2;
  const dim3 block(bx, 256 / bx);
  int64_t gy = (v.d + rows * block.y - 1) / (rows * block.y);
  const int64_t gx = (cols + bx - 1) / bx;
  while (gy > 1 && gx * gy > 152 * 16) gy = (gy + 1) / 2;
  HMC_REQUIRE(gx <= 0x7FFFFFFF, "hmc_kick_drift: too many chains");
  const dim3 grid((unsigned)gx, (unsigned)(gy < 65535 ? gy : 65535));
  const bool single = is_single(kick) && is_single(drift);
  if (do_kick && do_drift)
    kick_drift_kernel<T, MASS, 1, 1, VEC><<<grid, block, 0, st>>>(v, kick, drift, single);
  else if (do_kick)
    kick_drift_kernel<T, MASS, 1, 0, VEC><<<grid, block, 0, st>>>(v, kick, drift, single);
  else
    kick_drift_kernel<T, MASS, 0, 1, VEC><<<grid, block, 0, st>>>(v, kick, drift, single);
  return check_launch("kick_drift_kernel");
}

template <typename T, int MASS>
int kick_drift_any(const ChainView<T>& v, bool do_kick, bool do_drift, double kick, double drift, cudaStream_t st) {
  // 16-byte accesses need every row of the [d][C] state on a 16-byte boundary
  const bool aligned = ((uintptr_t)v.q | (uintptr_t)v.p | (uintptr_t)v.g | (uintptr_t)v.v) % 16 == 0;
  const ElementShape e = element_shape(v.d, v.C, (int)sizeof(T), aligned, KICK_ROWS);
  return e.vec ? kick_drift_launch<T, MASS, 16 / (int)sizeof(T)>(v, e.rows, do_kick, do_drift, kick, drift, st)
               : kick_drift_launch<T, MASS, 1>(v, e.rows, do_kick, do_drift, kick, drift, st);
}

template <typename T>
int kick_drift_impl(const hmc_chains* s, double kick, double drift, cudaStream_t st) {
  HMC_TRY(check_state<T>(s, "hmc_kick_drift"));
  HMC_REQUIRE(s->g != nullptr, "hmc_kick_drift: missing gradient buffer");
  ChainView<T> v = view<T>(s);
  const bool do_drift = drift != 0.0;
  const bool do_kick = kick != 0.0;
  HMC_REQUIRE(do_kick || do_drift, "hmc_kick_drift: kick and drift are both zero");
  switch (s->mass_kind) {
    case HMC_MASS_UNIT:
      return kick_drift_any<T, HMC_MASS_UNIT>(v, do_kick, do_drift, kick, drift, st);
    case HMC_MASS_DIAG:
      return kick_drift_any<T, HMC_MASS_DIAG>(v, do_kick, do_drift, kick, drift, st);
    default: {
      if (do_kick) {
        HMC_TRY((kick_drift_any<T, HMC_MASS_FULL>(v, true, false, kick, drift, st)));
        if (!do_drift) return HMC_OK;
      }
      const int dt = std::is_same<T, double>::value ? HMC_F64 : HMC_F32;
      HMC_TRY(gemm_dispatch(dt, s->dims, s->chains, s->dims, 1.0, s->mass_inv, s->p, nullptr, s->v, 0, st));
      return kick_drift_any<T, HMC_MASS_FULL>(v, false, true, kick, drift, st);
    }
  }
}

template <typename T>
int end_impl(const hmc_chains* s, cudaStream_t st) {
  HMC_TRY(check_state<T>(s, "hmc_end_trajectory"));
  ChainView<T> v = view<T>(s);
  const ColumnShape shape = column_shape(s->chains, s->dims, 320);
  const char* who = "end_kernel";
  switch (s->mass_kind) {
    case HMC_MASS_UNIT:
      return launch_columns(who, end_kernel<T, HMC_MASS_UNIT>, shape, s->chains, st, v, shape);
    case HMC_MASS_DIAG:
      return launch_columns(who, end_kernel<T, HMC_MASS_DIAG>, shape, s->chains, st, v, shape);
    default: {
      const int dt = std::is_same<T, double>::value ? HMC_F64 : HMC_F32;
      HMC_TRY(gemm_dispatch(dt, s->dims, s->chains, s->dims, 1.0, s->mass_inv, s->p, nullptr, s->v, 0, st));
      return launch_columns(who, end_kernel<T, HMC_MASS_FULL>, shape, s->chains, st, v, shape);
    }
  }
}

template <typename T>
int kinetic_impl(const hmc_chains* s, const void* p, double* out, cudaStream_t st) {
  HMC_REQUIRE(s && p && out, "hmc_kinetic_energy: null argument");
  HMC_REQUIRE(s->dims > 0 && s->chains > 0, "hmc_kinetic_energy: bad sizes");
  ChainView<T> v = view<T>(s);
  const ColumnShape shape = column_shape(s->chains, s->dims);
  const char* who = "kinetic_kernel";
  const T* pt = (const T*)p;
  switch (s->mass_kind) {
    case HMC_MASS_UNIT:
      return launch_columns(who, kinetic_kernel<T, HMC_MASS_UNIT>, shape, s->chains, st, v, pt, (const T*)nullptr, out,
                            shape);
    case HMC_MASS_DIAG:
      HMC_REQUIRE(s->mass_inv_diag, "hmc_kinetic_energy: missing inverse diagonal");
      return launch_columns(who, kinetic_kernel<T, HMC_MASS_DIAG>, shape, s->chains, st, v, pt, (const T*)nullptr, out,
                            shape);
    default: {
      HMC_REQUIRE(s->mass_inv && s->v, "hmc_kinetic_energy: full mass needs inverse and v");
      const int dt = std::is_same<T, double>::value ? HMC_F64 : HMC_F32;
      HMC_TRY(gemm_dispatch(dt, s->dims, s->chains, s->dims, 1.0, s->mass_inv, p, nullptr, s->v, 0, st));
      return launch_columns(who, kinetic_kernel<T, HMC_MASS_FULL>, shape, s->chains, st, v, pt, (const T*)s->v, out,
                            shape);
    }
  }
}

template <typename T>
__global__ void scale_rows_kernel(const T* scale, const T* x, T* out, int64_t d, int64_t C) {
  const int64_t total = d * C;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x)
    out[idx] = scale ? scale[idx / C] * x[idx] : x[idx];
}

template <typename T>
int kinetic_grad_impl(const hmc_chains* s, const void* p, void* out, cudaStream_t st) {
  HMC_REQUIRE(s && p && out, "hmc_kinetic_energy_gradient: null argument");
  HMC_REQUIRE(s->dims > 0 && s->chains > 0, "hmc_kinetic_energy_gradient: bad sizes");
  const int dt = std::is_same<T, double>::value ? HMC_F64 : HMC_F32;
  if (s->mass_kind == HMC_MASS_FULL) {
    HMC_REQUIRE(s->mass_inv, "hmc_kinetic_energy_gradient: missing inverse");
    return gemm_dispatch(dt, s->dims, s->chains, s->dims, 1.0, s->mass_inv, p, nullptr, out, 0, st);
  }
  const T* scale = s->mass_kind == HMC_MASS_DIAG ? (const T*)s->mass_inv_diag : nullptr;
  HMC_REQUIRE(s->mass_kind != HMC_MASS_DIAG || scale, "hmc_kinetic_energy_gradient: missing inverse diagonal");
  scale_rows_kernel<T><<<ew_grid(s->dims * s->chains), 256, 0, st>>>(scale, (const T*)p, (T*)out, s->dims,
                                                                      s->chains);
  return check_launch("scale_rows_kernel");
}

}  // namespace
// ---- replica exchange ----------------------------------------------------
// Decision per pair from the current misfits and inverse temperatures; pairs
// with an index outside [0, C) or a == b never swap.
__global__ void exchange_decide_kernel(int64_t npairs, int64_t C, const int32_t* __restrict__ pairs,
                                       const double* __restrict__ u, const double* __restrict__ beta,
                                       const double* __restrict__ x, int32_t* swapped, int64_t* total) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= npairs) return;
  const int32_t a = pairs[2 * k], b = pairs[2 * k + 1];
  int ok = 0;
  if (a >= 0 && a < C && b >= 0 && b < C && a != b) {
    const double ba = beta ? beta[a] : 1.0, bb = beta ? beta[b] : 1.0;
    ok = exp((ba - bb) * (x[a] - x[b])) > u[k] ? 1 : 0;  // NaN compares false
  }
  swapped[k] = ok;
  if (ok && total) atomicAdd((unsigned long long*)total, 1ull);
}

// Swap the columns of accepted pairs: thread (pair k, dimension i).  The
// exchange follows the last proposal's accept step; when that proposal was
// recorded in the thinned ring, its entry is swapped too, so the recorded
// sample is the post-exchange state, as in the reference (the sample is
// appended after the exchange, Samplers.py:589-678).  Its misfit entry is
// the tempered misfit of the swapped-in model.
template <typename T>
__global__ void exchange_swap_kernel(int64_t npairs, int64_t d, int64_t C, const int32_t* __restrict__ pairs,
                                     const int32_t* __restrict__ swapped, T* q_cur, double* x_cur,
                                     const int64_t* __restrict__ control, T* ring_q, double* ring_x,
                                     int64_t ring_slots, int64_t thin, const double* __restrict__ beta) {
  const int64_t n_last = control ? control[0] - 1 : -1;
  const bool rec = ring_q != nullptr && n_last >= 0 && n_last % thin == 0;
  const int64_t slot = rec ? (n_last / thin) % ring_slots : 0;
  const int64_t total = npairs * d;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = e / d, i = e - k * d;
    if (!swapped[k]) continue;
    const int64_t a = pairs[2 * k], b = pairs[2 * k + 1];
    const T t = q_cur[i * C + a];
    q_cur[i * C + a] = q_cur[i * C + b];
    q_cur[i * C + b] = t;
    if (rec) {
      T* r = ring_q + (slot * d + i) * C;
      r[a] = q_cur[i * C + a];
      r[b] = q_cur[i * C + b];
    }
    if (i == 0) {
      const double tx = x_cur[a];
      x_cur[a] = x_cur[b];
      x_cur[b] = tx;
      if (rec && ring_x) {
        ring_x[slot * C + a] = (beta ? beta[a] : 1.0) * x_cur[a];
        ring_x[slot * C + b] = (beta ? beta[b] : 1.0) * x_cur[b];
      }
    }
  }
}

template <typename T>
int exchange_impl(const hmc_chains* s, int64_t npairs, const int32_t* pairs, const double* u, int32_t* swapped,
                  int64_t* total, cudaStream_t st) {
  HMC_REQUIRE(s->dims > 0 && s->chains > 0 && s->q_cur && s->x_cur, "hmc_exchange: missing state");
  HMC_REQUIRE(npairs >= 0 && 2 * npairs <= s->chains, "hmc_exchange: %lld pairs for %lld chains",
              (long long)npairs, (long long)s->chains);
  if (npairs == 0) return HMC_OK;
  HMC_REQUIRE(pairs && u && swapped, "hmc_exchange: null pairs, uniforms or decisions");
  exchange_decide_kernel<<<blocks_for(npairs, 256), 256, 0, st>>>(npairs, s->chains, pairs, u, s->beta, s->x_cur,
                                                                   swapped, total);
  HMC_TRY(check_launch("exchange_decide_kernel"));
  if (s->ring_q) HMC_REQUIRE(s->ring_slots > 0 && s->thinning > 0, "hmc_exchange: bad sample ring");
  exchange_swap_kernel<T><<<ew_grid(npairs * s->dims), 256, 0, st>>>(
      npairs, s->dims, s->chains, pairs, swapped, (T*)s->q_cur, s->x_cur, s->proposal, (T*)s->ring_q, s->ring_x,
      s->ring_slots, s->thinning, s->beta);
  return check_launch("exchange_swap_kernel");
}

}  // namespace hmc

using namespace hmc;

extern "C" {

int hmc_exchange(const hmc_chains* s, int64_t npairs, const int32_t* pairs, const double* u, int32_t* swapped,
                 int64_t* accepted_total, void* stream) {
  if (!s) return fail(HMC_ERR_INVALID_ARG, "hmc_exchange: null state");
  return HMC_DISPATCH(s->dtype, T, [&] {
    return exchange_impl<T>(s, npairs, pairs, u, swapped, accepted_total, as_stream(stream));
  });
}

int hmc_begin_trajectory(const hmc_chains* s, double drift, void* stream) {
  if (!s) return fail(HMC_ERR_INVALID_ARG, "hmc_begin_trajectory: null state");
  return HMC_DISPATCH(s->dtype, T, [&] { return begin_impl<T>(s, drift, as_stream(stream)); });
}

int hmc_kick_drift(const hmc_chains* s, double kick, double drift, void* stream) {
  if (!s) return fail(HMC_ERR_INVALID_ARG, "hmc_kick_drift: null state");
  return HMC_DISPATCH(s->dtype, T, [&] { return kick_drift_impl<T>(s, kick, drift, as_stream(stream)); });
}

int hmc_end_trajectory(const hmc_chains* s, void* stream) {
  if (!s) return fail(HMC_ERR_INVALID_ARG, "hmc_end_trajectory: null state");
  return HMC_DISPATCH(s->dtype, T, [&] { return end_impl<T>(s, as_stream(stream)); });
}

int hmc_kinetic_energy(const hmc_chains* s, const void* p, double* out, void* stream) {
  if (!s) return fail(HMC_ERR_INVALID_ARG, "hmc_kinetic_energy: null state");
  return HMC_DISPATCH(s->dtype, T, [&] { return kinetic_impl<T>(s, p, out, as_stream(stream)); });
}

int hmc_kinetic_energy_gradient(const hmc_chains* s, const void* p, void* out, void* stream) {
  if (!s) return fail(HMC_ERR_INVALID_ARG, "hmc_kinetic_energy_gradient: null state");
  return HMC_DISPATCH(s->dtype, T, [&] { return kinetic_grad_impl<T>(s, p, out, as_stream(stream)); });
}

}  // extern "C"
