// Persistent proposals of many chains on a small dense target: a warp advances
// 1, 2 or 4 chains, a lane owns the rows lane, lane + 32, ... of each.
#include "persistent.cuh"

namespace hmc {
namespace pers {

// Sums over the warp of N values per lane (N a power of two): each halving
// sends half of the values away, so N values take N - 1 + 5 - log2 N adds
// instead of 5 N.  Lane l then holds the total of value l >> (5 - log2 N); the
// tree of every sum is the one of warp_sum.
template <int N>
__device__ __forceinline__ double warp_sums(double v[N], int lane) {
  int off = 16;
#pragma unroll
  for (int n = N / 2; n >= 1; n /= 2) {
    const bool up = lane & off;
#pragma unroll
    for (int j = 0; j < n; ++j) {
      const double give = up ? v[j] : v[j + n];
      v[j] = (up ? v[j + n] : v[j]) + __shfl_xor_sync(0xffffffffu, give, off);
    }
    off /= 2;
  }
  for (; off > 0; off /= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
  return v[0];
}

template <typename T, int CT>
struct alignas(sizeof(T) * CT <= 16 ? sizeof(T) * CT : 16) Chains {
  T v[CT];
};

// Slot of column j in a warp's published vector: the columns of the unrolled
// main part first, then up to three of the remainder (D: columns held in
// registers, 0: plain order).
template <int D>
__device__ __forceinline__ int column_slot(int j, int d) {
  const int main = d & ~3;
  return D == 0 || j < main ? j : D + j - main;
}

// The lane's rows of GtG q for CT chains, columns summed by j modulo 4 and
// combined as (s0 + s1) + (s2 + s3), remainder columns in s0.  D > 0: the
// lane's rows sit in registers (a), padded with zeros to D + 3 columns.
template <typename T, int E, int CT, int D>
__device__ __forceinline__ void lanes_matvec(const T (*a)[D > 0 ? D + 3 : 1], const T* A, int ld, int d,
                                             const Chains<T, CT>* qv, const int row[E], T out[E][CT]) {
  if constexpr (D > 0) {
    T half[2][E][CT];
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // residues 0 and 1, then 2 and 3
      T s[2][E][CT];
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int k = 0; k < E; ++k)
#pragma unroll
          for (int c = 0; c < CT; ++c) s[r][k][c] = (T)0;
#pragma unroll
      for (int j = 2 * h; j < D; j += 4)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const Chains<T, CT> x = qv[j + r];
#pragma unroll
          for (int k = 0; k < E; ++k)
#pragma unroll
            for (int c = 0; c < CT; ++c) s[r][k][c] = fma(a[k][j + r], x.v[c], s[r][k][c]);
        }
      if (h == 0) {
#pragma unroll
        for (int j = D; j < D + 3; ++j) {
          const Chains<T, CT> x = qv[j];
#pragma unroll
          for (int k = 0; k < E; ++k)
#pragma unroll
            for (int c = 0; c < CT; ++c) s[0][k][c] = fma(a[k][j], x.v[c], s[0][k][c]);
        }
      }
#pragma unroll
      for (int k = 0; k < E; ++k)
#pragma unroll
        for (int c = 0; c < CT; ++c) half[h][k][c] = s[0][k][c] + s[1][k][c];
    }
#pragma unroll
    for (int k = 0; k < E; ++k)
#pragma unroll
      for (int c = 0; c < CT; ++c) out[k][c] = half[0][k][c] + half[1][k][c];
  } else {
    T s[4][E][CT];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int k = 0; k < E; ++k)
#pragma unroll
        for (int c = 0; c < CT; ++c) s[r][k][c] = (T)0;
    int j = 0;
    for (; j + 4 <= d; j += 4) {
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const Chains<T, CT> x = qv[j + r];
#pragma unroll
        for (int k = 0; k < E; ++k) {
          const T av = A[row[k] * ld + j + r];
#pragma unroll
          for (int c = 0; c < CT; ++c) s[r][k][c] = fma(av, x.v[c], s[r][k][c]);
        }
      }
    }
    for (; j < d; ++j) {
      const Chains<T, CT> x = qv[j];
#pragma unroll
      for (int k = 0; k < E; ++k) {
        const T av = A[row[k] * ld + j];
#pragma unroll
        for (int c = 0; c < CT; ++c) s[0][k][c] = fma(av, x.v[c], s[0][k][c]);
      }
    }
#pragma unroll
    for (int k = 0; k < E; ++k)
#pragma unroll
      for (int c = 0; c < CT; ++c) out[k][c] = (s[0][k][c] + s[1][k][c]) + (s[2][k][c] + s[3][k][c]);
  }
}

// Shared memory of one warp: the published vector (CT values per column), then
// the kick and drift coefficients of every step.
template <typename T, int CT, int D>
__host__ __device__ constexpr int lanes_slots(int d) {
  return D > 0 ? D + 3 : d;
}

// Fused multiply-adds are written out: whether the compiler contracts a product
// with a sum across a branch differs between the instantiations.
//
// The matrix is read once per CT chains: from registers for FP32 up to 64
// columns (one 16-byte broadcast of four chains' column then feeds 8 fused
// multiply-adds per lane, where the warp-per-chain kernel read two words of
// shared memory for each), else from shared memory.  Each (quad, chain) of the
// momenta is drawn by one lane, and a warp sums the energies of its chains
// together.  Per proposal of 10 steps, FP32, 4096 chains: d = 50 18.3 us against
// 43.4 with one chain per warp and the matrix in shared memory, d = 100 52
// against 138; 1024 chains of d = 50 7.7 against 21.9 (one chain per warp).
template <typename T, int E, int CT, int D>
__global__ void __launch_bounds__(256) persistent_lanes_kernel(State<T> s, Target<T> tg, const __grid_constant__ hmc_schedule sch,
                                                               int64_t nprop, bool single, int dry) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using V = Chains<T, CT>;
  const int d = tg.d, ld = tg.ld;
  const bool diag = s.mass == HMC_MASS_DIAG;
  const int prior = tg.prior;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int slots = lanes_slots<T, CT, D>(d);
  V* qv = (V*)smem_raw + warp * (slots + 2 * sch.steps);
  V* coef = qv + slots;  // kick of step l at 2 l, drift at 2 l + 1
  T* A = (T*)((V*)smem_raw + warps * (slots + 2 * sch.steps));
  if (D == 0) {
    load_matrix(A, tg.GtG, d, ld);
    __syncthreads();
  }
  const int64_t c0 = (blockIdx.x * (int64_t)warps + warp) * CT;
  if (c0 >= s.C) return;  // whole warps only; no block barrier follows
  const int nc = s.C - c0 < CT ? (int)(s.C - c0) : CT;  // live chains of the warp
  const int64_t n0 = s.control[0];

  int row[E];
  bool live[E];
  T a[D > 0 ? E : 1][D > 0 ? D + 3 : 1];
  T minv[E], msq[E], gtd[E], pm[E], pw[E], qc[E][CT];
#pragma unroll
  for (int k = 0; k < E; ++k) {
    const int i = lane + 32 * k;
    live[k] = i < d;
    row[k] = live[k] ? i : d - 1;
    minv[k] = diag ? s.minv[row[k]] : (T)1;
    msq[k] = diag ? mass_root(s.mdiag[row[k]]) : (T)1;
    gtd[k] = tg.Gtd0[row[k]];
    pm[k] = prior != PRIOR_NONE ? tg.pmean[row[k]] : (T)0;
    pw[k] = prior != PRIOR_NONE ? tg.pw[row[k]] : (T)0;
#pragma unroll
    for (int c = 0; c < CT; ++c) qc[k][c] = c < nc ? s.q_cur[(int64_t)row[k] * s.C + c0 + c] : (T)0;
    if constexpr (D > 0) {
      const int main = d & ~3;
#pragma unroll
      for (int j = 0; j < D; ++j) a[k][j] = j < main ? tg.GtG[row[k] * d + j] : (T)0;
#pragma unroll
      for (int j = 0; j < 3; ++j) a[k][D + j] = main + j < d ? tg.GtG[row[k] * d + main + j] : (T)0;
    }
  }
  for (int j = lane; j < slots; j += 32)
#pragma unroll
    for (int c = 0; c < CT; ++c) qv[j].v[c] = (T)0;  // the padding stays zero
  __syncwarp();
  // lane c keeps the scalars of chain c
  const bool own = lane < nc;
  double xc = own ? s.x_cur[c0 + lane] : 0.0;
  const T eps0 = own ? s.eps[c0 + lane] : (T)0;
  int64_t n_acc = 0;

  auto publish = [&](const T q[E][CT]) {
#pragma unroll
    for (int k = 0; k < E; ++k)
      if (live[k]) {
        V x;
#pragma unroll
        for (int c = 0; c < CT; ++c) x.v[c] = q[k][c];
        qv[column_slot<D>(row[k], d)] = x;
      }
    __syncwarp();
  };

  for (int64_t t = 0; t < nprop; ++t) {
    const int64_t n = n0 + t;
    T e_own = eps0;
    double u = 0.0;
    if (own) {
      double ue = 0.0, ua = 0.0;
      if (!s.seps || !s.su) philox_scalars(s.seed, (uint32_t)(c0 + lane), (uint64_t)n, &ue, &ua);
      if (s.randomize) e_own *= s.seps ? s.seps[(n % s.slen) * s.C + c0 + lane] : (T)(0.5 + ue);
      u = s.su ? s.su[(n % s.slen) * s.C + c0 + lane] : ua;
    }
    T e[CT];
#pragma unroll
    for (int c = 0; c < CT; ++c) e[c] = __shfl_sync(0xffffffffu, e_own, c);
    for (int l = lane; l < sch.steps; l += 32)
#pragma unroll
      for (int c = 0; c < CT; ++c) {
        coef[2 * l].v[c] = scaled_step(sch.kick[l], single, e[c]);
        coef[2 * l + 1].v[c] = scaled_step(sch.drift[l], single, e[c]);
      }
    // momenta: the four rows of a (quad, chain) pair per lane, each pair once
    if (!s.sz) {
      for (int k = lane; k < ((d + 3) / 4) * CT; k += 32) {
        const int qd = k / CT, c = k % CT;
        T z[4];
        philox_normal4<T>(s.seed, (uint32_t)qd, (uint32_t)(c0 + c), (uint64_t)n, PURPOSE_MOMENTUM, z);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (4 * qd + j < d) qv[column_slot<D>(4 * qd + j, d)].v[c] = z[j];
      }
    } else {
      for (int i = lane; i < d; i += 32)
#pragma unroll
        for (int c = 0; c < CT; ++c)
          qv[column_slot<D>(i, d)].v[c] = c < nc ? s.sz[((n % s.slen) * d + i) * s.C + c0 + c] : (T)0;
    }
    __syncwarp();
    T p[E][CT], q[E][CT], g[E][CT];
    double sums[4 * CT];  // misfit, K1, K0 of every chain (and padding)
#pragma unroll
    for (int c = 0; c < 4 * CT; ++c) sums[c] = 0.0;
#pragma unroll
    for (int k = 0; k < E; ++k) {
      const V z = qv[column_slot<D>(row[k], d)];
#pragma unroll
      for (int c = 0; c < CT; ++c) {
        p[k][c] = diag ? msq[k] * z.v[c] : z.v[c];
        const T mp = diag ? minv[k] * p[k][c] : p[k][c];
        if (live[k]) sums[2 * CT + c] = fma(f64_of(p[k][c]), f64_of(mp), sums[2 * CT + c]);
        q[k][c] = fma(scaled_step(sch.first_drift, single, e[c]), mp, qc[k][c]);
      }
    }
    __syncwarp();

    for (int st = 0; st < sch.steps; ++st) {
      if (sch.gradient[st]) {
        publish(q);
        lanes_matvec<T, E, CT, D>(a, A, ld, d, qv, row, g);
        __syncwarp();
        const V ck = coef[2 * st];
#pragma unroll
        for (int k = 0; k < E; ++k)
#pragma unroll
          for (int c = 0; c < CT; ++c) {
            T gk = g[k][c] - gtd[k];
            if (prior == PRIOR_NORMAL) gk = fma(-pw[k], pm[k] - q[k][c], gk);
            if (prior == PRIOR_LAPLACE) gk = gk + sign_of(q[k][c] - pm[k]) * pw[k];
            p[k][c] = fma(-ck.v[c], gk, p[k][c]);
          }
      }
      if (sch.drift[st] != 0.0) {
        const V cd = coef[2 * st + 1];
#pragma unroll
        for (int k = 0; k < E; ++k)
#pragma unroll
          for (int c = 0; c < CT; ++c) {
            const T mp = diag ? minv[k] * p[k][c] : p[k][c];
            q[k][c] = fma(cd.v[c], mp, q[k][c]);
          }
      }
    }

    // misfit at the end point, K1 and the accept test (FP64)
    publish(q);
    lanes_matvec<T, E, CT, D>(a, A, ld, d, qv, row, g);
    __syncwarp();
#pragma unroll
    for (int k = 0; k < E; ++k) {
      if (!live[k]) continue;
#pragma unroll
      for (int c = 0; c < CT; ++c) {
        const T w = fma((T)-2, gtd[k], g[k][c]);
        double x = f64_of(q[k][c]) * f64_of(w);
        if (prior == PRIOR_NORMAL) {
          const T r = pm[k] - q[k][c];
          x = fma(f64_of(r), f64_of(pw[k] * r), x);
        }
        if (prior == PRIOR_LAPLACE) x = fma(2.0, f64_of((T)(fabs(q[k][c] - pm[k]) * pw[k])), x);
        sums[c] += x;
        const T mp = diag ? minv[k] * p[k][c] : p[k][c];
        sums[CT + c] = fma(f64_of(p[k][c]), f64_of(mp), sums[CT + c]);
      }
    }
    const double total = warp_sums<4 * CT>(sums, lane);
    constexpr int HOLD = 8 / CT;  // lanes per value of the 4 CT
    const double x1 = 0.5 * (__shfl_sync(0xffffffffu, total, (lane % CT) * HOLD) + tg.dtd);
    const double k1 = 0.5 * __shfl_sync(0xffffffffu, total, (CT + lane % CT) * HOLD);
    const double k0 = 0.5 * __shfl_sync(0xffffffffu, total, (2 * CT + lane % CT) * HOLD);
    bool accept = false;
    if (own) accept = exp((xc + k0) - (x1 + k1)) > u;  // strict; NaN compares false
    if (accept) {
      xc = x1;
      ++n_acc;
    }
    const unsigned taken = __ballot_sync(0xffffffffu, accept);
#pragma unroll
    for (int c = 0; c < CT; ++c)
      if (taken >> c & 1u) {
#pragma unroll
        for (int k = 0; k < E; ++k) qc[k][c] = q[k][c];
      }
    if (!dry && s.ring_q && (n % s.thin) == 0) {
      const int64_t slot = (n / s.thin) % s.ring_slots;
#pragma unroll
      for (int k = 0; k < E; ++k)
        if (live[k]) {
          T* o = s.ring_q + (slot * d + row[k]) * s.C + c0;
#pragma unroll
          for (int c = 0; c < CT; ++c)
            if (c < nc) o[c] = qc[k][c];
        }
      if (own) s.ring_x[slot * s.C + c0 + lane] = xc;
    }
  }
  if (dry) return;
#pragma unroll
  for (int k = 0; k < E; ++k)
    if (live[k])
#pragma unroll
      for (int c = 0; c < CT; ++c)
        if (c < nc) s.q_cur[(int64_t)row[k] * s.C + c0 + c] = qc[k][c];
  if (own) {
    s.x_cur[c0 + lane] = xc;
    s.accepted[c0 + lane] += n_acc;
  }
}


template <typename T, int E, int CT, int D>
int launch_one(const State<T>& st, const Target<T>& tg, const hmc_schedule& sch, int64_t nprop, int dry, bool single,
               int warps, cudaStream_t stream) {
  const size_t smem = lanes_smem<T>(tg.d, sch.steps, CT, warps);
  auto kern = persistent_lanes_kernel<T, E, CT, D>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(persistent_lanes_kernel)");
  }
  const int64_t per = (int64_t)CT * warps;
  kern<<<(unsigned)((st.C + per - 1) / per), 32 * warps, smem, stream>>>(st, tg, sch, nprop, single, dry);
  return check_launch("persistent_lanes_kernel");
}

// Rows in registers: FP32 up to 64 columns (two rows of 64 + 3 are 134
// registers); the columns unrolled are the next of 16, 32, 48, 64.
inline int register_columns(int d, size_t esize) {
  const int main = d & ~3;
  if (esize != 4 || d > 64) return 0;
  return d <= 32 ? (main <= 16 ? 16 : 32) : (main <= 48 ? 48 : 64);
}

template <typename T>
size_t lanes_smem(int d, int steps, int chains_per_warp, int warps) {
  const int D = register_columns(d, sizeof(T));
  const size_t vec = (size_t)(D > 0 ? D + 3 : d) + 2 * (size_t)steps;
  return (vec * warps * chains_per_warp + (D > 0 ? 0 : (size_t)d * (d | 1))) * sizeof(T);
}

template <typename T, int CT>
int launch_width(const State<T>& st, const Target<T>& tg, const hmc_schedule& sch, int64_t nprop, int dry, bool single,
                 int warps, cudaStream_t stream) {
  if constexpr (sizeof(T) == 4) {
    switch (register_columns(tg.d, sizeof(T))) {
      case 16: return launch_one<T, 1, CT, 16>(st, tg, sch, nprop, dry, single, warps, stream);
      case 32: return launch_one<T, 1, CT, 32>(st, tg, sch, nprop, dry, single, warps, stream);
      case 48: return launch_one<T, 2, CT, 48>(st, tg, sch, nprop, dry, single, warps, stream);
      case 64: return launch_one<T, 2, CT, 64>(st, tg, sch, nprop, dry, single, warps, stream);
      default: break;
    }
  } else {
    if (tg.d <= 32) return launch_one<T, 1, CT, 0>(st, tg, sch, nprop, dry, single, warps, stream);
    if (tg.d <= 64) return launch_one<T, 2, CT, 0>(st, tg, sch, nprop, dry, single, warps, stream);
  }
  if (tg.d <= 96) return launch_one<T, 3, CT, 0>(st, tg, sch, nprop, dry, single, warps, stream);
  return launch_one<T, 4, CT, 0>(st, tg, sch, nprop, dry, single, warps, stream);
}

template <typename T>
int launch_lanes(const State<T>& st, const Target<T>& tg, const hmc_schedule& sch, int64_t nprop, int dry, bool single,
                 int chains_per_warp, int warps, cudaStream_t stream) {
  switch (chains_per_warp) {
    case 1: return launch_width<T, 1>(st, tg, sch, nprop, dry, single, warps, stream);
    case 2: return launch_width<T, 2>(st, tg, sch, nprop, dry, single, warps, stream);
    default:
      if constexpr (sizeof(T) == 4) return launch_width<T, 4>(st, tg, sch, nprop, dry, single, warps, stream);
      return fail(HMC_ERR_INVALID_ARG, "persistent lanes: 4 chains per warp are FP32 only");
  }
}

template int launch_lanes<float>(const State<float>&, const Target<float>&, const hmc_schedule&, int64_t, int, bool, int,
                                 int, cudaStream_t);
template int launch_lanes<double>(const State<double>&, const Target<double>&, const hmc_schedule&, int64_t, int, bool,
                                  int, int, cudaStream_t);
template size_t lanes_smem<float>(int, int, int, int);
template size_t lanes_smem<double>(int, int, int, int);

}  // namespace pers
}  // namespace hmc
