// Persistent proposals of many chains on a small dense target: a group of warps
// advances 1, 2 or 4 chains, a thread per row.
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

// Slot of column j in a group's published vector: the columns of the unrolled
// main part first, then up to three of the remainder (D: columns held in
// registers, 0: plain order).
template <int D>
__device__ __forceinline__ int column_slot(int j, int d) {
  const int main = d & ~3;
  return D == 0 || j < main ? j : D + j - main;
}

// The thread's E rows of GtG q for CT chains, columns summed by j modulo 4 and
// combined as (s0 + s1) + (s2 + s3), remainder columns in s0.  D > 0 (one row):
// the row sits in registers (a), padded with zeros to D + 3 columns.
template <typename T, int E, int CT, int D>
__device__ __forceinline__ void group_matvec(const T a[D > 0 ? D + 3 : 1], const T* const A[E], int d,
                                             const Chains<T, CT>* qv, T out[E][CT]) {
  T s[4][E][CT];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int k = 0; k < E; ++k)
#pragma unroll
      for (int c = 0; c < CT; ++c) s[r][k][c] = (T)0;
  if constexpr (D > 0) {
#pragma unroll
    for (int j = 0; j < D + 3; ++j) {
      const Chains<T, CT> x = qv[j];
      const int r = j < D ? j % 4 : 0;
#pragma unroll
      for (int c = 0; c < CT; ++c) s[r][0][c] = fma(a[j], x.v[c], s[r][0][c]);
    }
  } else {
    int j = 0;
    for (; j + 4 <= d; j += 4) {
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const Chains<T, CT> x = qv[j + r];
#pragma unroll
        for (int k = 0; k < E; ++k) {
          const T av = A[k][j + r];
#pragma unroll
          for (int c = 0; c < CT; ++c) s[r][k][c] = fma(av, x.v[c], s[r][k][c]);
        }
      }
    }
    for (; j < d; ++j) {
      const Chains<T, CT> x = qv[j];
#pragma unroll
      for (int k = 0; k < E; ++k) {
        const T av = A[k][j];
#pragma unroll
        for (int c = 0; c < CT; ++c) s[0][k][c] = fma(av, x.v[c], s[0][k][c]);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < E; ++k)
#pragma unroll
    for (int c = 0; c < CT; ++c) out[k][c] = (s[0][k][c] + s[1][k][c]) + (s[2][k][c] + s[3][k][c]);
}

// Shared memory of one group of NW warps: two published vectors (CT values per
// column), the coefficients of every step, the warps' sums and the scalars.
template <typename T, int CT>
struct GroupShared {
  double part[4][2 * CT];
  Chains<T, CT> step;  // step sizes
  unsigned taken;      // bit c: chain c accepted
};

// Fused multiply-adds are written out: whether the compiler contracts a product
// with a sum across a branch differs between the instantiations.
//
// GtG is read once per CT chains: an FP32 row sits in its thread's registers
// (or, in large batches beyond 64 columns, four rows come from shared memory),
// where the warp-per-chain kernel read two words of shared memory for each
// multiply-add.  Each (quad, chain) of the momenta is drawn by one lane, a
// group sums the energies of its chains together, and one published vector per
// product needs one barrier.  Bound by FP64 (K, misfit and their sums) and
// shared-memory returns.  Per proposal of 10 steps, FP32, d = 50: 4096 chains
// 16.1 us against 43.4, 1024 chains 7.6 against 21.9, one chain 5.9 against 17.8;
// d = 100, 4096 chains 47 against 138.
template <typename T, int NW, int E, int CT, int D>
__global__ void __launch_bounds__(256) persistent_lanes_kernel(State<T> s, Target<T> tg,
                                                               const __grid_constant__ hmc_schedule sch, int64_t nprop,
                                                               bool single, int dry) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using V = Chains<T, CT>;
  using G = GroupShared<T, CT>;
  const int d = tg.d, ld = tg.ld;
  const bool diag = s.mass == HMC_MASS_DIAG;
  const int prior = tg.prior;
  constexpr int NT = 32 * NW;
  const int lane = threadIdx.x & 31, group = threadIdx.x / NT, groups = blockDim.x / NT;
  const int i = threadIdx.x % NT, warp = i >> 5;  // the thread's rows are i + NT k
  const int slots = D > 0 ? D + 3 : d;
  const int vecs = 2 * slots + 2 * sch.steps;
  V* base = (V*)smem_raw + (size_t)group * vecs;
  V* coef = base + 2 * slots;  // kick of step l at 2 l, drift at 2 l + 1
  G& sh = ((G*)((V*)smem_raw + (((size_t)groups * vecs + 15) & ~(size_t)15)))[group];
  T* A = (T*)((G*)((V*)smem_raw + (((size_t)groups * vecs + 15) & ~(size_t)15)) + groups);
  if (D == 0) {
    load_matrix(A, tg.GtG, d, ld);
    __syncthreads();
  }
  const int64_t c0 = (blockIdx.x * (int64_t)groups + group) * CT;
  if (c0 >= s.C) return;  // whole groups only; only the group's barrier follows
  const int nc = s.C - c0 < CT ? (int)(s.C - c0) : CT;  // live chains of the group
  const int64_t n0 = s.control[0];
  auto sync = [&] {
    if (NW == 1)
      __syncwarp();
    else
      asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(NT) : "memory");
  };

  bool live[E];
  int row[E];
  const T* rows[E];
  T a[D > 0 ? D + 3 : 1], qc[E][CT], minv[E], msq[E], gtd[E], pm[E], pw[E];
#pragma unroll
  for (int k = 0; k < E; ++k) {
    live[k] = i + NT * k < d;
    row[k] = live[k] ? i + NT * k : d - 1;
    rows[k] = A + row[k] * ld;
    minv[k] = diag ? s.minv[row[k]] : (T)1;
    msq[k] = diag ? mass_root(s.mdiag[row[k]]) : (T)1;
    gtd[k] = tg.Gtd0[row[k]];
    pm[k] = prior != PRIOR_NONE ? tg.pmean[row[k]] : (T)0;
    pw[k] = prior != PRIOR_NONE ? tg.pw[row[k]] : (T)0;
#pragma unroll
    for (int c = 0; c < CT; ++c) qc[k][c] = c < nc ? s.q_cur[(int64_t)row[k] * s.C + c0 + c] : (T)0;
  }
  if constexpr (D > 0) {
    const int main = d & ~3;
#pragma unroll
    for (int j = 0; j < D; ++j) a[j] = j < main ? tg.GtG[row[0] * d + j] : (T)0;
#pragma unroll
    for (int j = 0; j < 3; ++j) a[D + j] = main + j < d ? tg.GtG[row[0] * d + main + j] : (T)0;
  }
  for (int j = i; j < 2 * slots; j += NT)
#pragma unroll
    for (int c = 0; c < CT; ++c) base[j].v[c] = (T)0;  // the padding stays zero
  // lane c of the first warp keeps the scalars of chain c
  const bool own = warp == 0 && lane < nc;
  double xc = own ? s.x_cur[c0 + lane] : 0.0;
  const T eps0 = own ? s.eps[c0 + lane] : (T)0;
  int64_t n_acc = 0;
  int buf = 0;
  sync();

  // q published, then GtG q: the two buffers alternate, so one barrier per
  // product separates its reads from the next but one's writes.
  auto matvec = [&](const T q[E][CT], T g[E][CT]) {
    V* qv = base + buf * slots;
    buf ^= 1;
#pragma unroll
    for (int k = 0; k < E; ++k)
      if (live[k]) {
        V x;
#pragma unroll
        for (int c = 0; c < CT; ++c) x.v[c] = q[k][c];
        qv[column_slot<D>(row[k], d)] = x;
      }
    sync();
    group_matvec<T, E, CT, D>(a, rows, d, qv, g);
  };

  for (int64_t t = 0; t < nprop; ++t) {
    const int64_t n = n0 + t;
    double u = 0.0;
    if (own) {
      double ue = 0.0, ua = 0.0;
      if (!s.seps || !s.su) philox_scalars(s.seed, (uint32_t)(c0 + lane), (uint64_t)n, &ue, &ua);
      T e = eps0;
      if (s.randomize) e *= s.seps ? s.seps[(n % s.slen) * s.C + c0 + lane] : (T)(0.5 + ue);
      u = s.su ? s.su[(n % s.slen) * s.C + c0 + lane] : ua;
      sh.step.v[lane] = e;
    }
    // momenta: the four rows of a (quad, chain) pair per thread, each pair
    // once, passed through the buffer that the last product does not read
    V* zv = base + buf * slots;
    buf ^= 1;
    if (!s.sz) {
      for (int k = i; k < ((d + 3) / 4) * CT; k += NT) {
        const int qd = k / CT, c = k % CT;
        T z[4];
        philox_normal4<T>(s.seed, (uint32_t)qd, (uint32_t)(c0 + c), (uint64_t)n, PURPOSE_MOMENTUM, z);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (4 * qd + j < d) zv[column_slot<D>(4 * qd + j, d)].v[c] = z[j];
      }
    } else {
#pragma unroll
      for (int k = 0; k < E; ++k)
        if (live[k])
#pragma unroll
          for (int c = 0; c < CT; ++c)
            zv[column_slot<D>(row[k], d)].v[c] = c < nc ? s.sz[((n % s.slen) * d + row[k]) * s.C + c0 + c] : (T)0;
    }
    sync();
    const V e = sh.step;
    for (int l = i; l < sch.steps; l += NT)
#pragma unroll
      for (int c = 0; c < CT; ++c) {
        coef[2 * l].v[c] = scaled_step(sch.kick[l], single, e.v[c]);
        coef[2 * l + 1].v[c] = scaled_step(sch.drift[l], single, e.v[c]);
      }
    T p[E][CT], q[E][CT], g[E][CT];
    double sums[2 * CT];  // misfit and K1 - K0 of every chain
#pragma unroll
    for (int c = 0; c < 2 * CT; ++c) sums[c] = 0.0;
#pragma unroll
    for (int k = 0; k < E; ++k) {
      const V z = zv[column_slot<D>(row[k], d)];
#pragma unroll
      for (int c = 0; c < CT; ++c) {
        p[k][c] = diag ? msq[k] * z.v[c] : z.v[c];
        const T mp = diag ? minv[k] * p[k][c] : p[k][c];
        if (live[k]) sums[CT + c] = fma(-f64_of(p[k][c]), f64_of(mp), sums[CT + c]);
        q[k][c] = fma(scaled_step(sch.first_drift, single, e.v[c]), mp, qc[k][c]);
      }
    }
    if (sch.steps > 0 && !sch.gradient[0]) sync();  // the coefficients are read before a product's barrier

    for (int st = 0; st < sch.steps; ++st) {
      if (sch.gradient[st]) {
        matvec(q, g);
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
          for (int c = 0; c < CT; ++c) q[k][c] = fma(cd.v[c], diag ? minv[k] * p[k][c] : p[k][c], q[k][c]);
      }
    }

    // misfit at the end point, K1 and the accept test (FP64)
    matvec(q, g);
#pragma unroll
    for (int k = 0; k < E; ++k) {
      if (!live[k]) continue;
#pragma unroll
      for (int c = 0; c < CT; ++c) {
        const T w = fma((T)-2, gtd[k], g[k][c]);
        sums[c] = fma(f64_of(q[k][c]), f64_of(w), sums[c]);
        if (prior == PRIOR_NORMAL) {
          const T r = pm[k] - q[k][c];
          sums[c] = fma(f64_of(r), f64_of(pw[k] * r), sums[c]);
        }
        if (prior == PRIOR_LAPLACE) sums[c] = fma(2.0, f64_of((T)(fabs(q[k][c] - pm[k]) * pw[k])), sums[c]);
        sums[CT + c] = fma(f64_of(p[k][c]), f64_of(diag ? minv[k] * p[k][c] : p[k][c]), sums[CT + c]);
      }
    }
    constexpr int HOLD = 16 / CT;  // lanes per value of the 2 CT
    double total = warp_sums<2 * CT>(sums, lane);
    if (NW > 1) {
      if (lane % HOLD == 0) sh.part[warp][lane / HOLD] = total;
      sync();
      if (warp == 0) {
        total = sh.part[0][lane / HOLD];
#pragma unroll
        for (int k = 1; k < NW; ++k) total += sh.part[k][lane / HOLD];
      }
    }
    if (warp == 0) {
      const double x1 = 0.5 * (__shfl_sync(0xffffffffu, total, (lane % CT) * HOLD) + tg.dtd);
      const double dk = 0.5 * __shfl_sync(0xffffffffu, total, (CT + lane % CT) * HOLD);
      const bool accept = own && accept_test(xc - (x1 + dk), u);
      if (accept) {
        xc = x1;
        ++n_acc;
      }
      const unsigned taken = __ballot_sync(0xffffffffu, accept);
      if (lane == 0) sh.taken = taken;
    }
    sync();
    const unsigned taken = sh.taken;
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

// How a target's rows are laid out: warps per group, rows per thread, and the
// columns kept in registers (0: GtG in shared memory).  One FP32 row per thread
// in registers is the fastest for a chain, but every fused multiply-add then
// reads four bytes of the broadcast column, twice what shared memory returns
// per cycle at full rate.  At d <= 64 the rest of a proposal hides it; beyond,
// the batches that fill the chip run one warp per group with up to four rows
// per thread (two bytes each).  FP32, 4096 chains of d = 100: 47 us per proposal
// against 71; 1024 chains 26 against 19; one chain 26 against 8.
struct LanesLayout {
  int warps, rows, cols;
};
inline LanesLayout lanes_layout(int d, int64_t chains, size_t esize) {
  const int warps = (d + 31) / 32;
  if (esize == 8) return {warps, 1, 0};
  if (d > 64 && chains >= 2048) return {1, warps, 0};
  const int main = d & ~3;
  for (int D : {16, 32, 48, 64, 96})
    if (main <= D && d <= (D == 48 ? 64 : D)) return {warps, 1, D};
  return {warps, 1, 128};
}

template <typename T, int NW, int E, int CT, int D>
int launch_one(const State<T>& st, const Target<T>& tg, const hmc_schedule& sch, int64_t nprop, int dry, bool single,
               int groups, cudaStream_t stream) {
  HMC_REQUIRE(NW * groups <= 8, "persistent lanes: %d groups of %d warps exceed a block", groups, NW);
  const size_t slots = D > 0 ? D + 3 : tg.d;
  const size_t vecs = ((size_t)groups * (2 * slots + 2 * (size_t)sch.steps) + 15) & ~(size_t)15;
  const size_t smem = vecs * sizeof(Chains<T, CT>) + groups * sizeof(GroupShared<T, CT>) +
                      (D > 0 ? 0 : (size_t)tg.d * tg.ld * sizeof(T));
  HMC_REQUIRE(smem <= 227 * 1024, "persistent lanes: d = %d does not fit in shared memory", tg.d);
  auto kern = persistent_lanes_kernel<T, NW, E, CT, D>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(persistent_lanes_kernel)");
  }
  const int64_t per = (int64_t)CT * groups;
  kern<<<(unsigned)((st.C + per - 1) / per), 32 * NW * groups, smem, stream>>>(st, tg, sch, nprop, single, dry);
  return check_launch("persistent_lanes_kernel");
}

template <typename T, int CT>
int launch_width(const State<T>& st, const Target<T>& tg, const hmc_schedule& sch, int64_t nprop, int dry, bool single,
                 int groups, cudaStream_t stream) {
  const LanesLayout l = lanes_layout(tg.d, st.C, sizeof(T));
#define HMC_LANES(NW, E, D) launch_one<T, NW, E, CT, D>(st, tg, sch, nprop, dry, single, groups, stream)
  if constexpr (sizeof(T) == 4) {
    if (l.rows == 3) return HMC_LANES(1, 3, 0);
    if (l.rows == 4) return HMC_LANES(1, 4, 0);
    switch (l.cols) {
      case 16: return HMC_LANES(1, 1, 16);
      case 32: return HMC_LANES(1, 1, 32);
      case 48: return HMC_LANES(2, 1, 48);
      case 64: return HMC_LANES(2, 1, 64);
      case 96: return HMC_LANES(3, 1, 96);
      default: return HMC_LANES(4, 1, 128);
    }
  } else {
    switch (l.warps) {
      case 1: return HMC_LANES(1, 1, 0);
      case 2: return HMC_LANES(2, 1, 0);
      case 3: return HMC_LANES(3, 1, 0);
      default: return HMC_LANES(4, 1, 0);
    }
  }
#undef HMC_LANES
}

template <typename T>
int launch_lanes(const State<T>& st, const Target<T>& tg, const hmc_schedule& sch, int64_t nprop, int dry, bool single,
                 int chains, int groups, cudaStream_t stream) {
  switch (chains) {
    case 1: return launch_width<T, 1>(st, tg, sch, nprop, dry, single, groups, stream);
    case 2: return launch_width<T, 2>(st, tg, sch, nprop, dry, single, groups, stream);
    default:
      if constexpr (sizeof(T) == 4) return launch_width<T, 4>(st, tg, sch, nprop, dry, single, groups, stream);
      return fail(HMC_ERR_INVALID_ARG, "persistent lanes: 4 chains per group are FP32 only");
  }
}

template int launch_lanes<float>(const State<float>&, const Target<float>&, const hmc_schedule&, int64_t, int, bool, int,
                                 int, cudaStream_t);
template int launch_lanes<double>(const State<double>&, const Target<double>&, const hmc_schedule&, int64_t, int, bool,
                                  int, int, cudaStream_t);
}  // namespace pers
}  // namespace hmc
