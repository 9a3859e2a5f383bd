// Persistent proposals of a few chains on a small dense target: a cluster of
// blocks advances one chain, its blocks own consecutive rows and KC lanes
// share a row.
#include <cooperative_groups.h>

#include "persistent.cuh"

namespace hmc {
namespace pers {

constexpr int ROWS_MAX_CLUSTER = 8;
constexpr int ROWS_MAX_THREADS = 512;

template <typename T>
struct RowsShared {
  T q[2][MAX_D];           // published positions, double-buffered
  T z[4][MAX_D / 4];       // radius and angle parts of the block's quads
  T z2[2][MAX_D / 4];
  T kick[HMC_SCHEDULE_MAX], drift[HMC_SCHEDULE_MAX], first;
  double u;
  double part[ROWS_MAX_THREADS / 32][2];
  double total[ROWS_MAX_CLUSTER][2];  // misfit, K1 - K0
  int accept;
};

// Row stride of the block's part of GtG: KC lanes of 32 / KC rows read
// consecutive columns, without bank conflicts when the stride is KC modulo a
// 128-byte line (FP64 reads go by half warps).
template <typename T, int KC>
__host__ __device__ constexpr int rows_stride(int d) {
  const int line = 128 / (int)sizeof(T);
  int ld = (d + line - 1) / line * line + KC;
  return ld - line >= d ? ld - line : ld;
}

// Bound by the latency of one step: FP64 issues one warp instruction per 64
// cycles and scheduler, so a step of d = 50 is 7 products, 3 sums across the
// row's lanes and the update, then the cluster barrier that publishes q; the
// momenta (one warp per part of Box-Muller), the sums of the energies and the
// exponential take the rest of a proposal.  One FP64 chain, 10 steps: d = 50
// 17.9 us on four blocks against 69 us with the chain in one warp; d = 128
// 24.1 against 271 us.  FP32 chains do better with a thread per row (d = 100:
// 13.3 us here, 8.1 there).
template <typename T, int KC>
__global__ void __launch_bounds__(ROWS_MAX_THREADS) persistent_rows_kernel(State<T> s, Target<T> tg,
                                                                           const __grid_constant__ hmc_schedule sch,
                                                                           int64_t nprop, bool single, int cluster,
                                                                           int dry) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ RowsShared<T> sh;
  const cg::cluster_group peers = cg::this_cluster();
  const int d = tg.d, quads = (d + 3) / 4, own_quads = (quads + cluster - 1) / cluster;
  const int rank = (int)(blockIdx.x % (unsigned)cluster);
  const int64_t c = blockIdx.x / (unsigned)cluster;
  const int row0 = 4 * own_quads * rank;
  const int rows = d - row0 < 4 * own_quads ? d - row0 : 4 * own_quads;  // none or less for the last blocks
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r = tid / KC, kc = tid % KC;
  const bool live = r < rows;
  const int i = live ? row0 + r : 0;
  const bool diag = s.mass == HMC_MASS_DIAG;
  const int prior = tg.prior;
  const int ld = rows_stride<T, KC>(d);
  T* A = (T*)smem_raw;
  for (int k = tid; k < rows * d; k += blockDim.x) A[(k / d) * ld + k % d] = tg.GtG[(int64_t)(row0 + k / d) * d + k % d];
  const T* a = A + (live ? r : 0) * ld;
  const T minv = diag ? s.minv[i] : (T)1, msq = diag ? mass_root(s.mdiag[i]) : (T)1, gtd = tg.Gtd0[i];
  const T pm = prior != PRIOR_NONE ? tg.pmean[i] : (T)0, pw = prior != PRIOR_NONE ? tg.pw[i] : (T)0;
  T qc = s.q_cur[(int64_t)i * s.C + c];
  double xc = s.x_cur[c];
  const T eps0 = s.eps[c];
  int64_t n_acc = 0;
  const int64_t n0 = s.control[0];
  int buf = 0;
  auto sync = [&] {
    if (cluster > 1)
      peers.sync();
    else
      __syncthreads();
  };
  // GtG q of the thread's row from everyone's q: each row's lanes write it to
  // the blocks, the barrier publishes it, and the other buffer takes the next
  // one while slower blocks still read this one.
  auto matvec = [&](T q) -> T {
    if (live)
      for (int k = kc; k < cluster; k += KC) {
        T* to = cluster > 1 ? peers.map_shared_rank(&sh.q[buf][0], k) : sh.q[buf];
        to[i] = q;
      }
    sync();
    const T* x = sh.q[buf];
    buf ^= 1;
    T v = (T)0;
#pragma unroll 4
    for (int j = kc; j < d; j += KC) v = fma(a[j], x[j], v);
#pragma unroll
    for (int o = 1; o < KC; o *= 2) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  };
  __syncthreads();
  if (cluster > 1) peers.sync();  // every block of the cluster runs before its shared memory is written

  for (int64_t t = 0; t < nprop; ++t) {
    const int64_t n = n0 + t;
    // the four parts of Box-Muller of the block's quads, one warp each
    if (!s.sz && warp < 4 && lane < own_quads && row0 / 4 + lane < quads) {
      T u[4];
      philox_uniforms4<T>(s.seed, (uint32_t)(row0 / 4 + lane), (uint32_t)c, (uint64_t)n, PURPOSE_MOMENTUM, u);
      if (warp == 0) sh.z[0][lane] = normal_radius(u[0]);
      if (warp == 1) normal_angle(u[1], sh.z[1][lane], sh.z2[0][lane]);
      if (warp == 2) sh.z[2][lane] = normal_radius(u[2]);
      if (warp == 3) normal_angle(u[3], sh.z[3][lane], sh.z2[1][lane]);
    }
    // step size, accept uniform and the steps' coefficients: every lane of the
    // last warp forms the step size, lane l the coefficients of step l
    if (warp == (int)blockDim.x / 32 - 1) {
      double ue = 0.0, ua = 0.0;
      if (!s.seps || !s.su) philox_scalars(s.seed, (uint32_t)c, (uint64_t)n, &ue, &ua);
      T e = eps0;
      if (s.randomize) e *= s.seps ? s.seps[(n % s.slen) * s.C + c] : (T)(0.5 + ue);
      for (int l = lane; l < sch.steps; l += 32) {
        sh.kick[l] = scaled_step(sch.kick[l], single, e);
        sh.drift[l] = scaled_step(sch.drift[l], single, e);
      }
      if (lane == 31) {
        sh.u = s.su ? s.su[(n % s.slen) * s.C + c] : ua;
        sh.first = scaled_step(sch.first_drift, single, e);
      }
    }
    __syncthreads();
    T p = (T)0, q = qc;
    double dk = 0.0, x = 0.0;
    if (live) {
      T z;
      if (s.sz) {
        z = s.sz[((n % s.slen) * d + i) * s.C + c];
      } else {
        const int lq = r >> 2, j = r & 3;
        const T part = j == 0 ? sh.z[1][lq] : (j == 1 ? sh.z2[0][lq] : (j == 2 ? sh.z[3][lq] : sh.z2[1][lq]));
        z = sh.z[j & 2][lq] * part;
      }
      p = diag ? msq * z : z;
      const T mp = diag ? minv * p : p;
      dk = -(f64_of(p) * f64_of(mp));
      q = fma(sh.first, mp, qc);
    }
    for (int st = 0; st < sch.steps; ++st) {
      if (sch.gradient[st]) {
        const T dq = pm - q;  // the prior's part does not wait for the product
        T gk = matvec(q) - gtd;
        if (prior == PRIOR_NORMAL) gk = fma(-pw, dq, gk);
        if (prior == PRIOR_LAPLACE) gk = gk + sign_of(-dq) * pw;
        p = fma(-sh.kick[st], gk, p);
      }
      if (sch.drift[st] != 0.0) q = fma(sh.drift[st], diag ? minv * p : p, q);
    }
    const T w = fma((T)-2, gtd, matvec(q));
    if (live) {
      x = f64_of(q) * f64_of(w);
      if (prior == PRIOR_NORMAL) {
        const T dq = pm - q;
        x = fma(f64_of(dq), f64_of(pw * dq), x);
      }
      if (prior == PRIOR_LAPLACE) x = fma(2.0, f64_of((T)(fabs(q - pm) * pw)), x);
      dk = fma(f64_of(p), f64_of(diag ? minv * p : p), dk);
    }
    // sums over the rows: the lanes of a row hold the same value
#pragma unroll
    for (int o = KC; o < 32; o *= 2) {
      x += __shfl_xor_sync(0xffffffffu, x, o);
      dk += __shfl_xor_sync(0xffffffffu, dk, o);
    }
    if (lane == 0) {
      sh.part[warp][0] = x;
      sh.part[warp][1] = dk;
    }
    __syncthreads();
    if (tid < 2) {
      double v = 0.0;
      for (int k = 0; k < (int)blockDim.x / 32; ++k) v += sh.part[k][tid];
      for (int k = 0; k < cluster; ++k)
        *(cluster > 1 ? peers.map_shared_rank(&sh.total[rank][tid], k) : &sh.total[rank][tid]) = v;
    }
    sync();
    if (warp == 0) {  // the same sums in every block: all take the same decision
      double v = 0.0;
      if (lane < 2)
        for (int k = 0; k < cluster; ++k) v += sh.total[k][lane];
      const double x1 = 0.5 * (__shfl_sync(0xffffffffu, v, 0) + tg.dtd);
      const double d1 = 0.5 * __shfl_sync(0xffffffffu, v, 1);
      if (lane == 0) {
        sh.accept = accept_test(xc - (x1 + d1), sh.u) ? 1 : 0;
        if (sh.accept) {
          xc = x1;
          ++n_acc;
        }
      }
    }
    __syncthreads();
    if (sh.accept) qc = q;
    if (!dry && s.ring_q && (n % s.thin) == 0) {
      const int64_t slot = (n / s.thin) % s.ring_slots;
      if (live && kc == 0) s.ring_q[(slot * d + i) * s.C + c] = qc;
      if (rank == 0 && tid == 0) s.ring_x[slot * s.C + c] = xc;
    }
  }
  if (!dry) {
    if (live && kc == 0) s.q_cur[(int64_t)i * s.C + c] = qc;
    if (rank == 0 && tid == 0) {
      s.x_cur[c] = xc;
      s.accepted[c] += n_acc;
    }
  }
  if (cluster > 1) peers.sync();  // no block leaves while its shared memory may be written
}


template <typename T>
int launch_rows(const State<T>& st, const Target<T>& tg, const hmc_schedule& sch, int64_t nprop, int dry, bool single,
                int cluster, cudaStream_t stream) {
  constexpr int KC = 8;
  HMC_REQUIRE(cluster == 1 || cluster == 2 || cluster == 4 || cluster == 8, "persistent rows: cluster of %d blocks",
              cluster);
  const int quads = (tg.d + 3) / 4, own_quads = (quads + cluster - 1) / cluster;
  int threads = (KC * 4 * own_quads + 31) / 32 * 32;
  threads = threads < 128 ? 128 : threads;  // four warps draw the momenta
  HMC_REQUIRE(threads <= ROWS_MAX_THREADS, "persistent rows: d = %d needs a larger cluster", tg.d);
  HMC_REQUIRE(st.C * cluster <= 0x7FFFFFFF, "persistent rows: too many chains");
  const size_t smem = (size_t)4 * own_quads * rows_stride<T, KC>(tg.d) * sizeof(T);
  auto kern = persistent_rows_kernel<T, KC>;
  if (smem > 40 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(persistent_rows_kernel)");
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(st.C * cluster));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim = {(unsigned)cluster, 1, 1};
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, st, tg, sch, nprop, single, cluster, dry);
  if (e != cudaSuccess) return cuda_fail(e, "persistent_rows_kernel");
  return check_launch("persistent_rows_kernel");
}

template int launch_rows<double>(const State<double>&, const Target<double>&, const hmc_schedule&, int64_t, int, bool,
                                 int, cudaStream_t);

}  // namespace pers
}  // namespace hmc
