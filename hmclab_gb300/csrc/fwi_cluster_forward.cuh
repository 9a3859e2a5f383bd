// Forward elastic simulation of one shot, a cluster per chain (fwi_cluster.cuh).
#pragma once

#include "fwi_cluster.cuh"

namespace hmc {
namespace fwi {

#define HMC_DP(a, b, c, d) ((CC1 * ((a) - (b)) + CC2 * ((c) - (d))) * g.inv_h)

// The same expressions as velocity_kernel and stress_kernel, in the same order.
template <int RZ, int PITCH>
__global__ void __launch_bounds__(PITCH, (RZ <= 10 ? 512 : 256) / PITCH)
    cluster_forward_kernel(const __grid_constant__ ShotForward g, const __grid_constant__ Waves src) {
  extern __shared__ __align__(16) float smem[];
  __shared__ HaloBarriers bars;
  const int nx = g.nx, nz = g.nz;
  const int rank = (int)(blockIdx.x % (unsigned)g.R);
  const int64_t c = blockIdx.x / (unsigned)g.R;
  const int z0 = rank * RZ, i = threadIdx.x;
  const bool column = i < nx;
  const bool xin = i >= 2 && i < nx - 2;
  // shared memory, in rows of PITCH: thread-private parameters, the published
  // rows, then the halos (sxz and vz: rows -2, -1, RZ; szz and vx: -1, RZ, RZ + 1)
  constexpr int O_SXX = 6 * RZ, O_SXZ = 7 * RZ, O_VX = 8 * RZ, O_VZ = 9 * RZ;
  constexpr int H_SXZ = 10 * RZ, H_SZZ = H_SXZ + 3, H_VZ = H_SZZ + 3, H_VX = H_VZ + 3;
  float* const my = smem + i;
#define ROW(r) my[(r) * PITCH]
  float vx[RZ], vz[RZ], sxx[RZ], szz[RZ], sxz[RZ];
  unsigned inside = 0, valid = 0, rec_rows = 0, src_terms = 0;  // rows of the grid, updated rows, rows with a receiver
  bool tapered = false;
  int rec_first = 0;  // the receiver of the first such row (loading it from the map each step would stall the strip)
#pragma unroll
  for (int z = 0; z < RZ; ++z) {
    const int j = z0 + z;
    vx[z] = vz[z] = sxx[z] = szz[z] = sxz[z] = 0.f;
    ROW(z) = ROW(RZ + z) = ROW(2 * RZ + z) = ROW(3 * RZ + z) = ROW(4 * RZ + z) = 0.f;
    ROW(5 * RZ + z) = 1.f;
    if (j < nz) inside |= 1u << z;
    if (j >= 2 && j < nz - 2) valid |= 1u << z;
    if (column && j < nz) {
      const int cell = j * nx + i;
      const int64_t k = (int64_t)cell * g.C + c;
      ROW(z) = g.dt * g.bx[k];
      ROW(RZ + z) = g.dt * g.bz[k];
      ROW(2 * RZ + z) = g.l2m[k];
      ROW(3 * RZ + z) = g.lam[k];
      ROW(4 * RZ + z) = g.dt * g.muxz[k];
      const float tp = g.taper[cell];
      ROW(5 * RZ + z) = tp;
      tapered = tapered || tp != 1.f;
      const int r = g.rec_map[cell];
      if (r >= 0) {
        if (!rec_rows) rec_first = r;
        rec_rows |= 1u << z;
      }
      if (g.load) {
        vx[z] = g.vx[k];
        vz[z] = g.vz[k];
        sxx[z] = g.sxx[k];
        szz[z] = g.szz[k];
        sxz[z] = g.sxz[k];
      }
    }
  }
  for (int t = 0; t < src.n_terms; ++t)
    if (src.i[t] == i && src.j[t] >= z0 && src.j[t] < z0 + RZ) src_terms |= 1u << t;
  if (column)
#pragma unroll
    for (int k = 0; k < 12; ++k) ROW(H_SXZ + k) = 0.f;
  const bool has_up = rank > 0, has_down = rank + 1 < g.R;
  const uint32_t bytes = (uint32_t)((has_up ? 12 : 0) + (has_down ? 12 : 0)) * (uint32_t)nx;
  if (i == 0) {
    halo_init(bars);
    halo_arm(bars, 0, bytes);
    halo_arm(bars, 1, bytes);
  }
  __syncthreads();
  cluster_barrier();  // every block runs, with its halos cleared and its barriers ready
  const uint32_t base = smem_of(my), up = remote_of(base, has_up ? rank - 1 : rank),
                 down = remote_of(base, has_down ? rank + 1 : rank);
  const uint32_t up_bar = remote_of(smem_of(&bars), has_up ? rank - 1 : rank),
                 down_bar = remote_of(smem_of(&bars), has_down ? rank + 1 : rank);
  uint32_t parity = 0;
  bool dead = !halo_awaits(column);  // neither waits, sends nor arms
  const bool sends = halo_sends(column) && !(g.withhold && blockIdx.x == 0 && i == 0);

  // Edge rows to the neighbours: fa is differentiated downwards (rows -2, -1,
  // RZ) and fb upwards (rows -1, RZ, RZ + 1); k numbers the barrier.
#define PUSH(k, fa, fb, ha, hb)                                             \
  if (sends && !dead) {                                                     \
    if (has_down) {                                                         \
      halo_push(down + (ha) * PITCH * 4, fa[RZ - 2], down_bar + 8 * k);     \
      halo_push(down + (ha + 1) * PITCH * 4, fa[RZ - 1], down_bar + 8 * k); \
      halo_push(down + (hb) * PITCH * 4, fb[RZ - 1], down_bar + 8 * k);     \
    }                                                                       \
    if (has_up) {                                                           \
      halo_push(up + (ha + 2) * PITCH * 4, fa[0], up_bar + 8 * k);          \
      halo_push(up + (hb + 1) * PITCH * 4, fb[0], up_bar + 8 * k);          \
      halo_push(up + (hb + 2) * PITCH * 4, fb[1], up_bar + 8 * k);          \
    }                                                                       \
  }
  // The rows differentiated along x to this block's threads, then the
  // neighbours' edge rows.
#define PUBLISH(k, fa, oa, fb, ob)                           \
  if (column) {                                              \
    _Pragma("unroll") for (int z = 0; z < RZ; ++z) {         \
      ROW(oa + z) = fa[z];                                   \
      ROW(ob + z) = fb[z];                                   \
    }                                                        \
  }                                                          \
  __syncthreads();                                           \
  if (bytes) { /* some neighbour */                          \
    halo_wait(bars, k, parity, g.wait_ns, g.status, dead);   \
    if (i == 0 && !dead) halo_arm(bars, k, bytes);           \
  }

  const int64_t cells = (int64_t)nx * nz;
  float* store = g.store ? g.store + c * g.planes * cells + (int64_t)z0 * nx + i : nullptr;
  auto velocities = [&]() {
    if (xin) {
      const float a_m2 = ROW(H_SXZ), a_m1 = ROW(H_SXZ + 1), a_p = ROW(H_SXZ + 2);
      const float b_m1 = ROW(H_SZZ), b_p0 = ROW(H_SZZ + 1), b_p1 = ROW(H_SZZ + 2);
#pragma unroll
      for (int z = 0; z < RZ; ++z) {
        const bool ok = valid >> z & 1u;
        const float* x = &ROW(O_SXX + z);
        const float dsxx = HMC_DP(x[1], sxx[z], x[2], x[-1]);
        const float m1 = z >= 1 ? sxz[z >= 1 ? z - 1 : 0] : a_m1;
        const float m2 = z >= 2 ? sxz[z >= 2 ? z - 2 : 0] : (z == 1 ? a_m1 : a_m2);
        const float p1 = z + 1 < RZ ? sxz[z + 1 < RZ ? z + 1 : 0] : a_p;
        const float dsxz_z = HMC_DP(sxz[z], m1, p1, m2);
        const float nvx = vx[z] + ROW(z) * (dsxx + dsxz_z);
        vx[z] = ok ? nvx : vx[z];
        const float* y = &ROW(O_SXZ + z);
        const float dsxz_x = HMC_DP(sxz[z], y[-1], y[1], y[-2]);
        const float q1 = z + 1 < RZ ? szz[z + 1 < RZ ? z + 1 : 0] : b_p0;
        const float q2 = z + 2 < RZ ? szz[z + 2 < RZ ? z + 2 : 0] : (z + 2 == RZ ? b_p0 : b_p1);
        const float q0 = z >= 1 ? szz[z >= 1 ? z - 1 : 0] : b_m1;
        const float dszz = HMC_DP(q1, szz[z], q2, q0);
        const float nvz = vz[z] + ROW(RZ + z) * (dsxz_x + dszz);
        vz[z] = ok ? nvz : vz[z];
      }
    }
    if (tapered) {  // x * 1 = x
#pragma unroll
      for (int z = 0; z < RZ; ++z) {
        vx[z] *= ROW(5 * RZ + z);
        vz[z] *= ROW(5 * RZ + z);
      }
    }
  };
  auto stresses = [&](const int n) {
    if (xin) {
      const float a_m2 = ROW(H_VZ), a_m1 = ROW(H_VZ + 1), a_p = ROW(H_VZ + 2);
      const float b_m1 = ROW(H_VX), b_p0 = ROW(H_VX + 1), b_p1 = ROW(H_VX + 2);
#pragma unroll
      for (int z = 0; z < RZ; ++z) {
        const bool ok = valid >> z & 1u;
        const float* x = &ROW(O_VX + z);
        const float exx = HMC_DP(vx[z], x[-1], x[1], x[-2]);
        const float m1 = z >= 1 ? vz[z >= 1 ? z - 1 : 0] : a_m1;
        const float m2 = z >= 2 ? vz[z >= 2 ? z - 2 : 0] : (z == 1 ? a_m1 : a_m2);
        const float p1 = z + 1 < RZ ? vz[z + 1 < RZ ? z + 1 : 0] : a_p;
        const float ezz = HMC_DP(vz[z], m1, p1, m2);
        const float l2m = ROW(2 * RZ + z), lam = ROW(3 * RZ + z);
        const float nxx = sxx[z] + g.dt * (l2m * exx + lam * ezz), nzz = szz[z] + g.dt * (lam * exx + l2m * ezz);
        sxx[z] = ok ? nxx : sxx[z];
        szz[z] = ok ? nzz : szz[z];
        const float q1 = z + 1 < RZ ? vx[z + 1 < RZ ? z + 1 : 0] : b_p0;
        const float q2 = z + 2 < RZ ? vx[z + 2 < RZ ? z + 2 : 0] : (z + 2 == RZ ? b_p0 : b_p1);
        const float q0 = z >= 1 ? vx[z >= 1 ? z - 1 : 0] : b_m1;
        const float dvx = HMC_DP(q1, vx[z], q2, q0);
        const float* y = &ROW(O_VZ + z);
        const float dvz = HMC_DP(y[1], vz[z], y[2], y[-1]);
        const float nxz = sxz[z] + ROW(4 * RZ + z) * (dvx + dvz);
        sxz[z] = ok ? nxz : sxz[z];
      }
    }
    for (unsigned m = src_terms; m; m &= m - 1) {
      const int t = __ffs(m) - 1, row = src.j[t] - z0;
      const float s = src.s[src.first[t] + n - g.n0];
#pragma unroll
      for (int z = 0; z < RZ; ++z)
        if (z == row) {  // the amounts are rounded before they are added
          sxx[z] += __fmul_rn(src.xx[t], s);
          szz[z] += __fmul_rn(src.zz[t], s);
          sxz[z] += __fmul_rn(src.xz[t], s);
        }
    }
    if (tapered) {
#pragma unroll
      for (int z = 0; z < RZ; ++z) {
        sxx[z] *= ROW(5 * RZ + z);
        szz[z] *= ROW(5 * RZ + z);
        sxz[z] *= ROW(5 * RZ + z);
      }
    }
  };
  PUSH(0, sxz, szz, H_SXZ, H_SZZ)
  PUBLISH(0, sxx, O_SXX, sxz, O_SXZ)
  for (int n = g.n0; n < g.n1; ++n) {
    float* now = nullptr;
    if (store && column) {
      if (g.snap == 1) {
        now = store + 2 * (int64_t)n * cells;
      } else if (n % g.snap == 0) {
        now = store + 4 * (int64_t)(n / g.snap) * cells;
        float* prev = now + 2 * cells;  // a snapshot keeps the velocities of the step before too
#pragma unroll
        for (int z = 0; z < RZ; ++z)
          if (inside >> z & 1u) {
            prev[z * nx] = vx[z];
            prev[cells + z * nx] = vz[z];
          }
      }
    }
    velocities();
    PUSH(1, vz, vx, H_VZ, H_VX)
    if (now) {
#pragma unroll
      for (int z = 0; z < RZ; ++z)
        if (inside >> z & 1u) {
          now[z * nx] = vx[z];
          now[cells + z * nx] = vz[z];
        }
    }
    if (rec_rows) {
#pragma unroll
      for (int z = 0; z < RZ; ++z)
        if (rec_rows >> z & 1u) {
          const int r = (rec_rows & ((1u << z) - 1)) ? g.rec_map[(z0 + z) * nx + i] : rec_first;
          float* o = g.rec + ((int64_t)n * g.nrec + r) * 2 * g.C + c;
          o[0] = vx[z];
          o[g.C] = vz[z];
        }
    }
    PUBLISH(1, vx, O_VX, vz, O_VZ)
    parity ^= 1;
    stresses(n);
    PUSH(0, sxz, szz, H_SXZ, H_SZZ)
    PUBLISH(0, sxx, O_SXX, sxz, O_SXZ)
  }
  if (g.save && column) {
#pragma unroll
    for (int z = 0; z < RZ; ++z)
      if (inside >> z & 1u) {
        const int64_t k = ((int64_t)(z0 + z) * nx + i) * g.C + c;
        g.vx[k] = vx[z];
        g.vz[k] = vz[z];
        g.sxx[k] = sxx[z];
        g.szz[k] = szz[z];
        g.sxz[k] = sxz[z];
      }
  }
  halo_drain(dead && column, g.status);
  cluster_barrier();  // no block leaves while a neighbour may push to it
#undef PUSH
#undef PUBLISH
#undef ROW
}
#undef HMC_DP

template <int PITCH>
int cluster_forward_at(const ShotForward& a, const Waves& w, bool dry, Strip* strip, cudaStream_t st) {
  ClusterChoice best;
#define HMC_STRIP(RZ) \
  consider_strip(best, cluster_forward_kernel<RZ, PITCH>, RZ, forward_rows(RZ) * PITCH, a.nx, a.nz, a.C, 75.0, \
                 a.store ? STORING_STEP : FORWARD_STEP);
  HMC_FORWARD_STRIPS(HMC_STRIP)
#undef HMC_STRIP
  *strip = Strip{best.rz, best.step_us};
  if (dry || best.rz == 0) return HMC_OK;
  ShotForward g = a;
  g.R = best.R;
  switch (best.rz) {
#define HMC_STRIP(RZ) \
  case RZ: \
    return launch_cluster("cluster_forward_kernel", cluster_forward_kernel<RZ, PITCH>, forward_rows(RZ) * PITCH, a.nx, \
                          best.R, a.C, st, g, w);
    HMC_FORWARD_STRIPS(HMC_STRIP)
#undef HMC_STRIP
  }
  return HMC_OK;
}

}  // namespace fwi
}  // namespace hmc
