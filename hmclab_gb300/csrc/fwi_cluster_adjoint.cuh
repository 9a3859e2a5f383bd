// Adjoint elastic simulation and gradients of one shot, a cluster per chain
// (fwi_cluster.cuh).
#pragma once

#include "fwi_cluster.cuh"
#include "quotient.cuh"

namespace hmc {
namespace fwi {

#define HMC_DP(a, b, c, d) ((CC1 * ((a) - (b)) + CC2 * ((c) - (d))) * g.inv_h)

__device__ __forceinline__ void stage4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// The same expressions as adj_velocity_kernel and adj_stress_kernel, in the
// same order.  Registers hold the adjoint fields and the five gradient sums of
// the thread's column; the operands of the transposed operators (t1 .. t5), two
// stored planes of the forward velocities and the parameters sit in shared
// memory.  A plane's copy starts when the buffer's last reader is done (after
// the velocity pass) and is waited for before the barrier of the stress pass.
template <int RZ, int PITCH>
__global__ void __launch_bounds__(PITCH, PITCH == 128 || (PITCH == 192 && RZ <= 7) ? 2 : 1)
    cluster_adjoint_kernel(const __grid_constant__ ShotAdjoint g) {
  extern __shared__ __align__(16) float smem[];
  __shared__ HaloBarriers bars;
  const int nx = g.nx, nz = g.nz;
  const int rank = (int)(blockIdx.x % (unsigned)g.R);
  const int64_t c = blockIdx.x / (unsigned)g.R;
  const int z0 = rank * RZ, i = threadIdx.x;
  const bool column = i < nx;
  const bool xin = i >= 2 && i < nx - 2;
  // shared memory, in rows of PITCH: thread-private parameters and the taper,
  // then row 0 of t1 and t4, of t2, t3 and t5 (halos: t2 and t4 rows -1, RZ and
  // RZ + 1, t3 and t5 rows -2, -1 and RZ), then two buffers of stored vx (rows
  // -1 .. RZ + 1) and vz (rows -2 .. RZ).  In the tallest strips t4 takes the
  // rows of t1, which has no halo, once all threads have read it, and t1 those
  // of t4 likewise.
  constexpr bool SHARE = adjoint_shares(RZ);
  constexpr int TP = 5 * RZ;
  constexpr int T1 = 6 * RZ + 1, T4 = SHARE ? T1 : T1 + RZ + 1, T2 = T4 + RZ + 3, T3 = T2 + RZ + 4,
                T5 = T3 + RZ + 3, P0 = T5 + RZ + 1, BUF = 2 * (RZ + 3);
  static_assert(P0 + 2 * BUF == adjoint_rows(RZ), "shared-memory rows");
  float* const my = smem + i;
#define ROW(r) my[(r) * PITCH]
  const int64_t cells = (int64_t)nx * nz;
  const float* store = g.store + c * g.planes * cells;

  float avx[RZ], avz[RZ], asxx[RZ], aszz[RZ], asxz[RZ], gl2m[RZ], glam[RZ], gmu[RZ], gbx[RZ], gbz[RZ];
  unsigned valid = 0, rec_rows = 0;
  int rec_first = 0;  // the receiver of the first such row
  bool tapered = false, exact = true;
  for (int r = 6 * RZ; r < adjoint_rows(RZ); ++r) ROW(r) = 0.f;
#pragma unroll
  for (int z = 0; z < RZ; ++z) {
    const int j = z0 + z;
    avx[z] = avz[z] = asxx[z] = aszz[z] = asxz[z] = 0.f;
#pragma unroll
    for (int k = 0; k < 6; ++k) ROW(k * RZ + z) = 0.f;
    gl2m[z] = glam[z] = gmu[z] = gbx[z] = gbz[z] = 0.f;
    if (j >= 2 && j < nz - 2) valid |= 1u << z;
    if (column && j < nz) {
      const int cell = j * nx + i;
      const int64_t k = (int64_t)cell * g.C + c;
      ROW(z) = g.bx[k];
      ROW(RZ + z) = g.bz[k];
      ROW(2 * RZ + z) = g.l2m[k];
      ROW(3 * RZ + z) = g.lam[k];
      ROW(4 * RZ + z) = g.dt * g.muxz[k];
      const float tp = g.taper[cell];
      ROW(TP + z) = tp;
      tapered = tapered || tp != 1.f;
      exact = exact && plain_divisor(ROW(z)) && plain_divisor(ROW(RZ + z)) && plain_divisor(tp);
      const int r = g.rec_map[cell];
      if (r >= 0) {
        if (!rec_rows) rec_first = r;
        rec_rows |= 1u << z;
      }
      gl2m[z] = g.g_l2m[k];
      glam[z] = g.g_lam[k];
      gmu[z] = g.g_muxz[k];
      gbx[z] = g.g_bx[k];
      gbz[z] = g.g_bz[k];
    }
  }
  // copy two stored planes (vx, vz) into a buffer, with their halo rows
  auto load_planes = [&](int buf, int64_t plane) {
    if (!column) return;
    const float* px = store + plane * cells + i;
    const float* pz = px + cells;
    float* b = &ROW(P0) + buf * (BUF * PITCH);
#pragma unroll
    for (int r = 0; r < RZ + 3; ++r) {
      const int jx = z0 + r - 1, jz = z0 + r - 2;
      if (jx >= 0 && jx < nz) stage4(b + r * PITCH, px + jx * nx);
      if (jz >= 0 && jz < nz) stage4(b + (RZ + 3 + r) * PITCH, pz + jz * nx);
    }
  };
  auto load_step = [&](int n) {  // what step n correlates with; at interval 1 its planes are there already
    if (g.snap == 1) {
      if (n > 0) load_planes((n - 1) & 1, 2 * (int64_t)(n - 1));
    } else if (n >= 0 && n % g.snap == 0) {
      load_planes(0, 4 * (int64_t)(n / g.snap));
      load_planes(1, 4 * (int64_t)(n / g.snap) + 2);
    }
  };
  const bool has_up = rank > 0, has_down = rank + 1 < g.R;
  const uint32_t bytes = (uint32_t)((has_up ? 12 : 0) + (has_down ? 12 : 0)) * (uint32_t)nx;
  if (i == 0) {
    halo_init(bars);
    halo_arm(bars, 0, bytes);
    halo_arm(bars, 1, bytes);
  }
  __syncthreads();
  if (g.snap == 1) load_planes((g.nt - 1) & 1, 2 * (int64_t)(g.nt - 1));
  load_step(g.nt - 1);
  if (g.snap > 1 && (g.nt - 1) % g.snap != 0) load_step((g.nt - 1) / g.snap * g.snap);
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  cluster_barrier();  // every block runs, with its halos cleared and its barriers ready
  const uint32_t base = smem_of(my), up = remote_of(base, has_up ? rank - 1 : rank),
                 down = remote_of(base, has_down ? rank + 1 : rank);
  const uint32_t up_bar = remote_of(smem_of(&bars), has_up ? rank - 1 : rank),
                 down_bar = remote_of(smem_of(&bars), has_down ? rank + 1 : rank);
  uint32_t parity = 0;
  bool dead = !halo_awaits(column);  // neither waits, sends nor arms
  const bool sends = halo_sends(column) && !(g.withhold && blockIdx.x == 0 && i == 0);
  // edge rows of the operands a (rows -1, RZ, RZ + 1) and b (rows -2, -1, RZ) to
  // the neighbours; k numbers the barrier
#define PUSH(k, a, b)                                                             \
  if (sends && !dead) {                                                           \
    if (has_down) {                                                               \
      halo_push(down + ((a)-1) * PITCH * 4, ROW((a) + RZ - 1), down_bar + 8 * k); \
      halo_push(down + ((b)-2) * PITCH * 4, ROW((b) + RZ - 2), down_bar + 8 * k); \
      halo_push(down + ((b)-1) * PITCH * 4, ROW((b) + RZ - 1), down_bar + 8 * k); \
    }                                                                             \
    if (has_up) {                                                                 \
      halo_push(up + ((a) + RZ) * PITCH * 4, ROW(a), up_bar + 8 * k);             \
      halo_push(up + ((a) + RZ + 1) * PITCH * 4, ROW((a) + 1), up_bar + 8 * k);   \
      halo_push(up + ((b) + RZ) * PITCH * 4, ROW(b), up_bar + 8 * k);             \
    }                                                                             \
  }
#define SETTLE(k)                                          \
  __syncthreads();                                         \
  if (bytes) { /* some neighbour */                        \
    halo_wait(bars, k, parity, g.wait_ns, g.status, dead); \
    if (i == 0 && !dead) halo_arm(bars, k, bytes);         \
  }

  auto stresses = [&]() {
    if (!xin) return;
#pragma unroll
    for (int z = 0; z < RZ; ++z) {
      const bool ok = valid >> z & 1u;
      const float* a4 = &ROW(T4 + z);
      const float* a5 = &ROW(T5 + z);
      const float xx = asxx[z] - HMC_DP(a4[0], a4[-1], a4[1], a4[-2]);
      const float xz =
          asxz[z] - HMC_DP(a4[PITCH], a4[0], a4[2 * PITCH], a4[-PITCH]) - HMC_DP(a5[1], a5[0], a5[2], a5[-1]);
      const float zz = aszz[z] - HMC_DP(a5[0], a5[-PITCH], a5[PITCH], a5[-2 * PITCH]);
      asxx[z] = ok ? xx : asxx[z];
      asxz[z] = ok ? xz : asxz[z];
      aszz[z] = ok ? zz : aszz[z];
    }
    if (tapered) {
#pragma unroll
      for (int z = 0; z < RZ; ++z)
        if (valid >> z & 1u) {
          const float tp = ROW(TP + z);
          asxx[z] *= tp;
          asxz[z] *= tp;
          aszz[z] *= tp;
        }
    }
#pragma unroll
    for (int z = 0; z < RZ; ++z)
      if (valid >> z & 1u) {
        const float l2m = ROW(2 * RZ + z), lam = ROW(3 * RZ + z);
        ROW(T2 + z) = g.dt * (lam * asxx[z] + l2m * aszz[z]);
        ROW(T3 + z) = ROW(4 * RZ + z) * asxz[z];
      }
  };

  float res_x = 0.f, res_z = 0.f;
  if (rec_rows) {
    const float* r = g.resid + ((int64_t)(g.nt - 1) * g.nrec + rec_first) * 2 * g.C + c;
    res_x = r[0];
    res_z = r[g.C];
  }
  const float w = g.w;
  for (int n = g.nt - 1; n >= 0; --n) {
    const bool corr = g.snap == 1 || n % g.snap == 0;
    const int bn = g.snap == 1 ? n & 1 : 0;
    // ---- adjoint velocities; the edge rows travel during the correlations
    if (xin) {
#pragma unroll
      for (int z = 0; z < RZ; ++z) {
        const bool ok = valid >> z & 1u;
        const float* a1 = &ROW(T1 + z);
        const float* a2 = &ROW(T2 + z);
        const float* a3 = &ROW(T3 + z);
        const float ax =
            avx[z] - HMC_DP(a1[1], a1[0], a1[2], a1[-1]) - HMC_DP(a3[0], a3[-PITCH], a3[PITCH], a3[-2 * PITCH]);
        const float az =
            avz[z] - HMC_DP(a2[PITCH], a2[0], a2[2 * PITCH], a2[-PITCH]) - HMC_DP(a3[0], a3[-1], a3[1], a3[-2]);
        avx[z] = ok ? ax : avx[z];
        avz[z] = ok ? az : avz[z];
      }
      if (rec_rows) {
#pragma unroll
        for (int z = 0; z < RZ; ++z)
          if (rec_rows >> z & 1u) {
            const bool first = !(rec_rows & ((1u << z) - 1));
            const int k = first ? rec_first : g.rec_map[(z0 + z) * nx + i];
            const float* r = g.resid + ((int64_t)n * g.nrec + k) * 2 * g.C + c;
            avx[z] += first ? res_x : r[0];
            avz[z] += first ? res_z : r[g.C];
          }
      }
      if (tapered) {  // x * 1 = x
#pragma unroll
        for (int z = 0; z < RZ; ++z)
          if (valid >> z & 1u) {
            const float tp = ROW(TP + z);
            avx[z] *= tp;
            avz[z] *= tp;
          }
      }
    }
    if (SHARE) __syncthreads();  // t1 has been read: its rows take t4
    if (xin) {
#pragma unroll
      for (int z = 0; z < RZ; ++z)
        if (valid >> z & 1u) {
          ROW(T4 + z) = g.dt * ROW(z) * avx[z];
          ROW(T5 + z) = g.dt * ROW(RZ + z) * avz[z];
        }
    }
    PUSH(0, T4, T5)
    // ---- the gradients
    if (xin) {
      const float* fx = &ROW(P0 + 1) + bn * (BUF * PITCH);           // row 0 of vx
      const float* fz = fx + (RZ + 4) * PITCH;                       // row 0 of vz
      const float* ox = &ROW(P0 + 1) + (bn ^ 1) * (BUF * PITCH);
      const float* oz = ox + (RZ + 4) * PITCH;
      const bool before = g.snap > 1 || n > 0;
      if (corr) {
#pragma unroll
        for (int z = 0; z < RZ; ++z) {
          const bool ok = valid >> z & 1u;
          const float* px = fx + z * PITCH;
          const float* pz = fz + z * PITCH;
          const float exx = HMC_DP(px[0], px[-1], px[1], px[-2]);
          const float ezz = HMC_DP(pz[0], pz[-PITCH], pz[PITCH], pz[-2 * PITCH]);
          const float exz =
              HMC_DP(px[PITCH], px[0], px[2 * PITCH], px[-PITCH]) + HMC_DP(pz[1], pz[0], pz[2], pz[-1]);
          const float wdt = w * g.dt;
          const float n1 = gl2m[z] + wdt * (exx * asxx[z] + ezz * aszz[z]);
          // the rounding of the per-step kernels, written out
          const float n2 = glam[z] + wdt * fmaf(exx, aszz[z], __fmul_rn(ezz, asxx[z]));
          const float n3 = gmu[z] + wdt * exz * asxz[z];
          gl2m[z] = ok ? n1 : gl2m[z];
          glam[z] = ok ? n2 : glam[z];
          gmu[z] = ok ? n3 : gmu[z];
        }
        unsigned slow = exact ? 0u : valid;  // rows whose quotients take the general division
#pragma unroll
        for (int z = 0; z < RZ; ++z) {
          const float vxp = before ? ox[z * PITCH] : 0.f, vzp = before ? oz[z * PITCH] : 0.f;
          float vxt = fx[z * PITCH], vzt = fz[z * PITCH];
          bool plain = true;
          if (tapered) {  // x / 1 = x
            const float rtp = reciprocal(ROW(TP + z));
            vxt = quotient(vxt, ROW(TP + z), rtp, plain);
            vzt = quotient(vzt, ROW(TP + z), rtp, plain);
          }
          const float dvx = (vxt - vxp) * w;
          const float dvz = (vzt - vzp) * w;
          const float n1 = gbx[z] + quotient(dvx, ROW(z), reciprocal(ROW(z)), plain) * avx[z];
          const float n2 = gbz[z] + quotient(dvz, ROW(RZ + z), reciprocal(ROW(RZ + z)), plain) * avz[z];
          if (!plain) slow |= valid & 1u << z;
          const bool ok = (valid & ~slow) >> z & 1u;
          gbx[z] = ok ? n1 : gbx[z];
          gbz[z] = ok ? n2 : gbz[z];
        }
        if (slow) {
#pragma unroll
          for (int z = 0; z < RZ; ++z) {
            if (!(slow >> z & 1u)) continue;
            const float vxp = before ? ox[z * PITCH] : 0.f, vzp = before ? oz[z * PITCH] : 0.f;
            const float dvx = (fx[z * PITCH] / ROW(TP + z) - vxp) * w;
            const float dvz = (fz[z * PITCH] / ROW(TP + z) - vzp) * w;
            gbx[z] = gbx[z] + dvx / ROW(z) * avx[z];
            gbz[z] = gbz[z] + dvz / ROW(RZ + z) * avz[z];
          }
        }
      }
    }
    SETTLE(0)
    // the buffers whose last readers are past the barrier take the next planes
    if (g.snap == 1) {
      load_step(n - 1);
    } else if (corr) {
      load_step(n - g.snap);
    }
    if (rec_rows && n > 0) {  // the next step's residuals, ahead of their use
      const float* r = g.resid + ((int64_t)(n - 1) * g.nrec + rec_first) * 2 * g.C + c;
      res_x = r[0];
      res_z = r[g.C];
    }
    // ---- adjoint stresses
    stresses();
    PUSH(1, T2, T3)
    if (SHARE) __syncthreads();  // t4 has been read: its rows take t1
    if (xin) {
#pragma unroll
      for (int z = 0; z < RZ; ++z)
        if (valid >> z & 1u) ROW(T1 + z) = g.dt * (ROW(2 * RZ + z) * asxx[z] + ROW(3 * RZ + z) * aszz[z]);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    SETTLE(1)
    parity ^= 1;
  }
  if (column) {
#pragma unroll
    for (int z = 0; z < RZ; ++z) {
      const int j = z0 + z;
      if (j >= nz) break;
      const int64_t k = ((int64_t)j * nx + i) * g.C + c;
      g.g_l2m[k] = gl2m[z];
      g.g_lam[k] = glam[z];
      g.g_muxz[k] = gmu[z];
      g.g_bx[k] = gbx[z];
      g.g_bz[k] = gbz[z];
    }
  }
  halo_drain(dead && column, g.status);
  cluster_barrier();  // no block leaves while a neighbour may push to it
#undef SETTLE
#undef PUSH
#undef ROW
}
#undef HMC_DP

template <int PITCH>
int cluster_adjoint_at(const ShotAdjoint& a, bool dry, Strip* strip, cudaStream_t st) {
  ClusterChoice best;
#define HMC_STRIP(RZ) \
  consider_strip(best, cluster_adjoint_kernel<RZ, PITCH>, RZ, adjoint_rows(RZ) * PITCH, a.nx, a.nz, a.C, 210.0, \
                 ADJOINT_STEP);
  HMC_ADJOINT_STRIPS(HMC_STRIP)
#undef HMC_STRIP
  *strip = Strip{best.rz, best.step_us};
  if (dry || best.rz == 0) return HMC_OK;
  ShotAdjoint g = a;
  g.R = best.R;
  switch (best.rz) {
#define HMC_STRIP(RZ) \
  case RZ: \
    return launch_cluster("cluster_adjoint_kernel", cluster_adjoint_kernel<RZ, PITCH>, adjoint_rows(RZ) * PITCH, a.nx, \
                          best.R, a.C, st, g);
    HMC_ADJOINT_STRIPS(HMC_STRIP)
#undef HMC_STRIP
  }
  return HMC_OK;
}

}  // namespace fwi
}  // namespace hmc
