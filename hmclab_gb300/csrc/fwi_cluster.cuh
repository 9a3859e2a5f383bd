// Elastic time loops with the wavefield on chip: one thread-block cluster per
// chain advances a whole shot in one launch (fwi_cluster_forward.cuh,
// fwi_cluster_adjoint.cuh; fwi.cu holds the scheme and the per-step kernels).
//
// A block of the cluster owns RZ consecutive rows of the grid, a thread one
// column of them; the fields it owns stay in its registers for all time steps.
// Horizontal neighbours come from shared memory, vertical ones from the
// thread's own registers or, at the strip's edges, from halo rows that the two
// neighbouring blocks push into this block's shared memory with asynchronous
// remote stores, which complete on a barrier of this block: a half step waits
// for its neighbours only.  (A cluster barrier per half step took 650 cycles
// and, by its release, waited for the stored wavefield to reach L2.)  Nothing
// but the stored wavefield, the records and the parameters touches memory,
// where a launch per half step moved 172 MB through L2 per time step of 64
// chains.  Halos need one buffer: a neighbour sends the next ones only after
// it has this block's answer, which is sent after the last ones were read.
//
// What bounds a step (240 x 140 cells, one chain, 16 blocks of 9 rows, clocks):
// forward 3900, of which 840 and 1000 issue the two half steps' instructions at
// two warps per scheduler and 700 each wait for the halos; adjoint 7500 - 9000,
// of which shared-memory accesses (41 per cell) alone hold the SM's 128-byte
// port for 3000.  Sending the edge rows before the inner ones are computed
// (more overlap, less instruction-level parallelism) was 10 % slower.
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"
#include "fwi_choice.cuh"
#include "halo_rules.cuh"

namespace hmc {
namespace fwi {

constexpr float CC1 = 9.0f / 8.0f;
constexpr float CC2 = -1.0f / 24.0f;

constexpr int CLUSTER_MAX = 16;      // blocks per cluster (16 needs the non-portable opt-in)
constexpr int CLUSTER_COLUMNS = 256; // columns of the grid: one thread each, up to 255 registers
constexpr int WAVE_SAMPLES = 6000;   // source samples passed by value with a launch
constexpr int WAVE_TERMS = 32;       // stress terms (a moment tensor with Mxz takes four)

// Source terms of the steps n0 .. n1-1: term t adds xx s, zz s, xz s to the
// stresses of cell (i, j), s = the scaled sample of its source.
struct Waves {
  int n_terms;
  int16_t i[WAVE_TERMS], j[WAVE_TERMS];
  int32_t first[WAVE_TERMS];  // the source's first sample in s
  float xx[WAVE_TERMS], zz[WAVE_TERMS], xz[WAVE_TERMS];
  float s[WAVE_SAMPLES];
};

struct ShotForward {
  int nx, nz, R;
  int64_t C;
  float inv_h, dt;
  const float *bx, *bz, *l2m, *lam, *muxz, *taper;
  const int32_t* rec_map;
  float *vx, *vz, *sxx, *szz, *sxz;  // state between the launches of one shot
  float* rec;                        // [nt][nrec][2][C]
  float* store;                      // [C][planes][nz][nx] or null
  int64_t planes;                    // planes per chain
  int snap;                          // snapshot interval
  int nrec, n0, n1, load, save;
  uint64_t wait_ns;  // limit of a halo wait
  int withhold;      // test hook: one thread of block 0 sends no halos
  int* status;
};

struct ShotAdjoint {
  int nx, nz, R;
  int64_t C;
  float inv_h, dt, w;
  const float *bx, *bz, *l2m, *lam, *muxz, *taper;
  const int32_t* rec_map;
  const float* resid;  // [nt][nrec][2][C]
  const float* store;  // [C][planes][nz][nx]
  int64_t planes;
  int snap, nrec, nt;
  float *g_bx, *g_bz, *g_l2m, *g_lam, *g_muxz;  // [cells][C], accumulated
  uint64_t wait_ns;
  int withhold;
  int* status;
};

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Halo rows pushed between neighbouring blocks.  One barrier per kind of half
// step; the first thread arms it with the bytes both neighbours will send.
struct HaloBarriers {
  uint64_t bar[2];
};
__device__ __forceinline__ uint32_t smem_of(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t remote_of(uint32_t addr, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void halo_init(HaloBarriers& h) {
  for (int k = 0; k < 2; ++k)
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_of(&h.bar[k])) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void halo_arm(HaloBarriers& h, int k, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_of(&h.bar[k])), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void halo_push(uint32_t dst, float v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(dst),
               "r"(__float_as_uint(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ bool halo_try(const HaloBarriers& h, int k, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}"
      : "=r"(ok)
      : "r"(smem_of(&h.bar[k])), "r"(parity)
      : "memory");
  return ok != 0;
}
// Wait for the halos, at most limit_ns (2 s in production) or until another
// block has given up, which its neighbours' neighbours would otherwise notice
// one limit after the other; on expiry the
// status word is set, and from then on this thread neither waits, sends nor arms
// a barrier (whose phase never completed), so every block still reaches the end of
// its loop and the final cluster barrier.
__device__ __forceinline__ void halo_wait(const HaloBarriers& h, int k, uint32_t parity, uint64_t limit_ns, int* status,
                                          bool& dead) {
  if (dead || halo_try(h, k, parity)) return;
  uint64_t t0, t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  while (!halo_try(h, k, parity)) {
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    if (t - t0 > limit_ns || *(volatile int*)status != 0) {
      atomicExch(status, 1);
      dead = true;
      return;
    }
  }
}

// At the end of a launch: edge rows of a launch with a wait that ran out arrive
// before any block leaves.
__device__ __forceinline__ void halo_drain(bool dead, const int* status) {
  if (!halo_must_drain(dead, *(const volatile int*)status)) return;
  uint64_t t0, t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  do asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  while (t - t0 < HALO_DRAIN_NS);
}

// Rows of shared memory (one float per column) a block needs.
constexpr int forward_rows(int rz) { return 10 * rz + 12; }
// (strips above 11 rows fit only if t4 shares the rows of t1, which takes two
// more barriers of the block: 1.8 % of a single model's pass)
constexpr bool adjoint_shares(int rz) { return rz > 11; }
constexpr int adjoint_rows(int rz) { return adjoint_shares(rz) ? 14 * rz + 24 : 15 * rz + 25; }

// Strip heights compiled.
#define HMC_FORWARD_STRIPS(X) X(4) X(5) X(7) X(9) X(10) X(14)
#define HMC_ADJOINT_STRIPS(X) X(4) X(5) X(7) X(9) X(11) X(14)

struct Strip {
  int rows = 0;          // of a block; 0: no strip fits, the per-step kernels run
  double step_us = 0.0;  // expected time of a step
};
// Launch one shot.  dry: only tell the strip.  The pitch of a row
// in shared memory is a constant, so that offsets are immediates; a narrow grid
// takes a narrow one, which lets several blocks share an SM: 64 chains of 100 x
// 70 cells take 21.4 us per step of misfit and gradient with 256 columns and 15.0
// with 128 (compiled in fwi_cluster_128.cu, fwi_cluster_192.cu and
// fwi_cluster_256.cu).
template <int PITCH>
int cluster_forward_at(const ShotForward& a, const Waves& w, bool dry, Strip* strip, cudaStream_t st);
template <int PITCH>
int cluster_adjoint_at(const ShotAdjoint& a, bool dry, Strip* strip, cudaStream_t st);

// The strip height for C chains: the cheapest number of waves of resident
// clusters, a step of a wave costing its rows' instructions (those of all
// blocks of an SM) or, if that is more, one block's and two halo exchanges.
struct ClusterChoice {
  int rz = 0, R = 0;
  double cost = 0.0, step_us = 0.0;
};
template <typename Kernel>
void consider_strip(ClusterChoice& best, Kernel kern, int rz, int floats, int nx, int nz, int64_t C, double row_instr,
                    const StripModel& model) {
  const int R = (nz + rz - 1) / rz;
  const size_t smem = (size_t)floats * sizeof(float);
  if (R > CLUSTER_MAX || smem > 227 * 1024 - 64) return;
  const int threads = (nx + 31) / 32 * 32;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
      cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)R);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim = {(unsigned)R, 1, 1};
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  if (n < 1) return;
  const int64_t resident = C < n ? C : n;
  const double per_sm = resident * R > 152 ? (resident * R + 151) / 152 : 1;
  const double work = rz * row_instr * (threads / 32) / 4;
  const double step = work * per_sm > work + 900 ? work * per_sm : work + 900;
  const double cost = step * (double)((C + n - 1) / n);
  if (best.rz == 0 || cost < best.cost)
    best = ClusterChoice{rz, R, cost, strip_step_us(model, rz, R, n, threads / 32, C)};
}

template <typename Kernel, typename... A>
int launch_cluster(const char* who, Kernel kern, int floats, int nx, int R, int64_t C, cudaStream_t st, const A&... args) {
  HMC_REQUIRE(C * R <= 0x7FFFFFFF, "%s: too many chains", who);
  const size_t smem = (size_t)floats * sizeof(float);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(C * R));
  cfg.blockDim = dim3((unsigned)((nx + 31) / 32 * 32));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim = {(unsigned)R, 1, 1};
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, args...);
  if (e != cudaSuccess) return cuda_fail(e, who);
  return check_launch(who);
}

}  // namespace fwi
}  // namespace hmc
