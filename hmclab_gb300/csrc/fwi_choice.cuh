// What a time step of an elastic shot is expected to take on chip (fwi_cluster.cuh) and
// in the per-step kernels (fwi.cu): which of them run follows from these alone, so
// that it can be checked without a GPU.
//
// On chip, a step is a wave's instructions (rows times warps, shared by the blocks of an
// SM), a thread's own rows and the exchange of the edges, for each wave of resident
// clusters; narrow grids leave a block one or two warps, and then the latency of its
// rows is most of a step.  The per-step kernels are bound by their launches and by the
// bytes of cells x chains, 32 chains at a time.  Fitted to misfits and gradients of
// 1859 grids and batches (20 .. 256 x 20 .. 224 cells, 1 .. 500 chains), nine in ten of
// which they give within a sixth; the line they draw leaves 16 of 3718 passes more
// than 3 % slower than the per-step kernels, at most 15 %, where running every grid on chip that
// fits left 421, at most 4.5 times as slow.  Examples, us per gradient step: 240 x 140
// cells, 64 chains 62 on chip and 82 in the per-step kernels; 20 x 224 cells, 256
// chains 189 and 43; 160 x 178 cells, 64 chains 107 and 73; 20 x 224 cells, one chain
// 10 and 15.
#pragma once

#include <cstdint>

namespace hmc {
namespace fwi {

struct StripModel {
  double issue, row, wave;  // us per row and warp of a scheduler, row of a thread, wave
};
constexpr StripModel FORWARD_STEP = {0.0530, 0.0513, 0.923};
constexpr StripModel STORING_STEP = {0.0280, 0.0833, 1.234};  // the forward step that stores its velocities
constexpr StripModel ADJOINT_STEP = {0.1106, 0.4245, 0.4347};

// rz rows per block, R blocks per cluster, n clusters resident at a time.
inline double strip_step_us(const StripModel& m, int rz, int R, int n, int warps, int64_t C) {
  const int64_t waves = (C + n - 1) / n, last = C - (waves - 1) * n;
  const auto instructions = [&](int64_t clusters) {
    const double per_sm = (double)(clusters * R) / 152;
    return 0.25 * rz * warps * (per_sm > 1.0 ? per_sm : 1.0);
  };
  return m.issue * ((double)(waves - 1) * instructions(n) + instructions(last)) + (double)waves * (m.row * rz + m.wave);
}

inline double stencil_step_us(int64_t cells, int64_t C, bool staged, bool gradient) {
  const double n = (double)cells * (double)((C + 31) / 32 * 32);
  const auto beyond = [n](double fits) { return n > fits ? n - fits : 0.0; };  // what no longer fits L2
  if (gradient)
    return staged ? 30.5e-6 * n + 8.5e-6 * beyond(1.0e6) + 10.5 : 37.0e-6 * n + 18.0e-6 * beyond(1.2e6) + 9.3;
  return staged ? 8.3e-6 * n + 8.7e-6 * beyond(2.5e6) + 4.1 : 12.7e-6 * n + 13.5e-6 * beyond(2.2e6) + 3.9;
}

}  // namespace fwi
}  // namespace hmc
