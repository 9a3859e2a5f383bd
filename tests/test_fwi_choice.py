"""Where elastic shots run (csrc/fwi_choice.cuh): the expected step times against
measured ones, on the host, and equal results on either side of the line, on the GPU."""
import ctypes
import os
import subprocess

import pytest

import hmclab_gb300 as H
import test_fwi_onchip as OC
from test_fwi_strips import strips

_SOURCE = r"""
#include "fwi_choice.cuh"
using namespace hmc::fwi;
extern "C" double chip(int kind, int rz, int R, int n, int warps, int64_t C) {
  return strip_step_us(kind == 0 ? FORWARD_STEP : kind == 1 ? STORING_STEP : ADJOINT_STEP, rz, R, n, warps, C);
}
extern "C" double stencils(int64_t cells, int64_t C, int staged, int gradient) {
  return stencil_step_us(cells, C, staged != 0, gradient != 0);
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("fwi_choice")
    (d / "c.cpp").write_text(_SOURCE)
    csrc = os.path.join(os.path.dirname(H.__file__), "csrc")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", csrc, str(d / "c.cpp"), "-o", str(d / "c.so")],
                   check=True)
    lib = ctypes.CDLL(str(d / "c.so"))
    lib.chip.restype = lib.stencils.restype = ctypes.c_double
    lib.chip.argtypes = [ctypes.c_int] * 5 + [ctypes.c_int64]
    lib.stencils.argtypes = [ctypes.c_int64, ctypes.c_int64, ctypes.c_int, ctypes.c_int]
    return lib


# grid, chains, strips (rows, blocks, resident clusters, warps) of the forward pass and the
# adjoint, us of a gradient's step on chip and in the per-step kernels
MEASURED = [(240 * 140, 64, (9, 16, 14, 8), (14, 10, 13, 8), 62.0, 82.0), (240 * 140, 1, (9, 16, 14, 8), (9, 16, 7, 8), 7.5, 45.0),
            (20 * 224, 256, (14, 16, 14, 1), (14, 16, 14, 1), 189.0, 43.0), (20 * 224, 1, (14, 16, 14, 1), (14, 16, 14, 1), 10.0, 15.5),
            (160 * 178, 64, (14, 13, 7, 5), (14, 13, 7, 5), 107.0, 73.0), (192 * 112, 12, (7, 16, 14, 6), (7, 16, 14, 6), 12.0, 35.0)]


@pytest.mark.parametrize("cells,C,f,a,on_chip,per_step", MEASURED)
def test_expected_times_pick_the_faster_kernels(rule, cells, C, f, a, on_chip, per_step):
    chip = rule.chip(1, *f, C) + rule.chip(2, *a, C)
    stencils = rule.stencils(cells, C, C % 32 == 0, 1)
    assert (chip < stencils) == (on_chip < per_step)


@pytest.mark.gpu
@pytest.mark.parametrize("nxc,nzc,C,chip", [(20, 113, 256, False), (20, 113, 1, True), (33, 177, 64, False), (33, 177, 4, True),
                                            (160, 178, 64, False), (160, 178, 3, True), (240, 140, 33, True)])
def test_either_side_gives_the_same(nxc, nzc, C, chip):
    x = 0.4 * (nxc - 16) * 5.0
    cfg = OC._config(nxc - 16, nzc - 16, nt=30, src_x=(x,), rec_x=[x - 5.0, x + 5.0])
    (dist, _), _ = OC._pair(cfg, C)
    assert (strips(dist, C)[1] > 0) == chip
    OC._check(cfg, C)
