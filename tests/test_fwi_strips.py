"""Which kernels an elastic shot runs (hmc_fwi_strips), asked by the tests that
compare the on-chip shots with the per-step kernels: without it a comparison in
which nothing ran on chip would pass.  Every compiled strip height and row pitch is
compared, and the row-sharing adjoint of the tallest strips is repeated."""
import ctypes

import pytest

import test_fwi_onchip as OC
from hmclab_gb300 import _lib


def strips(dist, C, store=True):
    """(forward, adjoint) strip heights of a target's shots, 0 off chip."""
    ws = dist._workspace(C, "cuda", True)
    f, a = ctypes.c_int(-1), ctypes.c_int(-1)
    _lib.call("hmc_fwi_strips", ctypes.byref(dist._descriptor(ws, C)), int(store), ctypes.byref(f), ctypes.byref(a))
    return f.value, a.value


def _grid(nxc, nzc, **kw):
    return OC._config(nxc - 16, nzc - 16, **kw)


def test_null_arguments_are_refused():
    f = ctypes.c_int()
    assert _lib.load().hmc_fwi_strips(None, 1, ctypes.byref(f), ctypes.byref(f)) == _lib.HMC_ERR_INVALID_ARG


# one model: the lowest strips of which sixteen cover the grid
@pytest.mark.gpu
@pytest.mark.parametrize("nxc", [66, 128, 150, 192, 213, 256])
@pytest.mark.parametrize("nzc,heights", [(61, (4, 4)), (66, (5, 5)), (112, (7, 7)), (113, (9, 9)), (148, (10, 11)), (177, (14, 14)),
                                         (224, (14, 14))])
def test_every_strip_height_and_pitch(nxc, nzc, heights):
    cfg = _grid(nxc, nzc, nt=30)
    assert (cfg.nxc, cfg.nzc) == (nxc, nzc)
    (chip, direct), _ = OC._pair(cfg, 1)
    assert strips(chip, 1) == heights and strips(direct, 1) == (0, 0)
    OC._check(cfg, 1)


def _parameters(test):
    return {m.args[0]: m.args[1] for m in test.pytestmark if m.name == "parametrize"}


@pytest.mark.gpu
def test_the_compared_shots_run_on_chip():
    p = _parameters(OC.test_strips_and_columns)
    for nx, nz in p["nx,nz"]:
        for C in p["C"]:
            (chip, direct), _ = OC._pair(OC._config(nx, nz, nt=4), C)
            assert min(strips(chip, C)) > 0 and strips(direct, C) == (0, 0), (nx, nz, C)
    for k, nt in _parameters(OC.test_snapshots)["k,nt"]:
        assert min(strips(OC._pair(OC._config(50, 40, nt=nt, snapshot_interval=k), 2)[0][0], 2)) > 0
    for nx, nz, pad, C in ((60, 44, 8, 64), (200, 100, 20, 33), (44, 36, 8, 2), (30, 24, 8, 1), (112, 60, 8, 64), (60, 50, 8, 5)):
        assert min(strips(OC._pair(OC._config(nx, nz, nt=4, pad=pad), C)[0][0], C)) > 0, (nx, nz, C)
    for nx, nz, C in ((256, 40, 32), (40, 230, 2)):
        assert strips(OC._pair(OC._config(nx, nz, nt=4), C)[0][0], C) == (0, 0), (nx, nz, C)


@pytest.mark.gpu
@pytest.mark.parametrize("nxc,nzc", [(240, 140), (128, 182)])
def test_repeated_gradients_where_two_operands_share_rows(nxc, nzc):
    """Strips of 14 rows let t4 take the rows of t1 between two barriers of the block."""
    C = 64
    cfg = _grid(nxc, nzc, nt=50)
    (chip, direct), M = OC._pair(cfg, C)
    assert strips(chip, C)[1] == 14
    g = direct.gradient_batch(M)
    for _ in range(40):
        assert bool((chip.gradient_batch(M) == g).all())
    chip.check_device_status()
