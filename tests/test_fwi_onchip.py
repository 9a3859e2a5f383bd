"""Shots with the wavefield on chip (a cluster per chain) against the
direct-load kernels, which evaluate the same expressions: records, misfits and
gradients equal bit for bit, where strips, columns, snapshots, sources and
launches have their edges."""
import os
import subprocess

import numpy as np
import pytest

import hmclab_gb300 as H
from hmclab_gb300 import fwi as FW


def _pair(cfg, C, seed=0):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(seed)
    shape = (cfg.n_shots, cfg.nt, cfg.n_rec)
    ux, uz = 1e-3 * rng.normal(size=shape), 1e-3 * rng.normal(size=shape)
    out = []
    for staged in (True, False):
        d = H.Distributions.ElasticFullWaveform2D(cfg, ux, uz, data_std=1e-3, free_parameter_grid=[3, 2])
        d.staged_tiles = staged
        out.append(d)
    M = torch.from_numpy(rng.normal(size=(18, C)) * np.repeat([40.0, 20.0, 15.0], 6)[:, None]).float().cuda()
    return out, M.contiguous()


def _check(cfg, C, seed=0):
    (chip, direct), M = _pair(cfg, C, seed)
    for _ in range(2):  # a second evaluation replays the shots' graphs
        x, y = chip.misfit_batch(M).cpu().numpy(), direct.misfit_batch(M).cpu().numpy()
        g, h = chip.gradient_batch(M).cpu().numpy(), direct.gradient_batch(M).cpu().numpy()
        chip.check_device_status()
        assert np.all(np.isfinite(x)) and np.all(x > 0) and np.abs(h).max() > 0
        assert np.array_equal(x, y)
        assert np.array_equal(g, h)


def _config(nx, nz, nt=60, pad=8, **kw):
    kw.setdefault("src_x", (0.4 * nx * 5.0,))
    kw.setdefault("rec_x", np.linspace(12.0, nx * 5.0 - 12.0, 7))
    return FW.ElasticConfig(nx=nx, nz=nz, pad=pad, h=5.0, dt=5e-4, nt=nt, f0=25.0, sponge=0.05, src_z=12.0, rec_z=17.0, **kw)


@pytest.mark.gpu
@pytest.mark.parametrize("nx,nz", [(15, 12), (16, 21), (47, 39), (48, 40), (49, 41), (84, 64), (112, 65), (124, 66), (61, 96),
                                   (240, 97), (239, 138), (100, 208), (113, 50), (176, 45), (177, 30)])
@pytest.mark.parametrize("C", [1, 3])
def test_strips_and_columns(nx, nz, C):
    _check(_config(nx, nz), C)


@pytest.mark.gpu
def test_batches_of_several_waves():
    _check(_config(60, 44, nt=40), 64)
    _check(_config(200, 100, nt=12, pad=20), 33)


@pytest.mark.gpu
@pytest.mark.parametrize("k,nt", [(2, 41), (3, 60), (5, 52), (7, 50)])
def test_snapshots(k, nt):
    _check(_config(50, 40, nt=nt, snapshot_interval=k), 2)


@pytest.mark.gpu
def test_sources_and_several_launches():
    P = FW.PointSource
    shots = [[P(20, 15), P(31, 18, *FW.moment_tensor(30.0), delay=0.004), P(30, 18, *FW.moment_tensor(75.0))],
             [P(25, 9, *FW.moment_tensor(110.0))]]
    _check(_config(44, 36, nt=90, shots=shots), 2)
    # more samples than a launch carries: the state passes through memory
    many = [[P(12 + k, 14, delay=0.001 * k) for k in range(8)]]
    _check(_config(30, 24, nt=1600, shots=many), 1)


@pytest.mark.gpu
def test_grids_that_do_not_fit_keep_the_stencil_kernels():
    _check(_config(256, 40, nt=20), 32)  # 272 columns
    _check(_config(40, 230, nt=20), 2)  # 246 rows


@pytest.mark.gpu
def test_repeated_gradients_are_equal():
    """Blocks and warps drift against each other differently from run to run; what
    they hand over in shared memory must not depend on it."""
    cfg = _config(112, 60)
    (chip, direct), M = _pair(cfg, 64)
    g = direct.gradient_batch(M)
    for _ in range(40):
        assert bool((chip.gradient_batch(M) == g).all())
    chip.check_device_status()


@pytest.mark.gpu
@pytest.mark.parametrize("C", [1, 5])
def test_a_wait_that_runs_out_is_reported_and_the_context_survives(C):
    """Under the wait-limit hook one thread of the first block sends no halos, so
    its neighbours' waits run out after 1 ms; every block still ends."""
    from hmclab_gb300 import _lib
    from hmclab_gb300.Helpers.CustomExceptions import DeviceTimeoutError

    cfg = _config(60, 50)
    (chip, direct), M = _pair(cfg, C)
    x, g = direct.misfit_batch(M), direct.gradient_batch(M)
    for call in ("misfit_batch", "gradient_batch"):
        hooked = H.Distributions.ElasticFullWaveform2D(chip)  # a copy captures its shots' graphs under the hook
        with _lib.wait_limits(1_000_000, withhold=True):
            getattr(hooked, call)(M)
            x.cpu()
        with pytest.raises(DeviceTimeoutError):
            hooked.check_device_status()
        del hooked
    assert bool((chip.misfit_batch(M) == x).all()) and bool((chip.gradient_batch(M) == g).all())
    chip.check_device_status()


_QUOTIENT = r"""
#include "quotient.cuh"
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
int main() {
  std::mt19937_64 gen(3);
  long wrong = 0, taken = 0;
  for (long k = 0; k < 4000000; ++k) {
    const uint64_t u = gen();
    uint32_t ia = (uint32_t)u, ib = (uint32_t)(u >> 32);
    ib = (ib & 0x807fffffu) | ((96u + (ib >> 23) % 32) << 23);         // 2^-31 .. 2
    if (k % 3 == 0) ia &= 0x83ffffffu;                                 // tiny dividends
    if (k % 11 == 0) ia &= 0x80ffffffu;                                // subnormal ones
    if (k % 5 == 0) ib &= 0xfffff000u;                                 // few bits: ties, exact quotients
    if (k % 7 == 0) ib |= 0x7ffff0u;                                   // nearly all ones
    if (k % 13 == 0) ib &= 0xff800000u;                                // powers of two
    float a, b;
    memcpy(&a, &ia, 4);
    memcpy(&b, &ib, 4);
    bool plain = hmc::plain_divisor(b);
    if (!plain) continue;
    const float q = hmc::quotient(a, b, 1.f / b, plain);
    if (!plain) continue;
    volatile float t = a / b;
    ++taken;
    wrong += !(q == t);
  }
  printf("%ld %ld\n", taken, wrong);
}
"""


def test_quotient_is_correctly_rounded(tmp_path):
    src, exe = tmp_path / "q.cpp", tmp_path / "q"
    src.write_text(_QUOTIENT)
    csrc = os.path.join(os.path.dirname(H.__file__), "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", csrc, str(src), "-o", str(exe)], check=True)
    taken, wrong = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert taken > 3000000 and wrong == 0
