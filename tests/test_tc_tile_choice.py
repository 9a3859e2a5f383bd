"""The choice of a contraction's tiles (csrc/tc_tiles.cuh) on the host, and results that
do not depend on it on the GPU."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import hmclab_gb300 as H

_SOURCE = r"""
#include "tc_tiles.cuh"
extern "C" int narrow(int64_t C, int64_t rows, int64_t K, int products) { return hmc::tc::narrow_tiles(C, rows, K, products); }
"""


@pytest.fixture(scope="module")
def narrow(tmp_path_factory):
    d = tmp_path_factory.mktemp("tc_tiles")
    (d / "n.cpp").write_text(_SOURCE)
    csrc = os.path.join(os.path.dirname(H.__file__), "csrc")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", csrc, str(d / "n.cpp"), "-o", str(d / "n.so")],
                   check=True)
    f = ctypes.CDLL(str(d / "n.so")).narrow
    f.argtypes = [ctypes.c_int64] * 3 + [ctypes.c_int]
    return f


def test_long_products_take_narrow_tiles_only_in_one_wave(narrow):
    """Two waves of narrow tiles were up to 1.45 times as slow as one of wide ones."""
    for C, rows in ((512, 2000), (1024, 1000), (4096, 140), (256, 4000)):
        assert not narrow(C, rows, 2000, 3) and not narrow(C, rows, 4000, 1)
        assert narrow(C, rows, 600, 3) and narrow(C, rows, 1000, 1)
    for C, rows in ((64, 140), (128, 4000), (256, 1500), (1024, 513)):  # an SM for each narrow tile
        assert narrow(C, rows, 4000, 3) and narrow(C, rows, 4000, 1)
    assert not narrow(4096, 800, 64, 3)


@pytest.mark.gpu
@pytest.mark.parametrize("C,d", [(512, 2000), (1024, 1000)])
def test_the_first_chains_do_not_depend_on_the_tiles(narrow, C, d):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    assert narrow(128, d, d, 3) and not narrow(C, d, d, 3)
    rng = np.random.default_rng(d)
    G = rng.normal(size=(d + 10, d)) / np.sqrt(d)
    lik = H.Distributions.LinearMatrix(G, G @ rng.normal(size=(d, 1)), 0.1)
    M = torch.from_numpy(rng.normal(size=(d, C))).float().cuda().contiguous()
    all_, first = lik.gradient_batch(M), lik.gradient_batch(M[:, :128].contiguous())
    lik.check_device_status()
    assert torch.equal(all_[:, :128], first)
