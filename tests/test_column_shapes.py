"""The layouts of the per-chain sums (csrc/column_shape.cuh): the rule compiled for the
host, and sums and chains on the GPU where it changes."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import hmclab_gb300 as H

D = H.Distributions

_SOURCE = r"""
#include "column_shape.cuh"
extern "C" int element(int64_t d, int64_t C, int bytes, int aligned, int most) {
  const hmc::ElementShape s = hmc::element_shape(d, C, bytes, aligned != 0, most);
  return s.vec ? 100 + s.rows : s.rows;
}
extern "C" void shape(int64_t C, int64_t rows, int64_t narrow, int* out) {
  const hmc::ColumnShape s = narrow > 0 ? hmc::column_shape(C, rows, narrow) : hmc::column_shape(C, rows);
  out[0] = 1 << s.log_x;
  out[1] = s.cluster;
  out[2] = s.threads;
}
"""


@pytest.fixture(scope="module")
def shape(tmp_path_factory):
    d = tmp_path_factory.mktemp("column_shape")
    (d / "s.cpp").write_text(_SOURCE)
    csrc = os.path.join(os.path.dirname(H.__file__), "csrc")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", csrc, str(d / "s.cpp"), "-o", str(d / "s.so")],
                   check=True)
    lib = ctypes.CDLL(str(d / "s.so"))

    def call(C, rows, narrow=0):
        out = (ctypes.c_int * 3)()
        lib.shape(ctypes.c_int64(C), ctypes.c_int64(rows), ctypes.c_int64(narrow), out)
        return tuple(out)

    call.element = lambda d, C, nbytes, aligned, most: lib.element(ctypes.c_int64(d), ctypes.c_int64(C), nbytes, aligned, most)
    return call


def test_every_layout_is_one_a_kernel_can_run(shape):
    for C in (1, 2, 3, 5, 17, 31, 32, 33, 1000, 9728, 9729, 100_000, 10**7):
        for rows in (1, 4, 9, 63, 64, 65, 129, 256, 257, 321, 600, 4096, 10**6):
            for narrow in (0, 320):
                x, cluster, threads = shape(C, rows, narrow)
                assert x == min(32, 1 << (C - 1).bit_length()) and cluster in (1, 2, 4, 8) and threads in (128, 256, 512)


def test_few_rows_take_few_threads(shape):
    """Blocks of 512 threads and clusters were up to 2.5 times as slow as one 8-warp block per 32 chains here."""
    for C in (1, 8, 31, 100, 4096, 20_000, 100_000, 10**6):
        assert shape(C, 1)[1:] == shape(C, 4)[1:] == (1, 128)
    for C in (20_000, 100_000, 10**6):
        assert shape(C, 40)[1:] == (1, 128) and shape(C, 129)[1:] == (1, 256) and shape(C, 600)[1:] == (1, 512)
        assert shape(C, 300, 320)[1:] == (1, 128) and shape(C, 600, 320)[1:] == (1, 512)
    for C in (1, 4, 16):
        assert shape(C, 40)[1] == 1 and shape(C, 63)[1] == 1
    # layouts that the sums of many rows were measured with
    assert shape(1, 1000) == (1, 8, 512) and shape(1024, 4096) == (32, 8, 512) and shape(4096, 1000) == (32, 2, 512)
    assert shape(8192, 129) == (32, 1, 512)


def test_elements_take_few_threads_only_on_a_full_chip(shape):
    """Two to four rows and 16 bytes per thread made small FP64 updates up to 1.8 times as slow."""
    for d, C in ((40, 512), (4096, 4), (16, 1024), (1, 1), (9, 4096)):
        assert shape.element(d, C, 8, 1, 2) == shape.element(d, C, 8, 1, 4) == shape.element(d, C, 4, 1, 4) == 1
    assert shape.element(1500, 20_000, 8, 1, 4) == 102 and shape.element(600, 1024, 4, 1, 2) == 102
    assert shape.element(4096, 1024, 4, 1, 2) == 102 and shape.element(4096, 1024, 4, 1, 4) == 104
    assert shape.element(4096, 1024, 4, 0, 4) == 4 and shape.element(4096, 1023, 4, 1, 2) == 2  # no 16-byte rows


@pytest.mark.gpu
@pytest.mark.parametrize("d,C", [(125, 512), (124, 516), (250, 256), (1000, 2000), (1001, 2000), (80, 501), (80, 499), (1, 64_000),
                                 (40, 2048), (300, 1027)])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("kind", ["normal", "laplace"])
def test_prior_gradients(d, C, dtype, kind):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(d + C)
    mean, w = rng.normal(size=(d, 1)).astype(dtype), rng.uniform(0.5, 2.0, size=(d, 1)).astype(dtype)
    q = rng.normal(size=(d, C)).astype(dtype)
    make = D.Normal if kind == "normal" else D.Laplace
    iw = (1.0 / w.astype(float)).astype(dtype)
    want = -(iw * (mean - q)) if kind == "normal" else np.sign(q - mean) * iw
    post, M = make(mean.astype(float), w.astype(float)), torch.from_numpy(q).cuda()
    assert np.array_equal(post.gradient_batch(M).cpu().numpy(), want)
    twice = post.gradient_batch(M, out=torch.from_numpy(want.copy()).cuda(), accumulate=True)
    assert np.array_equal(twice.cpu().numpy(), want + want)


@pytest.mark.gpu
@pytest.mark.parametrize("d,C", [(1, 9728), (1, 9729), (4, 20_001), (40, 2), (63, 31), (64, 31), (65, 9760), (256, 9740), (257, 9731),
                                 (320, 9729), (321, 9729), (9, 4096), (17, 4096)])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_prior_sums(d, C, dtype):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(d + C)
    mean, w = rng.normal(size=(d, 1)).astype(dtype), rng.uniform(0.5, 2.0, size=(d, 1)).astype(dtype)
    q = rng.normal(size=(d, C)).astype(dtype)
    iw = (1.0 / w.astype(float)).astype(dtype)
    r = mean - q
    x = 0.5 * (r.astype(float) * (iw * r).astype(float)).sum(0)
    got = D.Normal(mean.astype(float), w.astype(float)).misfit_batch(torch.from_numpy(q).cuda())
    # FP64 sums of d terms that the reference above forms with the same roundings
    np.testing.assert_allclose(got.cpu().numpy(), x, rtol=2.3e-16 * (d + 4))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("d", [2, 40, 70, 260])
def test_the_first_chains_of_a_large_batch(d, dtype):
    """Momenta, accept test and recorded draws of a batch with more tiles than fill the
    chip: its first chains are those of a batch of their own."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(d)
    lower, upper = -1.2 * np.ones((d, 1)), 1.5 * np.ones((d, 1))
    post = D.Normal(rng.normal(size=(d, 1)), rng.uniform(0.2, 2.0, size=(d, 1)), lower_bounds=lower, upper_bounds=upper)
    q0 = rng.uniform(-1, 1, size=(d, 9750))
    m = H.MassMatrices.Diagonal(rng.uniform(0.5, 2, size=(d, 1)))
    runs = [H.Samplers.HMC(seed=4).sample(None, post, stepsize=0.15, amount_of_steps=4, initial_model=q0[:, :C], proposals=5,
                                          chains=C, dtype=dtype, mass_matrix=m, persistent=False,
                                          keep_samples=True).samples_numpy() for C in (9750, 70, 5)]
    for got in runs[1:]:
        n = got.shape[0]
        assert np.array_equal(got[:, :d], runs[0][:n, :d])
        np.testing.assert_allclose(got[:, d], runs[0][:n, d], rtol=1e-11)
