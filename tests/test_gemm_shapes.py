"""The rules that choose a product's kernel and blocks (csrc/gemm_shape.cuh),
compiled for the host, and products at the sizes where they change."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import hmclab_gb300 as H
from hmclab_gb300 import _lib

_SOURCE = r"""
#include "gemm_shape.cuh"
extern "C" {
int rows_per_thread(int64_t m, int64_t n, int64_t k) { return hmc::f32_rows_per_thread(m, n, k); }
int by_rows(int64_t m, int64_t n, int64_t k) { return hmc::f64_by_rows(m, n, k); }
int few_columns_fit(int64_t k) { return hmc::f32_offsets_fit(hmc::F32_FEW_ROWS, k); }
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("gemm_shape")
    (d / "r.cpp").write_text(_SOURCE)
    csrc = os.path.join(os.path.dirname(H.__file__), "csrc")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", csrc, str(d / "r.cpp"), "-o", str(d / "r.so")],
                   check=True)
    lib = ctypes.CDLL(str(d / "r.so"))
    for f, args in ((lib.rows_per_thread, 3), (lib.by_rows, 3), (lib.few_columns_fit, 1)):
        f.argtypes = [ctypes.c_int64] * args
    return lib


def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def test_offsets_of_a_block_stay_within_32_bits(rules):
    """A block's offsets reach its rows times k; rows too long for that go to
    the kernel with 64-bit offsets (0)."""
    for k in (1, 600, 29_800_000, 29_826_162, 30_200_000, 33_600_000, 40_000_000, 134_000_000, 135_000_000, 2**33):
        for m in (1, 33, 129, 144, 1000):
            for n in (5, 64, 8192):
                r = rules.rows_per_thread(m, n, k)
                assert r in (0, 2, 4, 6, 8, 9) and 16 * r * k < 2**32, (m, n, k, r)
                assert r > 0 or 32 * k >= 2**32 - 32
        assert rules.few_columns_fit(k) == (64 * k < 2**32 - 64)


TALL = 65535 * 64  # rows a product may have


def test_tall_matrices_fit_the_grid(rules):
    for m in (1, 2_097_120, 2_097_121, 2_097_153, 2_131_600, 3_000_000, 3_000_001, 4_194_177, TALL):
        for n in (5, 64, 8192):
            r = rules.rows_per_thread(m, n, 8)
            assert r > 0 and -(-m // (16 * r)) <= 65535, (m, n, r)


def test_two_rows_per_thread_where_blocks_are_missing(rules):
    """Padding alone took two rows per thread for each of these; where the chip is
    full that was slower than the tiles the kernel replaced."""
    for m, n, want in ((20_000, 1024, 4), (100_000, 1024, 4), (4000, 8192, 4), (2080, 8192, 9), (2080, 200, 2), (200, 8192, 2),
                       (20_000, 8, 9), (33, 64, 4), (129, 8192, 9), (160, 64, 2)):
        r = rules.rows_per_thread(m, n, 60)
        assert (r == 2) == (want == 2), (m, n, r)


def test_fp64_rows_only_where_the_tiles_are_slower(rules):
    """(m, n, k) on either side of the line, by the kernel that was faster."""
    for m, n, k in ((50, 64, 50), (1000, 1, 1000), (1000, 64, 1000), (9000, 8, 60), (9000, 32, 1000), (4000, 64, 4000),
                    (9664, 4, 16), (7500, 56, 1600), (6000, 32, 200)):
        assert rules.by_rows(m, n, k), (m, n, k)
    for m, n, k in ((9000, 48, 1000), (9000, 64, 1000), (9000, 32, 60), (9000, 64, 200), (7500, 64, 16), (6000, 64, 4000),
                    (9665, 1, 1000), (50, 65, 50)):
        assert not rules.by_rows(m, n, k), (m, n, k)


def test_tall_matrices_are_not_refused():
    """Without a device the launch fails, but no size is refused before it."""
    lib, one = _lib.load(), ctypes.c_void_p(16)
    torch = pytest.importorskip("torch")
    if torch.cuda.is_available():
        pytest.skip("a device would run the products on these addresses")
    for n in (1, 4, 5, 64):
        for m in (2_097_153, 3_000_001, TALL):
            assert lib.hmc_gemm(_lib.HMC_F32, m, n, 1, 1.0, one, one, None, one, 0, None) != _lib.HMC_ERR_INVALID_ARG
        assert lib.hmc_gemm(_lib.HMC_F32, TALL + 1, n, 1, 1.0, one, one, None, one, 0, None) == _lib.HMC_ERR_INVALID_ARG


@pytest.mark.gpu
@pytest.mark.parametrize("m,n", [(2_097_153, 5), (3_000_001, 64), (TALL, 8), (TALL, 3)])
def test_tall_matrices(m, n):
    torch = _cuda()
    k = 3
    A = torch.from_numpy(np.random.default_rng(n).integers(-9, 9, size=(m, k)).astype(np.float32)).cuda()
    B = torch.from_numpy(np.random.default_rng(k).integers(-9, 9, size=(k, n)).astype(np.float32)).cuda()
    out = torch.full((m, n), float("nan"), device="cuda")
    _lib.call("hmc_gemm", _lib.HMC_F32, m, n, k, 1.0, A.data_ptr(), B.data_ptr(), None, out.data_ptr(), 0,
              torch.cuda.current_stream().cuda_stream)
    want = sum(A[:, j:j + 1] * B[j:j + 1] for j in range(k))  # whole numbers: exact
    assert torch.equal(out, want)


@pytest.mark.gpu
@pytest.mark.parametrize("m", [97, 127, 128])
@pytest.mark.parametrize("n,offset", [(5, 0), (32, 0), (36, 0), (32, 1)])
def test_eight_rows_per_thread(rules, m, n, offset):
    torch = _cuda()
    k = 33
    assert rules.rows_per_thread(m, n, k) == 8
    rng = np.random.default_rng(m + n)
    A, B, bias = (rng.normal(size=s).astype(np.float32) for s in ((m, k), (k, n), (m,)))

    def put(a):  # offset: four bytes past a 16-byte boundary
        t = torch.zeros(a.size + offset, device="cuda")
        t[offset:] = torch.from_numpy(a.ravel()).cuda()
        return t[offset:]

    tA, tB, tb = put(A), put(B), put(bias)
    out = torch.full((m, n), float("nan"), device="cuda")
    _lib.call("hmc_gemm", _lib.HMC_F32, m, n, k, 1.5, tA.data_ptr(), tB.data_ptr(), tb.data_ptr(), out.data_ptr(), 0,
              torch.cuda.current_stream().cuda_stream)
    A, B, bias = (a.astype(np.float64) for a in (A, B, bias))
    bound = 2.0**-24 * (k + 4) * (1.5 * np.abs(A) @ np.abs(B) + np.abs(bias)[:, None])
    assert np.all(np.abs(out.cpu().numpy() - (1.5 * A @ B + bias[:, None])) <= bound)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(144, 8, 30_200_000), (64, 2, 68_000_000), (31, 8, 139_000_000)])
def test_long_rows(m, n, k):
    """Rows whose offsets pass 2^32 (17 GB): one entry per row, so every product is
    exact and an entry read from elsewhere shows."""
    torch = _cuda()
    A = torch.zeros((m, k), device="cuda")
    B = torch.zeros((k, n), device="cuda")
    rng = np.random.default_rng(k)
    at = np.sort(rng.choice(k, size=m, replace=False))
    A[torch.arange(m), torch.from_numpy(at)] = torch.arange(1.0, m + 1, device="cuda")
    b = rng.integers(1, 100, size=(m, n)).astype(np.float32)
    B[torch.from_numpy(at).cuda()] = torch.from_numpy(b).cuda()
    out, work = torch.empty((m, n), device="cuda"), torch.empty(256 * m * n, device="cuda")
    _lib.call("hmc_gemm_splitk", _lib.HMC_F32, m, n, k, 1.0, A.data_ptr(), B.data_ptr(), out.data_ptr(), 0, work.data_ptr(),
              work.numel(), torch.cuda.current_stream().cuda_stream)
    assert np.array_equal(out.cpu().numpy(), np.arange(1.0, m + 1)[:, None] * b)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(9000, 32, 60), (7500, 64, 16), (9000, 48, 1000), (6000, 56, 200)])
def test_fp64_product_on_either_side_of_the_line(m, n, k):
    torch = _cuda()
    rng = np.random.default_rng(m + n + k)
    A, B, bias = rng.normal(size=(m, k)), rng.normal(size=(k, n)), rng.normal(size=m)
    tA, tB, tb = (torch.from_numpy(a).cuda() for a in (A, B, bias))
    out = torch.full((m, n), float("nan"), dtype=torch.float64, device="cuda")
    _lib.call("hmc_gemm", _lib.HMC_F64, m, n, k, 1.5, tA.data_ptr(), tB.data_ptr(), tb.data_ptr(), out.data_ptr(), 0,
              torch.cuda.current_stream().cuda_stream)
    # k products and a sum of them: k ulp of the sum of their sizes
    bound = 2.3e-16 * (k + 4) * (1.5 * np.abs(A) @ np.abs(B) + np.abs(bias)[:, None])
    assert np.all(np.abs(out.cpu().numpy() - (1.5 * A @ B + bias[:, None])) <= bound)
