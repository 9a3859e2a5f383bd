"""The FP32 product at the edges of its blocks (row groups, 16-deep chunks,
32 columns or 4), with unaligned operands, and split over k."""
import numpy as np
import pytest


def _data(m, n, k):
    rng = np.random.default_rng(m * 1000 + n * 10 + k)
    return [rng.normal(size=s).astype(np.float32) for s in ((m, k), (k, n), (m,), (m, n))]


SIZES = [(1, 1, 1), (3, 4, 16), (33, 1, 17), (65, 3, 40), (129, 5, 129), (160, 32, 31), (161, 33, 32), (129, 100, 129), (8, 64, 257),
         (9, 36, 15), (321, 31, 48), (1000, 8, 5), (2000, 2, 64)]


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", SIZES)
@pytest.mark.parametrize("accumulate,offset", [(0, 0), (1, 1)])
def test_product(m, n, k, accumulate, offset):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hmclab_gb300 import _lib

    A, B, bias, out = _data(m, n, k)

    def put(a):  # offset: four bytes past a 16-byte boundary
        t = torch.zeros(a.size + offset, device="cuda")
        t[offset:] = torch.from_numpy(a.ravel()).cuda()
        return t[offset:]

    tA, tB, tb, to = put(A), put(B), put(bias), put(out)
    _lib.call("hmc_gemm", _lib.HMC_F32, m, n, k, 1.5, tA.data_ptr(), tB.data_ptr(), tb.data_ptr(), to.data_ptr(),
              accumulate, torch.cuda.current_stream().cuda_stream)
    A, B, bias, out = (a.astype(np.float64) for a in (A, B, bias, out))
    want = 1.5 * A @ B + bias[:, None] + (out if accumulate else 0.0)
    bound = 2.0**-24 * (k + 4) * (1.5 * np.abs(A) @ np.abs(B) + np.abs(bias)[:, None] + np.abs(out))
    assert np.all(np.abs(to.cpu().numpy().reshape(m, n) - want) <= bound)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(60, 1, 3000), (200, 64, 2500), (33, 5, 511), (7, 40, 4000)])
def test_split_product(m, n, k):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hmclab_gb300 import _lib

    A, B, _, out = _data(m, n, k)
    tA, tB, to = (torch.from_numpy(a).cuda().contiguous() for a in (A, B, out))
    work = torch.empty(8 * m * n, device="cuda")
    _lib.call("hmc_gemm_splitk", _lib.HMC_F32, m, n, k, 0.5, tA.data_ptr(), tB.data_ptr(), to.data_ptr(), 1, work.data_ptr(),
              work.numel(), torch.cuda.current_stream().cuda_stream)
    A, B, out = (a.astype(np.float64) for a in (A, B, out))
    bound = 2.0**-24 * (k + 12) * (0.5 * np.abs(A) @ np.abs(B) + np.abs(out))
    assert np.all(np.abs(to.cpu().numpy() - (0.5 * A @ B + out)) <= bound)
