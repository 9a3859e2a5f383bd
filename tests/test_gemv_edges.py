"""The row kernel of FP64 products with few columns, at the edges of its warps
and column groups and where it hands over to the tile kernel."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (3, 1, 33), (130, 1, 1000), (5, 2, 7), (64, 4, 64), (67, 5, 100),
                                   (9, 8, 31), (200, 9, 257), (65, 64, 40), (65, 65, 40), (9800, 3, 17)])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_fp64_product_of_few_columns(m, n, k, accumulate):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hmclab_gb300 import _lib

    rng = np.random.default_rng(m * 1000 + n)
    A, B, bias, out = rng.normal(size=(m, k)), rng.normal(size=(k, n)), rng.normal(size=m), rng.normal(size=(m, n))
    tA, tB, tb, to = (torch.from_numpy(a).cuda().contiguous() for a in (A, B, bias, out))
    _lib.call("hmc_gemm", _lib.HMC_F64, m, n, k, 1.5, tA.data_ptr(), tB.data_ptr(), tb.data_ptr(), to.data_ptr(),
              accumulate, torch.cuda.current_stream().cuda_stream)
    want = 1.5 * A @ B + bias[:, None] + (out if accumulate else 0.0)
    # k products and a sum of them: k ulp of the sum of their sizes
    bound = 2.3e-16 * (k + 4) * (1.5 * np.abs(A) @ np.abs(B) + np.abs(bias)[:, None] + np.abs(out))
    assert np.all(np.abs(to.cpu().numpy() - want) <= bound)
