"""Ranks and ESS where their kernels change shape: draws around one sort tile
(8192), ties, signed zeros, infinities and NaN; half-chains around the staged
windows (384, 1024 draws) and lag windows around the rounds (16, 48, ...)."""
import numpy as np
import pytest

from oracle import hmc_oracle as O
from test_ess import ar1


def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.gpu
@pytest.mark.parametrize("N,d,C", [(1, 3, 1), (7, 2, 5), (64, 3, 4), (257, 2, 1), (8192, 1, 1), (8193, 2, 1), (97, 2, 190)])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_ranks_equal_sorted_positions(N, d, C, dtype):
    """Scores of the pooled ranks, ties averaged: the counts are whole
    numbers, so the scores agree with the oracle's to the rounding of the
    inverse normal distribution (a few ulp of scores below 6)."""
    torch = _cuda()
    from hmclab_gb300 import diagnostics

    rng = np.random.default_rng(N + C)
    x = rng.normal(size=(N, d, C)).astype(dtype)
    x[:, -1] = np.round(x[:, -1] * 2) / 2  # ties, and both signs of zero
    flat = x.reshape(-1)
    if flat.size > 8:
        flat[rng.integers(0, flat.size, 2)] = np.inf
        flat[rng.integers(0, flat.size, 2)] = -np.inf
    z = diagnostics.rank_normalize(torch.from_numpy(x).cuda()).cpu().numpy()
    np.testing.assert_allclose(z, O.rank_normalize(x.astype(np.float64)), rtol=0, atol=1e-12)


@pytest.mark.gpu
@pytest.mark.parametrize("draws", [40, 9000])
def test_nan_draws_do_not_move_other_ranks(draws):
    torch = _cuda()
    from hmclab_gb300 import diagnostics

    rng = np.random.default_rng(draws)
    x = rng.normal(size=(draws, 1, 1))
    x[3], x[17] = np.nan, np.nan
    ok = ~np.isnan(x[:, 0, 0])
    z = diagnostics.rank_normalize(torch.from_numpy(x).cuda()).cpu().numpy()[:, 0, 0]
    from scipy.special import ndtri
    from scipy.stats import rankdata

    np.testing.assert_allclose(z[ok], ndtri((rankdata(x[ok, 0, 0]) - 0.375) / (draws + 0.25)), rtol=0, atol=1e-12)
    np.testing.assert_allclose(z[~ok], ndtri((0.5 - 0.375) / (draws + 0.25)), rtol=0, atol=1e-12)


@pytest.mark.gpu
@pytest.mark.parametrize("N,C,lags", [(4, 1, 2), (40, 3, 15), (40, 17, 16), (100, 16, 17), (100, 33, 31), (200, 8, 32),
                                      (200, 8, 33), (200, 9, 49), (300, 2, 112), (768, 3, 200), (770, 3, 130),
                                      (2048, 2, 90), (2051, 2, 90)])
def test_ess_across_lag_rounds(N, C, lags):
    """The estimate does not depend on where a round ends; parameters that
    truncate early, late and not at all share a call (1e-9: FP64 sums of up
    to 1025 products of FP32 values)."""
    torch = _cuda()
    from hmclab_gb300 import diagnostics

    x = ar1(N, 5, C, [0.0, 0.4, 0.8, 0.97, -0.5], seed=N + C).astype(np.float32)
    t = torch.from_numpy(x).cuda()
    e, rh = diagnostics.ess(t, lags=lags, return_rhat=True)
    e_ref, rh_ref = O.ess_split(x.astype(np.float64), min(lags, N // 2))
    np.testing.assert_allclose(e, e_ref, rtol=1e-9)
    np.testing.assert_allclose(rh, rh_ref, rtol=1e-9)
