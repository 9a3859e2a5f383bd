"""Per-chain sums and the launch-per-step sampler over the tile shapes they
choose between: fewer than 32 chains, ragged tiles, rows that fill one block or
a cluster, and chain counts with and without 16-byte rows."""
import numpy as np
import pytest


def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.gpu
@pytest.mark.parametrize("d,C", [(1, 1), (5, 1), (129, 1), (1000, 2), (17, 3), (600, 7), (4097, 31), (3, 32), (64, 33),
                                 (1025, 100), (4096, 1024), (130, 8192)])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("kind", ["normal", "laplace"])
def test_prior_sums_and_gradients(d, C, dtype, kind):
    torch = _cuda()
    from hmclab_gb300 import Distributions as D

    rng = np.random.default_rng(d + C)
    mean, w = rng.normal(size=(d, 1)).astype(dtype), rng.uniform(0.5, 2.0, size=(d, 1)).astype(dtype)
    q = rng.normal(size=(d, C)).astype(dtype)
    q[rng.integers(0, d), rng.integers(0, C)] = mean[0, 0]
    q[rng.integers(0, d), rng.integers(0, C)] = np.float32(1e-41)  # subnormal in FP32
    post = D.Normal(mean.astype(float), w.astype(float)) if kind == "normal" else D.Laplace(mean.astype(float), w.astype(float))
    iw = (1.0 / w.astype(float)).astype(dtype)
    if kind == "normal":
        r = mean - q
        x, g = 0.5 * (r.astype(float) * (iw * r).astype(float)).sum(0), -(iw * r)
    else:
        x, g = (np.abs(q - mean) * iw).astype(float).sum(0), np.sign(q - mean) * iw
    M = torch.from_numpy(q).cuda()
    # FP64 sums of d terms that the reference above forms with the same roundings
    np.testing.assert_allclose(post.misfit_batch(M).cpu().numpy(), x, rtol=2.3e-16 * (d + 4))
    assert np.array_equal(post.gradient_batch(M).cpu().numpy(), g)
    twice = post.gradient_batch(M, out=torch.from_numpy(g.copy()).cuda(), accumulate=True)
    assert np.array_equal(twice.cpu().numpy(), g + g)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("mass", ["unit", "diagonal", "full"])
@pytest.mark.parametrize("d", [6, 70])
def test_chains_do_not_depend_on_the_batch(dtype, mass, d):
    """Chain c draws from its own counter, so it is the same chain in every
    batch: 16-byte rows and others, one lane group per chain and full tiles."""
    _cuda()
    import hmclab_gb300 as H

    rng = np.random.default_rng(d)
    lower, upper = -1.2 * np.ones((d, 1)), 1.5 * np.ones((d, 1))
    post = H.Distributions.Normal(rng.normal(size=(d, 1)), rng.uniform(0.2, 2.0, size=(d, 1)), lower_bounds=lower,
                                  upper_bounds=upper)
    q0 = rng.uniform(-1, 1, size=(d, 70))
    a = rng.normal(size=(d, d))
    m = {"unit": None, "diagonal": H.MassMatrices.Diagonal(rng.uniform(0.5, 2, size=(d, 1))),
         "full": H.MassMatrices.Full(np.eye(d) + 0.1 * a @ a.T / d)}[mass]
    runs = {}
    for C in (1, 3, 4, 32, 33, 70):
        runs[C] = H.Samplers.HMC(seed=4).sample(
            None, post, stepsize=0.15, amount_of_steps=4, initial_model=q0[:, :C], proposals=6, chains=C, dtype=dtype,
            mass_matrix=m, persistent=False, keep_samples=True).samples_numpy()
    for C, got in runs.items():
        if mass == "full" and dtype == "float64":  # its products sum in another order for few chains
            np.testing.assert_allclose(got[:, :d], runs[70][:C, :d], rtol=1e-11, atol=1e-12)
        else:
            assert np.array_equal(got[:, :d], runs[70][:C, :d]), C
        np.testing.assert_allclose(got[:, d], runs[70][:C, d], rtol=1e-11)
