"""Every persistent kernel and launch shape against the warp-per-chain kernel:
the FP32 states are bitwise the same, the FP64 ones agree to the rounding of
their sums, at the edges of rows per lane, unrolled columns, remainders and
cluster parts."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _sampler(d, C, dtype, prior, mass, seed, integrator="lf", streams=None):
    import hmclab_gb300 as H

    rng = np.random.default_rng(seed)
    G = rng.normal(size=(2 * d + 3, d)) / np.sqrt(d)
    m = rng.normal(size=(d, 1))
    lik = H.Distributions.LinearMatrix(G, G @ m + 0.1 * rng.normal(size=(2 * d + 3, 1)), 0.01, dtype=np.float64)
    D = H.Distributions
    post = {"none": lik, "normal": D.BayesRule([D.Normal(np.zeros((d, 1)), np.full((d, 1), 2.0)), lik]),
            "laplace": D.BayesRule([D.Laplace(0.1 * np.ones((d, 1)), np.ones((d, 1))), lik])}[prior]
    mm = None if mass == "unit" else H.MassMatrices.Diagonal(rng.uniform(0.5, 2.0, size=(d, 1)))
    w = np.sqrt(np.linalg.eigvalsh(G.T @ G / 0.01).max() * 2 + 1)
    q0 = m + 0.03 * rng.normal(size=(d, C))
    return H.Samplers.HMC(seed=seed).prepare(
        None, post, stepsize=0.5 / w, amount_of_steps=5, initial_model=q0, proposals=6, chains=C, dtype=dtype,
        mass_matrix=mm, integrator=integrator, proposals_per_graph=6, online_thinning=2, rng_streams=streams)


def _run(smp, shape):
    h = smp.stream.cuda_stream
    smp._load_streams(0, 6)
    smp._persistent._call(6, shape, False, h)
    smp.stream.synchronize()
    return [t.cpu().numpy().copy() for t in (smp.q_cur, smp.x_cur, smp.accepted, smp.ring_q, smp.ring_x)]


@pytest.mark.parametrize("d,C,prior,mass,integrator", [
    (1, 3, "normal", "unit", "lf"), (4, 1, "none", "diag", "lf"), (7, 5, "laplace", "unit", "3s"),
    (16, 9, "normal", "diag", "lf"), (19, 4, "none", "unit", "lf"), (20, 33, "normal", "unit", "4s"),
    (32, 6, "laplace", "diag", "lf"), (33, 2, "normal", "unit", "lf"), (50, 35, "normal", "diag", "3s"),
    (51, 3, "laplace", "unit", "lf"), (52, 5, "none", "diag", "lf"), (64, 17, "normal", "unit", "lf"),
    (67, 2, "laplace", "diag", "lf"), (97, 7, "normal", "unit", "lf"), (128, 5, "normal", "diag", "4s"),
    (70, 2050, "normal", "unit", "lf"), (98, 2049, "laplace", "diag", "lf"), (128, 2051, "none", "unit", "lf")])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_kernels_agree(d, C, prior, mass, integrator, dtype):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hmclab_gb300 import _lib
    from hmclab_gb300._persistent import _lanes_groups

    def fresh():
        return _sampler(d, C, dtype, prior, mass, d + C, integrator)

    ref = _run(fresh(), (_lib.HMC_PERSISTENT_WARPS, 4, 0))
    shapes = [(_lib.HMC_PERSISTENT_LANES, ct, g) for ct in ((1, 2, 4) if dtype == "float32" else (1, 2))
              for g in _lanes_groups(d, C, 4 if dtype == "float32" else 8)]
    shapes += [(_lib.HMC_PERSISTENT_ROWS, r, 0) for r in (1, 2, 4, 8) if dtype == "float64" and (r > 1 or d <= 64)]
    assert 0 < ref[2].sum()
    for shape in shapes:
        got = _run(fresh(), shape)
        assert np.array_equal(got[2], ref[2]), shape
        for k in (0, 3):
            if dtype == "float32":
                assert np.array_equal(got[k], ref[k]), shape
            else:  # 6 proposals of up to 20 products of d terms
                np.testing.assert_allclose(got[k], ref[k], rtol=0, atol=1e-12 * np.abs(ref[k]).max())
        for k in (1, 4):
            np.testing.assert_allclose(got[k], ref[k], rtol=1e-11)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_kernels_agree_on_injected_streams(dtype):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hmclab_gb300 import _lib

    d, C = 13, 6
    rng = np.random.default_rng(0)
    streams = (rng.normal(size=(6, d, C)), rng.uniform(0.5, 1.5, size=(6, C)), rng.uniform(size=(6, C)))
    ref = _run(_sampler(d, C, dtype, "normal", "diag", 3, streams=streams), (_lib.HMC_PERSISTENT_WARPS, 2, 0))
    for shape in ((_lib.HMC_PERSISTENT_LANES, 2, 2),) + (((_lib.HMC_PERSISTENT_ROWS, 2, 0),) if dtype == "float64" else ()):
        got = _run(_sampler(d, C, dtype, "normal", "diag", 3, streams=streams), shape)
        assert np.array_equal(got[2], ref[2])
        np.testing.assert_allclose(got[0], ref[0], rtol=0, atol=0 if dtype == "float32" else 1e-13)
