"""Every target writes all of its output when it does not accumulate: outputs
that hold NaN before the call come out as those that held zeros, and the batched
calls, which then hand out uncleared memory, return the same."""
import numpy as np
import pytest
import scipy.sparse as sp

import hmclab_gb300 as H
from hmclab_gb300 import fwi as FW

D = H.Distributions


def _targets():
    rng = np.random.default_rng(5)
    d, n = 7, 11
    G, obs = rng.normal(size=(n, d)), rng.normal(size=(n, 1))
    S = sp.random(n, d, 0.3, random_state=3).tolil()
    S[2, :], S[:, 4] = 0.0, 0.0  # a row and a column without entries
    A = rng.normal(size=(d, d))
    normal = D.Normal(np.zeros((d, 1)), np.ones((d, 1)))
    loc = [rng.normal(size=(1, 6)) for _ in range(3)]
    seen = rng.normal(size=(2, 6))
    seen[0, 3] = np.nan
    cfg = FW.ElasticConfig(nx=30, nz=20, pad=6, h=5.0, dt=5e-4, nt=20, f0=25.0, sponge=0.05, src_x=(60.0,), src_z=12.0,
                           rec_x=(30.0, 90.0), rec_z=17.0)
    u = rng.normal(size=(1, 20, 2))
    return {
        "normal": normal,
        "normal_full": D.Normal(np.zeros((d, 1)), A @ A.T + np.eye(d)),
        "laplace": D.Laplace(np.zeros((d, 1)), np.ones((d, 1))),
        "uniform": D.Uniform(-9 * np.ones((d, 1)), 9 * np.ones((d, 1))),
        "dense": D.LinearMatrix(G, obs, 0.5),
        "dense_residual": D.LinearMatrix(G, obs, 0.5, premultiplication=False),
        "sparse": D.LinearMatrix(S.tocsr(), obs, 0.5, premultiplication=False),
        "sparse_premultiplied": D.LinearMatrix(S.tocsr(), obs, 0.5, premultiplication=True),
        "location": D.SourceLocation3D(*loc, seen, 0.1, infer_velocity=True),
        "sum": D.BayesRule([normal, D.LinearMatrix(G, obs, 0.5)]),
        "fwi": D.ElasticFullWaveform2D(cfg, u, u, data_std=1.0, free_parameter_grid=[3, 2]),
        "fwi_cells": D.ElasticFullWaveform2D(cfg, u, u, data_std=1.0),
    }


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(_targets()))
@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("C", [1, 5, 64])
def test_outputs_are_written(name, dtype, C):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    t = _targets()[name]
    if name.startswith("fwi") and dtype == "float64":
        pytest.skip("FP32 kernels only")
    rng = np.random.default_rng(1)
    M = torch.from_numpy(1.0 + 0.1 * rng.normal(size=(t.dimensions, C))).to("cuda", getattr(torch, dtype)).contiguous()
    for call, shape, kind in ((t.misfit_batch, (C,), torch.float64), (t.gradient_batch, (t.dimensions, C), M.dtype)):
        zero = call(M, out=torch.zeros(shape, dtype=kind, device="cuda"))
        nan = call(M, out=torch.full(shape, float("nan"), dtype=kind, device="cuda"))
        torch.full((4 * t.dimensions * C,), float("nan"), dtype=kind, device="cuda")  # freed: the next allocation's memory
        assert bool(torch.isfinite(zero).all())
        assert torch.equal(zero, nan) and torch.equal(zero, call(M))


@pytest.mark.gpu
def test_a_subclass_keeps_cleared_outputs():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")

    class Part(D.Normal):
        def _device_gradient(self, M, out, accumulate, dtype, stream):
            out[0] += 1.0

    part = Part(np.zeros((3, 1)), np.ones((3, 1)))
    M = torch.ones((3, 4), device="cuda")
    torch.full((12,), float("nan"), device="cuda")
    for t in (part, D.BayesRule([part])):
        g = t.gradient_batch(M)
        assert torch.equal(g, torch.tensor([[1.0], [0.0], [0.0]], device="cuda").expand(3, 4))
    # no part at all: zeros, as before
    assert D.BayesRule([part])._fills("_device_misfit") and not part._fills("_device_gradient")
