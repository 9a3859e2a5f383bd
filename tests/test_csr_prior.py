"""A prior's gradient added in the last pass of the sparse product against the two
passes, bit for bit: every kernel and prior, chain counts at the edges of the
four-chain and 32-chain forms, both orders of the parts, further parts, outputs
to accumulate into, unaligned models, and subclasses that override a gradient."""
import numpy as np
import pytest
import scipy.sparse as sp

import hmclab_gb300 as H
from hmclab_gb300 import _csr, _lib

D = H.Distributions


def _parts(kind, n=40, d=90, seed=2):
    rng = np.random.default_rng(seed)
    G = sp.random(n, d, 0.1, random_state=seed, format="lil")
    G[3, :], G[:, 7] = 0.0, 0.0  # a row and a column without entries
    lik = D.LinearMatrix(G.tocsr(), rng.normal(size=(n, 1)), 0.3, premultiplication=False)
    mean, scale = rng.normal(size=(d, 1)), rng.uniform(0.2, 3.0, size=(d, 1))
    return (D.Normal(mean, scale) if kind == 1 else D.Laplace(mean, scale)), lik


def _models(torch, lik, prior, C):
    M = torch.from_numpy(np.random.default_rng(C).normal(size=(lik.dimensions, C))).float().cuda().contiguous()
    M[5] = torch.from_numpy(prior.means[5].astype(np.float32)).cuda()  # on the mean: the Laplace sign is zero
    return M


def _two_passes(prior, lik, M):
    g = prior.gradient_batch(M)
    return lik.gradient_batch(M, out=g, accumulate=True)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [1, 2])
@pytest.mark.parametrize("C", [1, 3, 4, 33, 128, 1028])
def test_every_kernel(kind, C):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    prior, lik = _parts(kind)
    M = _models(torch, lik, prior, C)
    want = _two_passes(prior, lik, M)
    plan = lik._csr_plan(C, M.device, torch.cuda.current_stream().cuda_stream)
    for shape in _csr.candidates(C):
        if shape[0] == _lib.HMC_CSR_SLAB and shape[1] not in (128, 448):
            continue
        plan.desc_gt = plan.gt.descriptor(*shape)
        plan._ref_gt = _lib._ct.byref(plan.desc_gt)
        assert torch.equal(_two_passes(prior, lik, M), want)
        for parts in ([prior, lik], [lik, prior]):
            out = torch.full_like(M, float("nan"))
            assert torch.equal(D.BayesRule(parts).gradient_batch(M, out=out), want), (shape, parts[0])


@pytest.mark.gpu
def test_where_the_two_passes_stay():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    prior, lik = _parts(1)
    C = 64
    M = _models(torch, lik, prior, C)
    want = _two_passes(prior, lik, M)
    post = D.BayesRule([prior, lik])
    # accumulating, a third part, and a model that starts off a 16-byte boundary
    assert torch.equal(post.gradient_batch(M, out=torch.zeros_like(M), accumulate=True), want)
    third = D.Laplace(np.zeros((lik.dimensions, 1)), np.ones((lik.dimensions, 1)))
    assert torch.equal(D.BayesRule([prior, lik, third]).gradient_batch(M), third.gradient_batch(M, out=want.clone(), accumulate=True))
    room = torch.zeros(M.numel() + 1, device="cuda")
    room[1:] = M.reshape(-1)
    off = room[1:].view_as(M)
    if lik._csr_plan(C, M.device, torch.cuda.current_stream().cuda_stream).shape_g[0] != _lib.HMC_CSR_GATHER4:
        assert torch.equal(post.gradient_batch(off), want)
    assert not lik._gradient_with_prior(prior, off, torch.empty_like(M), "float32", torch.cuda.current_stream().cuda_stream)

    class Doubled(D.Normal):
        def _device_gradient(self, M, out, accumulate, dtype, stream):
            super()._device_gradient(M, out, accumulate, dtype, stream)
            out *= 2.0

    class Halved(D.LinearMatrix):
        def _device_gradient(self, M, out, accumulate, dtype, stream):
            pass

    double = Doubled(prior.means, prior.covariance)
    assert double._row_prior("float32") is None
    g = D.BayesRule([double, lik]).gradient_batch(M)
    assert torch.equal(g, lik.gradient_batch(M, out=2.0 * prior.gradient_batch(M), accumulate=True))
    none = Halved(lik.G, lik.d, 0.3, premultiplication=False)
    assert torch.equal(D.BayesRule([prior, none]).gradient_batch(M), prior.gradient_batch(M))
    full = D.Normal(np.zeros((lik.dimensions, 1)), np.eye(lik.dimensions))
    assert full._row_prior("float32") is None
