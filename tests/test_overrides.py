"""Methods replaced on an object, not in a subclass: the batched calls hand them
cleared outputs, and a sum calls them instead of the path that fuses its parts."""
import types

import numpy as np
import pytest
import scipy.sparse as sp

import hmclab_gb300 as H

D = H.Distributions


def _add_one(self, M, out, accumulate, dtype, stream):
    out[0] += 1.0


def _parts():
    d, n = 6, 8
    G = sp.random(n, d, 0.5, random_state=1, format="csr")
    lik = D.LinearMatrix(G, np.ones((n, 1)), 0.5, premultiplication=False)
    return D.Normal(np.zeros((d, 1)), np.ones((d, 1))), D.Laplace(np.zeros((d, 1)), np.ones((d, 1))), lik


def test_the_marks_follow_the_object():
    for t in _parts():
        assert t._fills("_device_gradient") and t._fills("_device_misfit")
        t._device_gradient = types.MethodType(_add_one, t)
        assert not t._fills("_device_gradient") and t._fills("_device_misfit")
        t._device_misfit = lambda *a: None
        assert not t._fills("_device_misfit")
    for prior in _parts()[:2]:
        prior._device_gradient = types.MethodType(_add_one, prior)
        assert prior._row_prior("float32") is None
    prior, _, lik = _parts()

    class Model:  # aligned
        data_ptr = staticmethod(lambda: 0)

    lik._device_gradient = types.MethodType(_add_one, lik)
    assert lik._gradient_with_prior(prior, Model, None, "float32", None) is False


@pytest.mark.gpu
def test_replaced_gradients_are_called():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    M = torch.randn(6, 8, device="cuda")
    one = torch.zeros(6, 8, device="cuda")
    one[0] = 1.0
    prior, laplace, lik = _parts()
    want = lik.gradient_batch(M) + one
    for p in (prior, laplace):
        p._device_gradient = types.MethodType(_add_one, p)
        torch.full((48,), float("nan"), device="cuda")  # freed: the next allocation's memory
        assert torch.equal(p.gradient_batch(M), one)
        assert torch.equal(D.BayesRule([lik, p]).gradient_batch(M), want)
    prior, _, lik = _parts()
    lik._device_gradient = types.MethodType(_add_one, lik)
    assert torch.equal(D.BayesRule([prior, lik]).gradient_batch(M), prior.gradient_batch(M) + one)
