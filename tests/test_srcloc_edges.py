"""The FP32 source location where its event groups (8 per block, up to 8 blocks
per cluster, then rounds), station chunks (512) and chain tiles (32) have their
edges, against FP64 on the host.  A term is a handful of FP32 operations on
numbers of the size of the travel time, the origin time and the observation, so
2^-19 of the sum of these sizes (16 units in the last place each) bounds it."""
import numpy as np
import pytest

import hmclab_gb300 as H


@pytest.mark.gpu
@pytest.mark.parametrize("E,S,C", [(1, 1, 1), (1, 40, 1000), (7, 3, 33), (8, 200, 32), (9, 511, 31), (16, 512, 64), (17, 513, 65),
                                   (64, 10, 40), (65, 7, 33), (130, 5, 3), (3, 1025, 5)])
@pytest.mark.parametrize("infer", [True, False])
def test_against_the_host(E, S, C, infer):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(E * 1000 + S)
    r = rng.uniform(-5.0, 5.0, size=(3, S)).astype(np.float32).astype(np.float64)
    obs = rng.uniform(0.0, 4.0, size=(E, S)).astype(np.float32).astype(np.float64)
    std = rng.uniform(0.5, 2.0, size=(E, S))
    if S > 1:
        obs[0, S // 2] = np.nan
    t = H.Distributions.SourceLocation3D(*(a[None] for a in r), obs, std, infer_velocity=infer,
                                         medium_velocity=None if infer else 3.0)
    M = np.concatenate([rng.uniform(-4.0, 4.0, size=(4 * E, C)), rng.uniform(2.0, 5.0, size=(1, C))])[: t.dimensions]
    M = M.astype(np.float32)
    T = torch.from_numpy(M).cuda()
    x, g = t.misfit_batch(T).cpu().numpy(), t.gradient_batch(T).cpu().numpy()
    g2 = t.gradient_batch(T, out=torch.ones_like(T), accumulate=True).cpu().numpy()

    m = M.astype(np.float64)
    v = m[-1] if infer else np.full(C, 3.0)
    w = (1.0 / std**2).astype(np.float32).astype(np.float64)[:, :, None] * np.isfinite(obs)[:, :, None]
    o = np.nan_to_num(obs)[:, :, None]
    e = m[: 4 * E].reshape(E, 4, C)
    d = [e[:, k, None, :] - r[k][None, :, None] for k in range(3)]
    dist = np.sqrt(sum(a * a for a in d))
    res = e[:, 3, None, :] + dist / v - o
    size = np.abs(e[:, 3, None, :]) + dist / v + np.abs(o)
    tol = 2.0**-19
    want = 0.5 * (w * res**2).sum((0, 1))
    assert np.all(np.abs(x - want) <= tol * (w * size**2).sum((0, 1)))
    rows, bound = np.empty((E, 4, C)), np.empty((E, 4, C))
    for k in range(3):
        rows[:, k] = (w * res * d[k] / dist / v).sum(1)
        bound[:, k] = (w * size / v).sum(1)
    rows[:, 3], bound[:, 3] = (w * res).sum(1), (w * size).sum(1)
    assert np.all(np.abs(g[: 4 * E] - rows.reshape(4 * E, C)) <= tol * bound.reshape(4 * E, C))
    if infer:
        assert np.all(np.abs(g[-1] + (w * res * dist).sum((0, 1)) / v**2) <= tol * (w * size * dist).sum((0, 1)) / v**2)
    assert np.allclose(g2, g + 1.0, rtol=2.0**-22, atol=2.0**-22)
