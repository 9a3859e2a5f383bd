"""The work that programs built on hmclab_gb300 give it, as cases that can be timed.

Most programs prepare a sampler once and then run blocks of proposals; others
evaluate one model at a time through the plugin API, train the learned
gradient, or reduce a finished run to its diagnostics.  Each case prepares
what such a program holds (posterior, sampler state, network, samples) and
`run` is the call that it repeats.

  point          misfit(m) and gradient(m) of one FP64 vector: the plugin API
                 that optimisers and the reference's own scripts call
  chain          a block of proposals of FP64 chains on a small dense linear
                 problem (the reference's single-chain use)
  chain_large    the same on a dense problem of a thousand parameters
  small_chains   thousands of FP32 chains on a small dense problem
  dense          thousands of FP32 chains on a dense problem of a thousand
                 parameters
  tomo           FP32 chains on sparse straight-ray tomography
  srcloc         FP32 chains on a network's earthquake locations, full mass
  srcloc_few     the location gradient of one or a few events
  fwi            elastic waveform misfit gradient of many models at once
  fwi_point      misfit(m) and gradient(m) of one elastic model
  surrogate      one training step of the learned potential, and the
                 gradients it predicts for the next leapfrog step
  diagnostics    ESS, rank-normalised ESS, split-R-hat and moments of a run
"""
import math

import numpy as np
import torch

import hmclab_gb300 as H
from hmclab_gb300 import diagnostics, fwi, problems, surrogate


def listed():
    return [
        # one model at a time: every call is a handful of small launches
        {"name": "point_d50", "kind": "point", "d": 50, "n": 100, "prior": "normal"},
        # the reference's own configuration: one FP64 chain, d = 50
        {"name": "chain_f64_d50", "kind": "chain", "d": 50, "n": 100, "chains": 1, "L": 10, "P": 100,
         "prior": "normal"},
        # one FP64 chain on the large dense problem
        {"name": "chain_f64_d1000", "kind": "chain_large", "d": 1000, "n": 2000, "chains": 1, "L": 10, "P": 2,
         "prior": "normal"},
        # many chains of the small problem
        {"name": "chains_f32_d50", "kind": "small_chains", "d": 50, "n": 100, "chains": 4096, "L": 10, "P": 32,
         "prior": "normal", "mass": "unit"},
        # the benchmark's dense problem
        {"name": "dense_f32_d1000", "kind": "dense", "d": 1000, "n": 2000, "chains": 4096, "L": 20, "P": 2,
         "prior": "normal"},
        # the benchmark's tomography
        {"name": "tomo_64x64", "kind": "tomo", "side": 64, "rays": 2000, "chains": 1024, "L": 20, "P": 1},
        # the benchmark's source location
        {"name": "srcloc_32x200", "kind": "srcloc", "events": 32, "stations": 200, "chains": 8192, "L": 5, "P": 4,
         "velocity": True},
        # a single event with a local network
        {"name": "srcloc_one_event", "kind": "srcloc_few", "events": 1, "stations": 40, "chains": 1000,
         "velocity": True},
        # the benchmark's elastic grid, fewer time steps and shots
        {"name": "fwi_200x100_c64", "kind": "fwi", "nx": 200, "nz": 100, "nt": 300, "shots": 2, "chains": 64,
         "bx": 20, "bz": 10},
        # one elastic model at a time
        {"name": "fwi_point", "kind": "fwi_point", "nx": 100, "nz": 60, "nt": 300, "shots": 2, "bx": 10, "bz": 6},
        # training and prediction at the benchmark's network size
        {"name": "surrogate_d600", "kind": "surrogate", "d": 600, "hidden": 512, "batch": 256, "chains": 64},
        # diagnostics of a run of the elastic benchmark's size
        {"name": "diagnostics_d600", "kind": "diagnostics", "d": 600, "draws": 100, "chains": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["point", "chain", "chain_large", "small_chains", "dense", "tomo", "srcloc", "srcloc_few", "fwi",
                       "fwi_point", "surrogate", "diagnostics"])
    prior = rng.choice(["normal", "laplace"])
    if kind == "point":
        d = _log_int(rng, 2, 300)
        return {"kind": kind, "d": d, "n": d + _log_int(rng, 1, 2 * d), "prior": prior}
    if kind == "chain":
        d = _log_int(rng, 4, 128)
        return {"kind": kind, "d": d, "n": d + _log_int(rng, 2, 2 * d), "chains": _log_int(rng, 1, 16),
                "L": rng.randint(4, 20), "P": rng.randint(20, 120), "prior": prior}
    if kind == "chain_large":
        d = _log_int(rng, 150, 1500)
        return {"kind": kind, "d": d, "n": d + _log_int(rng, 10, d), "chains": _log_int(rng, 1, 4),
                "L": rng.randint(4, 12), "P": rng.randint(1, 3), "prior": prior}
    if kind == "small_chains":
        d = _log_int(rng, 4, 100)
        return {"kind": kind, "d": d, "n": d + _log_int(rng, 2, 2 * d), "chains": _log_int(rng, 64, 8192),
                "L": rng.randint(4, 16), "P": rng.randint(8, 32), "prior": prior,
                "mass": rng.choice(["unit", "diagonal"])}
    if kind == "dense":
        d = _log_int(rng, 140, 1000)
        return {"kind": kind, "d": d, "n": d + _log_int(rng, 10, d), "chains": _log_int(rng, 64, 4096),
                "L": rng.randint(4, 20), "P": rng.randint(1, 2), "prior": prior}
    if kind == "tomo":
        return {"kind": kind, "side": rng.randint(16, 64), "rays": _log_int(rng, 100, 2000),
                "chains": _log_int(rng, 16, 1024), "L": rng.randint(4, 20), "P": 1}
    if kind == "srcloc":
        return {"kind": kind, "events": rng.randint(4, 32), "stations": _log_int(rng, 20, 200),
                "chains": _log_int(rng, 128, 8192), "L": rng.randint(3, 6), "P": rng.randint(1, 4),
                "velocity": rng.random() < 0.5}
    if kind == "srcloc_few":
        return {"kind": kind, "events": rng.randint(1, 3), "stations": _log_int(rng, 6, 200),
                "chains": _log_int(rng, 1, 8192), "velocity": rng.random() < 0.5}
    if kind == "fwi":
        bx, bz = rng.randint(4, 20), rng.randint(2, 10)
        return {"kind": kind, "nx": rng.randint(60, 200), "nz": rng.randint(30, 100), "nt": rng.randint(60, 250),
                "shots": rng.randint(1, 2), "chains": rng.choice([8, 13, 24, 32, 32, 40, 64, 64]), "bx": bx, "bz": bz}
    if kind == "fwi_point":
        bx, bz = rng.randint(3, 12), rng.randint(2, 8)
        return {"kind": kind, "nx": rng.randint(40, 200), "nz": rng.randint(30, 100), "nt": rng.randint(60, 300),
                "shots": rng.randint(1, 2), "bx": bx, "bz": bz}
    if kind == "surrogate":
        return {"kind": kind, "d": rng.randint(40, 600), "hidden": rng.choice([128, 256, 512]),
                "batch": rng.randint(64, 256), "chains": _log_int(rng, 8, 128)}
    d = _log_int(rng, 8, 600)
    draws = rng.randint(20, 200)
    return {"kind": kind, "d": d, "draws": draws, "chains": max(2, min(128, _log_int(rng, 200, 7000) // draws))}


# ---- inputs ------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _f32(a):
    """Values that FP32 holds exactly, so that every precision sees the same problem."""
    return np.asarray(a, np.float32).astype(np.float64)


def _dense_problem(case, seed):
    """G ~ N(0, 1/d), data with noise 0.05, a diagonal mass, chains in equilibrium."""
    d, n, C = case["d"], case["n"], case.get("chains", 1)
    rng = np.random.default_rng(seed)
    G = _f32(rng.standard_normal((n, d), dtype=np.float32) / math.sqrt(d))
    m = rng.normal(size=(d, 1))
    noise = 0.05
    data = _f32(G @ m + noise * rng.normal(size=(n, 1)))
    diag = _f32(rng.uniform(0.5, 2.0, size=(d, 1)))
    q0 = _gaussian_draws(G, data, noise**2, np.zeros((d, 1)), 1.0,
                         rng.standard_normal((d, C), dtype=np.float32))
    # the largest frequency of the posterior (edge of the spectrum of G^T G)
    w2 = (math.sqrt(n / d) + 1.0) ** 2 / noise**2 + 1.0
    return {"G": G, "data": data, "var": noise**2, "diag": diag, "q0": q0, "w2": w2}


def _gaussian_draws(G, data, var, mean, prior_var, z):
    """Draws of a linear problem's posterior under a normal prior: where running chains are."""
    dev = _device()
    G, data, mean, z = (torch.from_numpy(np.asarray(a, np.float64)).to(dev) for a in (G, data, mean, z))
    A = G.T @ G / var + torch.eye(G.shape[1], dtype=torch.float64, device=dev) / prior_var
    chol = torch.linalg.cholesky(A)
    centre = mean + torch.cholesky_solve(G.T @ (data - G @ mean) / var, chol)
    return _f32((centre + torch.linalg.solve_triangular(chol.T, z, upper=True)).cpu().numpy())


def _linear_posterior(p, prior, dtype):
    d = p["G"].shape[1]
    zero, one = np.zeros((d, 1)), np.ones((d, 1))
    pr = H.Distributions.Normal(zero, one) if prior == "normal" else H.Distributions.Laplace(zero, one)
    return H.Distributions.BayesRule([pr, H.Distributions.LinearMatrix(p["G"], p["data"], p["var"], dtype=dtype)])


def _stepsize(w2, diag_min, fraction):
    return float(np.float32(fraction / math.sqrt(w2 / diag_min)))


def _tomo_problem(case, seed):
    t = problems.tomography(case["side"], case["side"], case["rays"], 1.0, 0.01, seed)
    G, bg = t["G"].astype(np.float32).astype(np.float64), _f32(t["background"])
    data = _f32(t["d"])
    diag = _f32(np.asarray(G.power(2).sum(axis=0)).reshape(-1, 1) / 0.01**2 + 1 / 0.05**2)
    rng = np.random.default_rng(seed + 1)
    # largest frequency of the mass-scaled posterior by power iteration
    s = 1.0 / np.sqrt(diag)
    v = rng.normal(size=diag.shape)
    for _ in range(30):
        v = s * (G.T @ (G @ (s * v))) / 0.01**2 + s * s * v / 0.05**2
        w2 = float(np.linalg.norm(v))
        v /= w2
    q0 = _gaussian_draws(G.toarray(), data, 0.01**2, bg, 0.05**2,
                         rng.standard_normal((diag.size, case["chains"]), dtype=np.float32))
    return {"G": G, "data": data, "bg": bg, "diag": diag, "q0": q0, "eps": float(np.float32(0.55 / math.sqrt(w2)))}


_VELOCITY, _PICK_STD = 5.0, 0.0625


def _srcloc_problem(case, seed):
    E, S = case["events"], case["stations"]
    t = problems.source_location(E, S, 40.0, 10.0, _VELOCITY, _PICK_STD, seed)
    rx, ry, rz, obs = (_f32(t[k]) for k in ("rx", "ry", "rz", "obs"))
    m = t["m_true"] if case["velocity"] else t["m_true"][:-1]
    rng = np.random.default_rng(seed + 1)
    ex, ey, ez = (m[k:4 * E:4] for k in range(3))
    dx, dy, dz = ex - rx, ey - ry, ez - rz
    dist = np.sqrt(dx**2 + dy**2 + dz**2)
    d = m.size
    # Gauss-Newton Hessian at the truth, with a little damping for events that
    # a small network does not resolve
    J = np.zeros((E, S, d))
    for e in range(E):
        J[e, :, 4 * e], J[e, :, 4 * e + 1], J[e, :, 4 * e + 2] = (a[e] / (_VELOCITY * dist[e]) for a in (dx, dy, dz))
        J[e, :, 4 * e + 3] = 1.0
        if case["velocity"]:
            J[e, :, -1] = -dist[e] / _VELOCITY**2
    J = J.reshape(E * S, d)
    hess = J.T @ J / _PICK_STD**2 + np.eye(d)
    z = rng.standard_normal((d, case["chains"]), dtype=np.float32)
    q0 = _f32(m + 0.5 * np.linalg.solve(np.linalg.cholesky(hess).T, z))
    return {"rx": rx, "ry": ry, "rz": rz, "obs": obs, "hess": hess, "q0": q0}


def _srcloc(case, p):
    extra = {} if case["velocity"] else {"infer_velocity": False, "medium_velocity": _VELOCITY}
    return H.Distributions.SourceLocation3D(p["rx"], p["ry"], p["rz"], p["obs"], _PICK_STD, **extra)


_PAD, _H, _DT, _F0, _SPONGE, _AMP = 20, 5.0, 5e-4, 25.0, 0.015, 1e9
_TRACE = 4.0e-3  # size of a direct arrival at one grid spacing from an explosion of unit amplitude


def _fwi_geometry(case):
    """Sources and receivers near the surface, spread over the model."""
    width = case["nx"] * _H
    sx = [width * (k + 0.5) / case["shots"] for k in range(case["shots"])]
    rx = np.linspace(25.0, width - 25.0, 20)
    return sx, rx


def _fwi_problem(case, seed):
    sx, rx = _fwi_geometry(case)
    rng = np.random.default_rng(seed)
    C, nb = case.get("chains", 1), case["bx"] * case["bz"]
    # records: a direct arrival per trace and white noise of several times its size
    t = np.arange(case["nt"]) * _DT
    obs = np.empty((2, case["shots"], case["nt"], len(rx)))
    for s, x in enumerate(sx):
        r = np.maximum(np.abs(rx - x), _H)
        a = (np.pi * _F0 * (t[:, None] - 1.2 / _F0 - r / 1800.0)) ** 2
        obs[:, s] = _TRACE * (1.0 - 2.0 * a) * np.exp(-a) / np.sqrt(r / _H)
    std = 10.0 * float(np.sqrt(np.mean(obs**2)))
    obs = _f32(obs + std * rng.standard_normal(obs.shape, dtype=np.float32))
    scale = np.repeat([60.0, 35.0, 40.0], nb)[:, None]
    q = _f32(scale * rng.standard_normal((3 * nb, C), dtype=np.float32))
    return {"sx": sx, "rx": rx, "ux": obs[0], "uz": obs[1], "std": std, "q": q}


def _fwi(case, p):
    cfg = fwi.ElasticConfig(nx=case["nx"], nz=case["nz"], pad=_PAD, h=_H, dt=_DT, nt=case["nt"], f0=_F0, sponge=_SPONGE,
                            amplitude=_AMP, src_x=p["sx"], src_z=10.0, rec_x=p["rx"], rec_z=10.0)
    return H.Distributions.ElasticFullWaveform2D(cfg, p["ux"], p["uz"], data_std=p["std"],
                                                 free_parameter_grid=[case["bx"], case["bz"]])


def _training_pairs(case, seed):
    """Gradients of a potential that is a quadratic plus a smooth bounded part, as FP32 rows."""
    d, n = case["d"], 2048
    rng = np.random.default_rng(seed)
    q = rng.standard_normal((n, d), dtype=np.float32)
    w = rng.uniform(0.5, 3.0, size=d).astype(np.float32)
    g = w * q + np.tanh(q[:, ::-1]) + 0.1 * rng.standard_normal((n, d), dtype=np.float32)
    idx = rng.integers(0, n, size=case["batch"])
    qc = rng.standard_normal((d, case["chains"]), dtype=np.float32)
    return q, g.astype(np.float32), idx, qc


def _samples(case, seed):
    """Autocorrelated draws [N][d][C], each parameter with its own memory."""
    N, d, C = case["draws"], case["d"], case["chains"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    phi = torch.linspace(0.0, 0.9, d, device="cuda")[:, None]
    x = torch.empty((N, d, C), device="cuda")
    x[0] = torch.randn((d, C), generator=gen, device="cuda")
    for k in range(1, N):
        x[k] = phi * x[k - 1] + torch.sqrt(1 - phi**2) * torch.randn((d, C), generator=gen, device="cuda")
    return x


def _sampler(seed, post, case, q0, eps, dtype, mass=None):
    P = case["P"]
    return H.Samplers.HMC(seed=seed).prepare(
        None, post, stepsize=eps, amount_of_steps=case["L"], mass_matrix=mass, initial_model=q0,
        proposals=P * 1_000_000, proposals_per_graph=P, chains=case["chains"], dtype=dtype)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("point", "chain", "chain_large", "small_chains", "dense"):
        p = _dense_problem(case, seed)
        f64 = kind in ("point", "chain", "chain_large")
        post = _linear_posterior(p, case["prior"], np.float64 if f64 else None)
        if kind == "point":
            s.update(post=post, m=p["q0"])
            return s
        mass, diag_min = None, 1.0
        if kind == "dense" or case.get("mass") == "diagonal":
            mass, diag_min = H.MassMatrices.Diagonal(p["diag"]), 0.5
        eps = _stepsize(p["w2"], diag_min, 0.5)
        s["sampler"] = _sampler(seed, post, case, p["q0"], eps, "float64" if f64 else "float32", mass)
        return s
    if kind == "tomo":
        p = _tomo_problem(case, seed)
        prior = H.Distributions.Normal(p["bg"], np.full_like(p["bg"], 0.05**2))
        post = H.Distributions.BayesRule([prior, H.Distributions.LinearMatrix(p["G"], p["data"], 0.01**2)])
        s["sampler"] = _sampler(seed, post, case, p["q0"], p["eps"], "float32", H.MassMatrices.Diagonal(p["diag"]))
        return s
    if kind in ("srcloc", "srcloc_few"):
        p = _srcloc_problem(case, seed)
        post = _srcloc(case, p)
        if kind == "srcloc":
            s["sampler"] = _sampler(seed, post, case, p["q0"], 0.5, "float32", H.MassMatrices.Full(p["hess"]))
        else:
            s.update(post=post, q=torch.from_numpy(p["q0"]).float().cuda().contiguous())
        return s
    if kind in ("fwi", "fwi_point"):
        p = _fwi_problem(case, seed)
        s["post"] = _fwi(case, p)
        if kind == "fwi":
            s["q"] = torch.from_numpy(p["q"]).float().cuda().contiguous()
        else:
            s["m"] = p["q"]
        return s
    if kind == "surrogate":
        q, g, idx, qc = _training_pairs(case, seed)
        d, hidden = case["d"], case["hidden"]
        net = surrogate.PotentialSurrogate(d, hidden=(hidden, hidden), seed=seed)
        data = surrogate.TrainingSet(d, len(q))
        stream = torch.cuda.current_stream().cuda_stream
        columns = [torch.from_numpy(a).cuda().t().contiguous() for a in (q, g)]
        data.record(*columns, stream)
        net.fit_normalization(data)
        qc = torch.from_numpy(qc).cuda().contiguous()
        s.update(net=net, data=data, idx=idx, q=qc, g=torch.empty_like(qc))
        return s
    s["samples"] = _samples(case, seed)
    return s


def run(s):
    kind = s["case"]["kind"]
    if "sampler" in s:
        smp = s["sampler"]
        smp.run(s["case"]["P"])
        return {"q": smp.q_cur, "x": smp.x_cur, "accepted": smp.accepted}
    if kind in ("point", "fwi_point"):
        return {"misfit": s["post"].misfit(s["m"]), "gradient": s["post"].gradient(s["m"])}
    if kind in ("srcloc_few", "fwi"):
        return {"gradient": s["post"].gradient_batch(s["q"])}
    if kind == "surrogate":
        net = s["net"]
        loss = net.train_step(s["data"], s["idx"], lr=1e-3)
        net.predict_into(s["q"], s["g"], torch.cuda.current_stream().cuda_stream)
        return {"loss": loss[:1], "params": net.params, "grads": net.grads, "predicted": s["g"]}
    ess, rhat = diagnostics.ess(s["samples"], return_rhat=True)
    bulk, rank_rhat = diagnostics.ess(s["samples"], return_rhat=True, rank_normalize=True)
    mean, std = diagnostics.moments(s["samples"])
    return {"ess": ess, "rhat": rhat, "bulk": bulk, "rank_rhat": rank_rhat, "mean": mean, "std": std}


# ---- what a pass cannot do without -----------------------------------------
def work(case):
    kind = case["kind"]
    C = case.get("chains", 1)
    if kind == "point":
        d = case["d"]
        return {"bytes": 8.0 * (d * d + 8 * d), "flops": 4.0 * d * d + 10.0 * d}
    if kind in ("chain", "chain_large", "small_chains", "dense"):
        d, n, L, P = case["d"], case["n"], case["L"], case["P"]
        e = 8.0 if kind in ("chain", "chain_large") else 4.0
        # the matrix and the chains' positions in, positions and misfits out
        return {"bytes": e * (d * d + 6 * d) + C * (2 * e * d + 24.0) + (e * n * d if kind == "dense" else 0.0),
                "flops": P * C * (2.0 * d * d * L + (2.0 * n * d if kind == "dense" else 2.0 * d * d)
                                  + 8.0 * d * L + 60.0 * d)}
    if kind == "tomo":
        d, n = case["side"] ** 2, case["rays"]
        nnz = 1.1 * case["side"] * n
        return {"bytes": 8.0 * nnz + 8.0 * n + 20.0 * d + C * (8.0 * d + 24.0),
                "flops": case["P"] * C * (nnz * (4.0 * case["L"] + 2.0) + 10.0 * d * case["L"] + 60.0 * d)}
    if kind in ("srcloc", "srcloc_few"):
        E, S = case["events"], case["stations"]
        d = 4 * E + int(case["velocity"])
        if kind == "srcloc_few":
            return {"bytes": 8.0 * E * S + 12.0 * S + 8.0 * d * C, "flops": 23.0 * C * E * S}
        return {"bytes": 8.0 * E * S + 12.0 * S + 8.0 * d * d + C * (8.0 * d + 24.0),
                "flops": case["P"] * C * (case["L"] * (23.0 * E * S + 2.0 * d * d) + 12.0 * E * S + 6.0 * d * d)}
    if kind in ("fwi", "fwi_point"):
        cells = (case["nx"] + 2 * _PAD) * (case["nz"] + 2 * _PAD)
        nb = case["bx"] * case["bz"]
        steps = float(case["nt"]) * case["shots"]
        forwards = 1 if kind == "fwi" else 2
        # the models, records and gradients; the forward wavefield at every
        # step is kept for the adjoint (written and read once)
        return {"bytes": 4.0 * (2 * 3 * nb * C + 2 * steps * 20 + 2 * nb * cells) + 16.0 * steps * cells * C,
                "flops": steps * cells * C * (50.0 * forwards + 90.0) + 12.0 * cells * nb * C}
    if kind == "surrogate":
        d, h, B = case["d"], case["hidden"], case["batch"]
        weights = h * d + h * h + 3 * h
        per_row = 2.0 * (h * d + h * h + h * h + h * d + d * d)
        return {"bytes": 28.0 * weights + 4.0 * d * d + 8.0 * B * d + 8.0 * d * C,
                "flops": B * per_row * 3.0 + C * per_row}
    N, d = case["draws"], case["d"]
    half, S = N // 2, N * C
    lags = max(2, min(half, 200))
    pairs = sum(half - t for t in range(lags))
    return {"bytes": 4.0 * N * d * C + 8.0 * 6 * d,
            "flops": 2 * 2.0 * pairs * 2 * C * d + 2.0 * S * math.log2(max(S, 2)) * d + 4.0 * N * C * d}


# ---- the same in 64 bits, without the package --------------------------------
def _philox(c0, c1, c2, c3, k0, k1):
    """Philox4x32-10 (Salmon et al. 2011) on int64 tensors that hold 32-bit words."""
    mask = 0xFFFFFFFF
    for r in range(10):
        a, b = c0 * 0xD2511F53, c2 * 0xCD9E8D57
        c0, c1, c2, c3 = ((b >> 32) & mask) ^ c1 ^ k0, b & mask, ((a >> 32) & mask) ^ c3 ^ k1, a & mask
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return c0, c1, c2, c3


def _unit(hi, lo):
    return (((hi << 21) ^ (lo >> 11)).double() + 0.5) / 9007199254740992.0


def _random(seed, d, C, n, single, device):
    """Momentum normals [d][C], step factors and accept uniforms [C] of proposal n."""
    key = (seed & 0xFFFFFFFF, seed >> 32)
    quads = (d + 3) // 4
    qi = torch.arange(quads, device=device)[:, None].expand(quads, C)
    ci = torch.arange(C, device=device)[None, :].expand(quads, C)
    zero = torch.zeros_like(qi)
    r = _philox(qi, ci, zero + n, zero, *key)
    if single:
        u = [((w >> 8).double() + 0.5) / 16777216.0 for w in r]
    else:
        s = _philox(qi, ci, zero + n, zero + 0x08000000, *key)
        u = [_unit(r[0], r[1]), _unit(r[2], r[3]), _unit(s[0], s[1]), _unit(s[2], s[3])]
    a, b = torch.sqrt(-2.0 * torch.log(u[0])), torch.sqrt(-2.0 * torch.log(u[2]))
    t, v = 2.0 * math.pi * u[1], 2.0 * math.pi * u[3]
    z = torch.stack([a * torch.cos(t), a * torch.sin(t), b * torch.cos(v), b * torch.sin(v)], 1)
    c = torch.arange(C, device=device)
    o = torch.zeros_like(c)
    w = _philox(o, c, o + n, o + (1 << 28), *key)
    return z.reshape(4 * quads, C)[:d], 0.5 + _unit(w[0], w[1]), _unit(w[2], w[3])


def _hmc(case, seed, q0, eps, single, misfit, gradient, draw_p, velocity):
    """One block of proposals (position Verlet, Metropolis) of every chain."""
    dev = _device()
    q = torch.from_numpy(q0).to(dev)
    d, C = q.shape
    x = misfit(q)
    accepted = torch.zeros(C, dtype=torch.int64, device=dev)
    for n in range(case["P"]):
        z, f, u = _random(seed, d, C, n, single, dev)
        e = eps * f
        p = draw_p(z)
        h0 = x + 0.5 * (p * velocity(p)).sum(0)
        m = q + 0.5 * e * velocity(p)
        for k in range(case["L"]):
            p = p - e * gradient(m)
            m = m + (1.0 if k < case["L"] - 1 else 0.5) * e * velocity(p)
        xm = misfit(m)
        ok = torch.exp(h0 - xm - 0.5 * (p * velocity(p)).sum(0)) > u
        q, x = torch.where(ok, m, q), torch.where(ok, xm, x)
        accepted += ok
    return {"q": q, "x": x, "accepted": accepted}


def _linear_exact(p, prior):
    dev = _device()
    G, data = torch.from_numpy(p["G"]).to(dev), torch.from_numpy(p["data"]).to(dev)

    def misfit(q):
        r = G @ q - data
        return 0.5 * (r * r).sum(0) / p["var"] + (0.5 * (q * q).sum(0) if prior == "normal" else q.abs().sum(0))

    def gradient(q):
        return G.T @ (G @ q - data) / p["var"] + (q if prior == "normal" else torch.sign(q))

    return misfit, gradient


def _location_exact(case, p):
    dev = _device()
    E = case["events"]
    rx, ry, rz, obs = (torch.from_numpy(p[k]).to(dev) for k in ("rx", "ry", "rz", "obs"))

    def parts(q):
        ev = q[:4 * E].reshape(E, 4, -1)
        v = q[4 * E] if case["velocity"] else torch.full_like(q[0], _VELOCITY)
        dx, dy, dz = (ev[:, k, None] - r.reshape(1, -1, 1) for k, r in enumerate((rx, ry, rz)))
        dist = torch.sqrt(dx * dx + dy * dy + dz * dz)
        return dx, dy, dz, dist, v, ev[:, 3, None] + dist / v - obs[:, :, None]

    def misfit(q):
        return 0.5 * (parts(q)[5] ** 2).sum((0, 1)) / _PICK_STD**2

    def gradient(q):
        dx, dy, dz, dist, v, r = parts(q)
        r = r / _PICK_STD**2
        g = torch.stack([(r * a / (dist * v)).sum(1) for a in (dx, dy, dz)] + [r.sum(1)], 1).reshape(4 * E, -1)
        return torch.cat([g, -(r * dist).sum((0, 1))[None] / v**2]) if case["velocity"] else g

    return misfit, gradient


def _in_chunks(f, q, size):
    return torch.cat([f(c) for c in torch.split(q, size, dim=1)], dim=-1)


def _elastic_exact(case, p):
    """Misfit [C] and its gradient [3 nb][C] by automatic differentiation."""
    dev = _device()
    nx, nz, nb = case["nx"], case["nz"], case["bx"] * case["bz"]
    X, Z = np.meshgrid((np.arange(nx) + 0.5) * _H, (np.arange(nz) + 0.5) * _H)
    dx, dz = (X.max() - X.min()) / case["bx"], (Z.max() - Z.min()) / case["bz"]
    B = np.stack([np.exp(-2.0 * (((X - X.min() - (i + 0.5) * dx) / dx) ** 2 + ((Z - Z.min() - (j + 0.5) * dz) / dz) ** 2))
                  for i in range(case["bx"]) for j in range(case["bz"])], -1)
    depth = nz * _H
    vp = np.where(Z < 0.3 * depth, 1800.0, np.where(Z < 0.6 * depth, 2200.0, 2600.0))
    back = (vp, vp / 1.8, 310.0 * vp**0.25)
    NX, NZ = nx + 2 * _PAD, nz + 2 * _PAD
    jj, ii = np.clip(np.arange(NZ) - _PAD, 0, nz - 1), np.clip(np.arange(NX) - _PAD, 0, nx - 1)
    B = torch.from_numpy(B[jj][:, ii].reshape(NZ * NX, nb)).to(dev)
    back = [torch.from_numpy(f[jj][:, ii].reshape(-1, 1)).to(dev) for f in back]
    edge = np.minimum(np.minimum(np.arange(NX), NX - 1 - np.arange(NX))[None, :],
                      np.minimum(np.arange(NZ), NZ - 1 - np.arange(NZ))[:, None]).astype(float)
    taper = torch.from_numpy(np.exp(-((_SPONGE * np.maximum(_PAD - edge, 0.0)) ** 2))[..., None]).to(dev)
    t = np.arange(case["nt"]) * _DT
    a = (np.pi * _F0 * (t - 1.2 / _F0)) ** 2
    pulse = _AMP * (1.0 - 2.0 * a) * np.exp(-a) * _DT / _H**2
    cell = lambda x: _PAD + int(round(x / _H - 0.5))  # noqa: E731
    rec = torch.tensor([cell(x) for x in p["rx"]], device=dev)
    zs = cell(10.0)
    obs = [torch.from_numpy(np.ascontiguousarray(p[k])).to(dev) for k in ("ux", "uz")]

    def shifted(f, axis, k):  # f[. + k] on the interior cells
        sl = [slice(2, -2), slice(2, -2)]
        n = f.shape[axis]
        sl[axis] = slice(2 + k, n - 2 + k)
        return f[sl[0], sl[1]]

    def forward_diff(f, axis):
        return (9 / 8 * (shifted(f, axis, 1) - shifted(f, axis, 0)) - (shifted(f, axis, 2) - shifted(f, axis, -1)) / 24) / _H

    def backward_diff(f, axis):
        return (9 / 8 * (shifted(f, axis, 0) - shifted(f, axis, -1)) - (shifted(f, axis, 1) - shifted(f, axis, -2)) / 24) / _H

    def inner(f):
        return f[2:-2, 2:-2]

    def outer(f):
        return torch.nn.functional.pad(f, (0, 0, 2, 2, 2, 2))

    tin = inner(taper)

    def one(m):
        C = m.shape[1]
        fields = [(b + B @ m[k * nb:(k + 1) * nb]).reshape(NZ, NX, C) for k, b in enumerate(back)]
        vp, vs, rho = fields
        nxt = lambda f, axis: torch.cat([f.narrow(axis, 1, f.shape[axis] - 1), f.narrow(axis, f.shape[axis] - 1, 1)], axis)  # noqa: E731
        mu = rho * vs * vs
        lam = rho * vp * vp - 2 * mu
        bx, bz = 0.5 * (1 / rho + 1 / nxt(rho, 1)), 0.5 * (1 / rho + 1 / nxt(rho, 0))
        mux = 0.25 * (mu + nxt(mu, 1) + nxt(mu, 0) + nxt(nxt(mu, 1), 0))
        l2m = inner(lam + 2 * mu) * _DT
        lam, bx, bz, mux = (inner(f) * _DT for f in (lam, bx, bz, mux))
        total = torch.zeros(C, dtype=torch.float64, device=dev)
        for s, x in enumerate(p["sx"]):
            src = torch.zeros((NZ, NX, 1), dtype=torch.float64, device=dev)
            src[zs, cell(x)] = 1.0
            src = inner(src)
            vx, vz, sxx, szz, sxz = (torch.zeros((NZ, NX, C), dtype=torch.float64, device=dev) for _ in range(5))
            for n in range(case["nt"]):
                vx = outer((inner(vx) + bx * (forward_diff(sxx, 1) + backward_diff(sxz, 0))) * tin)
                vz = outer((inner(vz) + bz * (backward_diff(sxz, 1) + forward_diff(szz, 0))) * tin)
                total = total + ((vx[zs, rec] - obs[0][s, n][:, None]) ** 2).sum(0) \
                    + ((vz[zs, rec] - obs[1][s, n][:, None]) ** 2).sum(0)
                exx, ezz = backward_diff(vx, 1), backward_diff(vz, 0)
                f = src * float(pulse[n])
                sxx = outer((inner(sxx) + l2m * exx + lam * ezz + f) * tin)
                szz = outer((inner(szz) + lam * exx + l2m * ezz + f) * tin)
                sxz = outer((inner(sxz) + mux * (forward_diff(vx, 0) + forward_diff(vz, 1))) * tin)
        return 0.5 * total / p["std"] ** 2

    xs, gs = [], []
    q = torch.from_numpy(p["q"]).to(dev)
    size = max(1, int(1.2e11 / (case["nt"] * case["shots"] * NX * NZ * 8 * 40)))
    for m in torch.split(q, size, dim=1):
        m = m.clone().requires_grad_(True)
        x = one(m)
        x.sum().backward()
        xs.append(x.detach())
        gs.append(m.grad)
    return torch.cat(xs), torch.cat(gs, 1)


def _surrogate_exact(case, seed):
    dev = _device()
    q, g, idx, qc = _training_pairs(case, seed)
    d, h = case["d"], case["hidden"]
    rng = np.random.default_rng(seed)
    start = {}
    for name, bound, shape in (("W1", d**-0.5, (h, d)), ("b1", d**-0.5, (h,)), ("W2", h**-0.5, (h, h)),
                               ("b2", h**-0.5, (h,)), ("w3", 0.1 * h**-0.5, (h,))):
        start[name] = torch.from_numpy(_f32(rng.uniform(-bound, bound, size=shape))).to(dev).requires_grad_(True)
    q, g = torch.from_numpy(q).double().to(dev), torch.from_numpy(g).double().to(dev)
    mu, sq, sg = q.mean(0), q.std(0), g.std(0)
    x = (q - mu) / sq
    # ridge least-squares gradient of a quadratic, symmetrised
    x1 = torch.cat([x, torch.ones_like(x[:, :1])], 1)
    reg = 1e-3 * len(x) * torch.eye(d + 1, dtype=torch.float64, device=dev)
    reg[-1, -1] = 0.0
    sol = torch.linalg.solve(x1.T @ x1 + reg, x1.T @ (g * sq))
    A, beta = 0.5 * (sol[:d].T + sol[:d]), sol[d]
    gelu = torch.nn.functional.gelu

    def field(P, x, create):
        x = x.detach().requires_grad_(True)
        f = gelu(gelu(x @ P["W1"].T + P["b1"]) @ P["W2"].T + P["b2"]) @ P["w3"]
        return torch.autograd.grad(f.sum(), x, create_graph=create)[0] + x.detach() @ A + beta

    rows = torch.from_numpy(idx).to(dev)
    err = (field(start, x[rows], True) / sq - g[rows]) / sg
    loss = 0.5 * (err**2).sum(1).mean()
    grads = dict(zip(start, torch.autograd.grad(loss, list(start.values()))))
    params = {k: start[k].detach() - 1e-3 * grads[k] / (grads[k].abs() + 1e-8) for k in start}
    y = field(params, (torch.from_numpy(qc).double().to(dev).T - mu) / sq, False) / sq
    return {"loss": loss.detach()[None], "params": params, "grads": grads, "predicted": y.T.detach()}


def _ess_exact(x):
    """Split-chain ESS (Geyer's initial monotone sequence) and split-R-hat of [N][d][C]."""
    N, d, C = x.shape
    n = N // 2
    h = torch.cat([x[:n], x[n:2 * n]], 2)  # n, d, 2C
    M, lags = 2 * C, max(2, min(n, 200))
    mean = h.mean(0)
    r = h - mean
    gamma = torch.stack([(r[:n - t] * r[t:]).sum(0).mean(1) / n for t in range(lags)])  # lags, d
    W = gamma[0] * n / (n - 1)
    between = n * mean.var(1)
    var = (n - 1) / n * W + between / n
    rho = (1.0 - (W - gamma) / var).T.cpu().numpy()
    out = np.empty(d)
    for i in range(d):
        total, last, cut = 0.0, math.inf, False
        for t in range(0, lags - 1, 2):
            pair = rho[i, t] + rho[i, t + 1]
            if pair < 0:
                cut = True
                break
            last = min(last, pair)
            total += last
        out[i] = (1.0 if cut else -1.0) * M * n / (2.0 * total - 1.0)
    return out, torch.sqrt(var / W).cpu().numpy()


def _scores_exact(x):
    """Normal scores of the pooled ranks, ties averaged."""
    N, d, C = x.shape
    v = x.permute(1, 0, 2).reshape(d, N * C).contiguous()
    order = torch.sort(v, dim=1).values
    rank = 0.5 * (torch.searchsorted(order, v) + torch.searchsorted(order, v, right=True) + 1).double()
    return torch.special.ndtri((rank - 0.375) / (N * C + 0.25)).reshape(d, N, C).permute(1, 0, 2).contiguous()


def exact(case, seed):
    kind = case["kind"]
    dev = _device()
    if kind in ("point", "chain", "chain_large", "small_chains", "dense"):
        p = _dense_problem(case, seed)
        misfit, gradient = _linear_exact(p, case["prior"])
        if kind == "point":
            q = torch.from_numpy(p["q0"]).to(dev)
            return {"misfit": misfit(q)[0].item(), "gradient": gradient(q)}
        diag, diag_min = torch.ones_like(torch.from_numpy(p["diag"])).to(dev), 1.0
        if kind == "dense" or case.get("mass") == "diagonal":
            diag, diag_min = torch.from_numpy(p["diag"]).to(dev), 0.5
        return _hmc(case, seed, p["q0"], _stepsize(p["w2"], diag_min, 0.5), kind in ("small_chains", "dense"), misfit,
                    gradient, lambda z: torch.sqrt(diag) * z, lambda v: v / diag)
    if kind == "tomo":
        p = _tomo_problem(case, seed)
        G = torch.from_numpy(p["G"].toarray()).to(dev)
        data, bg, diag = (torch.from_numpy(p[k]).to(dev) for k in ("data", "bg", "diag"))

        def misfit(q):
            return 0.5 * ((G @ q - data) ** 2).sum(0) / 0.01**2 + 0.5 * ((q - bg) ** 2).sum(0) / 0.05**2

        def gradient(q):
            return G.T @ (G @ q - data) / 0.01**2 + (q - bg) / 0.05**2

        return _hmc(case, seed, p["q0"], p["eps"], True, misfit, gradient, lambda z: torch.sqrt(diag) * z,
                    lambda v: v / diag)
    if kind in ("srcloc", "srcloc_few"):
        p = _srcloc_problem(case, seed)
        misfit, gradient = _location_exact(case, p)
        if kind == "srcloc_few":
            return {"gradient": _in_chunks(gradient, torch.from_numpy(p["q0"]).to(dev), 1024)}
        hess = torch.from_numpy(p["hess"]).to(dev)
        chol, inv = torch.linalg.cholesky(hess), torch.linalg.inv(hess)
        return _hmc(case, seed, p["q0"], 0.5, True, lambda q: _in_chunks(misfit, q, 1024),
                    lambda q: _in_chunks(gradient, q, 1024), lambda z: chol @ z, lambda v: inv @ v)
    if kind in ("fwi", "fwi_point"):
        x, g = _elastic_exact(case, _fwi_problem(case, seed))
        return {"gradient": g} if kind == "fwi" else {"misfit": x[0].item(), "gradient": g}
    if kind == "surrogate":
        return _surrogate_exact(case, seed)
    x = _samples(case, seed).double()
    ess, rhat = _ess_exact(x)
    bulk, rank_rhat = _ess_exact(_scores_exact(x))
    return {"ess": ess, "rhat": rhat, "bulk": bulk, "rank_rhat": rank_rhat, "mean": x.mean((0, 2)),
            "std": x.var((0, 2), unbiased=False).sqrt()}
