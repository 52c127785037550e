"""Performance cases of the SVPF engine: the calls its users make, over the range they make them in.

Every case goes through a public entry point of the package (``SVPF``, ``Batch``, ``MultiScale``,
``Stream``, ``svpf_loglik``, ``SVPFParamEstimator``).  ``exact`` restates the first pass of a case in
64-bit torch from the model's equations, with the noise generator (Philox4x32-10, Salmon et al.,
SC'11) restated too.
"""
from __future__ import annotations

import importlib
import importlib.util
import math
import os
import sys

import numpy as np
import torch

# --------------------------------------------------------------------------- the cases


def listed():
    return [
        # one instrument, one observation at a time: the plain single-filter workload of the benchmark
        {"name": "filter_512", "kind": "filter", "n": 512, "knobs": "production", "nu": 30.0},
        # the Python binding's own defaults (400 particles, 8 to 16 Stein iterations, everything adaptive)
        {"name": "filter_400_binding", "kind": "filter", "n": 400, "knobs": "binding", "nu": 30.0},
        # the largest particle count of the scenario sweep, one instrument
        {"name": "filter_4096", "kind": "filter", "n": 4096, "knobs": "production", "nu": 30.0},
        # one two-factor instrument, a count that fills no tile
        {"name": "two_factor_1000", "kind": "two_factor", "n": 1000, "nu": 6.0},
        # a desk's book: some hundred instruments with ragged particle counts, host arrays in and out
        {"name": "batch_300_ragged", "kind": "batch", "filters": 300, "n_lo": 100, "n_hi": 1500, "ragged": True,
         "device": False},
        # the benchmark's batched workload, device arrays, one graph replay per tick
        {"name": "batch_4096", "kind": "batch", "filters": 4096, "n_lo": 256, "n_hi": 4096, "ragged": False,
         "device": True},
        # the two-scale composition (256 reactive and 1024 inertial particles per instrument)
        {"name": "scales_200", "kind": "scales", "instruments": 200, "nr": 256, "ni": 1024},
        # the request loop at its usual round size: a tenth of the fleet has a new observation
        {"name": "requests_200_of_2000", "kind": "requests", "fleet": 2000, "count": 200, "n_lo": 256, "n_hi": 2048,
         "ragged": False},
        # one training step: value and gradient of 256 filters, N = 512, a window of the run
        {"name": "gradient_256x512", "kind": "gradient", "filters": 256, "n": 512, "ticks": 32},
        # the torch estimator's training step, one window of its train() settings
        {"name": "estimator_1", "kind": "estimator", "paths": 1, "n": 64, "steps": 2, "ticks": 250},
        # the same for a minibatch of windows
        {"name": "estimator_1024", "kind": "estimator", "paths": 1024, "n": 64, "steps": 2, "ticks": 250},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["filter", "two_factor", "batch", "scales", "requests", "gradient", "estimator"])
    if kind == "filter":
        return {"kind": kind, "n": _log_int(rng, 100, 4096), "knobs": rng.choice(["production", "binding"]), "nu": 30.0}
    if kind == "two_factor":
        return {"kind": kind, "n": _log_int(rng, 128, 2048), "nu": 6.0}
    if kind == "batch":
        lo = _log_int(rng, 64, 512)
        return {"kind": kind, "filters": _log_int(rng, 32, 1500), "n_lo": lo, "n_hi": lo * rng.randint(2, 8),
                "ragged": rng.random() < 0.7, "device": rng.random() < 0.5}
    if kind == "scales":
        return {"kind": kind, "instruments": _log_int(rng, 10, 400), "nr": rng.choice([128, 200, 256]),
                "ni": rng.choice([512, 777, 1024])}
    if kind == "requests":
        fleet = _log_int(rng, 100, 2000)
        return {"kind": kind, "fleet": fleet, "count": max(1, int(fleet * rng.uniform(0.05, 0.6))), "n_lo": 256,
                "n_hi": rng.choice([1024, 2048]), "ragged": rng.random() < 0.5}
    if kind == "gradient":
        return {"kind": kind, "filters": _log_int(rng, 16, 256), "n": rng.choice([100, 128, 250, 256, 400, 512]),
                "ticks": rng.randint(8, 32)}
    return {"kind": kind, "paths": _log_int(rng, 1, 1024), "n": 2 * rng.randint(16, 64), "steps": rng.randint(1, 3),
            "ticks": rng.randint(100, 250)}


# --------------------------------------------------------------------------- knobs

# svpf_create's defaults with full Newton, up to 8 iterations over 3 annealing stages
PRODUCTION = dict(
    lik_offset=0.45, use_exact_gradient=0, use_svld=1, use_annealing=1, use_adaptive_beta=1, n_anneal_steps=3,
    temperature=1.0, rmsprop_rho=0.9, rmsprop_eps=1e-6, use_mim=1, mim_jump_prob=0.05, mim_jump_scale=5.0,
    use_asymmetric_rho=1, rho_up=0.98, rho_down=0.93, use_guided=0, use_guide=1, use_guide_preserving=1,
    guide_strength=0.05, guide_strength_base=0.05, use_adaptive_guide=0, use_rejuvenation=1, use_newton=1,
    use_full_newton=1, use_adaptive_mu=0, use_adaptive_sigma=0, stein_repulsive_sign=0, stein_min_steps=4,
    stein_max_steps=8)
# the defaults of the reference's Python binding
BINDING = dict(
    PRODUCTION, lik_offset=0.345, use_exact_gradient=1, temperature=0.45, n_anneal_steps=5, mim_jump_prob=0.25,
    mim_jump_scale=9.0, rejuv_ksd_threshold=0.05, use_guided=1, guided_alpha_base=0.0, guided_alpha_shock=0.40,
    guided_innovation_threshold=1.5, use_adaptive_guide=1, guide_strength_max=0.30, guide_innovation_threshold=1.0,
    use_adaptive_mu=1, mu_process_var=0.001, mu_obs_var_scale=11.0, mu_min=-4.0, mu_max=-1.0, use_adaptive_sigma=1,
    sigma_boost_threshold=0.95, sigma_boost_max=3.2, stein_min_steps=8, stein_max_steps=16)
# the two scales of the multiscale composition (the engine sets them itself)
REACTIVE = dict(
    PRODUCTION, lik_offset=0.35, use_exact_gradient=1, temperature=0.55, use_annealing=0, n_anneal_steps=1,
    mim_jump_prob=0.30, mim_jump_scale=10.0, rho_up=0.94, rho_down=0.88, use_guide=0, use_newton=0, use_full_newton=0,
    stein_min_steps=2, stein_max_steps=5)
INERTIAL = dict(BINDING, lik_offset=0.35, n_anneal_steps=3, stein_min_steps=8, stein_max_steps=16)
# the two-factor test's knobs
TWO_FACTOR = dict(
    PRODUCTION, use_newton=0, use_full_newton=0, use_two_factor=1, rho_fast=0.80, sigma_fast=0.30, rho_slow=0.995,
    sigma_slow=0.05, bw_floor_fast=0.01, bw_floor_slow=0.05, n_anneal_steps=5, temperature=0.45, mim_jump_prob=0.25,
    mim_jump_scale=9.0, guide_strength=0.12, use_exact_gradient=1, lik_offset=0.345)
# the differentiable set (grad_config): the model's own rho, a fixed schedule and budget
GRADIENT = dict(
    PRODUCTION, use_asymmetric_rho=0, use_rejuvenation=0, use_adaptive_beta=0, use_exact_gradient=1, stein_min_steps=8,
    stein_max_steps=8)

OBS = 64   # observations a state holds; passes walk through them


def _pkg():
    """The package of the tree we run in (its folder's name is not an identifier)."""
    if "svpf_b200" not in sys.modules:
        folder = os.path.join(os.getcwd(), "newton-stein-variational-particle-filter_b200")
        spec = importlib.util.spec_from_file_location("svpf_b200", os.path.join(folder, "__init__.py"),
                                                      submodule_search_locations=[folder])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["svpf_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["svpf_b200"]


def _config(knobs, steps, nu):
    return _pkg().default_config(steps, nu).update(**knobs)


# --------------------------------------------------------------------------- inputs, from the seed alone


def _sv_paths(rng, T, rho, sz, mu, nu):
    """Returns [T, F] of the one-factor model with Student-t noise."""
    F = len(rho)
    h = mu + sz / np.sqrt(1 - rho ** 2) * rng.standard_normal(F)
    ys = np.empty((T, F), np.float32)
    for t in range(T):
        h = mu + rho * (h - mu) + sz * rng.standard_normal(F)
        ys[t] = np.exp(h / 2) * rng.standard_t(nu)
    return ys


def _two_factor_paths(rng, T, F, mu, nu):
    f = 0.30 / math.sqrt(1 - 0.8 ** 2) * rng.standard_normal(F)
    s = 0.05 / math.sqrt(1 - 0.995 ** 2) * rng.standard_normal(F)
    ys = np.empty((T, F), np.float32)
    for t in range(T):
        f = 0.8 * f + 0.3 * rng.standard_normal(F)
        s = 0.995 * s + 0.05 * rng.standard_normal(F)
        ys[t] = np.exp((mu + f + s) / 2) * rng.standard_t(nu, F)
    return ys


def _counts(rng, case, F):
    lo, hi = case["n_lo"], case["n_hi"]
    if case["ragged"]:
        return np.exp(rng.uniform(math.log(lo), math.log(hi), F)).round().astype(np.int32)
    powers = [lo << k for k in range(16) if lo << k <= hi]
    return rng.choice(powers, F).astype(np.int32)


def _inputs(case, seed):
    rng = np.random.default_rng([seed, 11])
    kind = case["kind"]
    if kind == "filter":
        mu = -1.0 if case["knobs"] == "production" else -3.5
        ys = _sv_paths(rng, OBS, np.array([0.97]), np.array([0.15]), np.array([mu]), np.array([30.0]))[:, 0]
        return {"mu": mu, "gamma": 0.0 if case["knobs"] == "production" else -0.5, "y": ys}
    if kind == "two_factor":
        return {"y": _two_factor_paths(rng, OBS, 1, -3.5, case["nu"])[:, 0]}
    if kind == "batch":
        F = case["filters"]
        rho, sz = rng.uniform(0.90, 0.995, F), rng.uniform(0.05, 0.4, F)
        mu, nu = rng.uniform(-2.0, 0.0, F), rng.uniform(4.0, 30.0, F)
        return {"n": _counts(rng, case, F), "rho": rho, "sz": sz, "mu": mu, "nu": nu,
                "y": _sv_paths(rng, OBS + 1, rho, sz, mu, nu)}
    if kind == "scales":
        F = case["instruments"]
        rho, sz, mu = rng.uniform(0.94, 0.99, F), rng.uniform(0.08, 0.2, F), rng.uniform(-4.0, -2.5, F)
        return {"rho": rho, "sz": sz, "mu": mu, "y": _sv_paths(rng, OBS, rho, sz, mu, np.full(F, 5.0))}
    if kind == "requests":
        F = case["fleet"]
        n = _counts(rng, case, F)
        slots = np.stack([rng.permutation(F)[:case["count"]] for _ in range(8)]).astype(np.int32)
        return {"n": n, "slots": slots, "y": _two_factor_paths(rng, 8, case["count"], -3.5, 6.0)}
    if kind == "gradient":
        F = case["filters"]
        theta = np.stack([rng.uniform(-2, 0, F), rng.uniform(0.9, 0.99, F), rng.uniform(0.1, 0.3, F),
                          rng.uniform(5, 20, F)], 1).astype(np.float32)
        t64 = theta.astype(np.float64)
        return {"theta": theta, "y": _sv_paths(rng, case["ticks"], t64[:, 1], t64[:, 2], t64[:, 0], t64[:, 3]).T.copy()}
    P = case["paths"]
    ys = _sv_paths(rng, case["ticks"], np.full(P, 0.97), np.full(P, 0.15), np.full(P, -3.5), np.full(P, 8.0))
    return {"y": ys.T.copy()}


# --------------------------------------------------------------------------- what a program has in hand before the call


def prepare(case, seed):
    pkg = _pkg()
    kind, x = case["kind"], _inputs(case, seed)
    s = {"kind": kind, "x": x, "t": 0}
    if kind == "filter":
        knobs = PRODUCTION if case["knobs"] == "production" else BINDING
        f = pkg.SVPF(case["n"], knobs["stein_max_steps"] if knobs is PRODUCTION else 8, case["nu"])
        f.configure(**{k: getattr(_config(knobs, 8, case["nu"]), k) for k, _ in pkg.CONFIG_FIELDS})
        f.initialize(0.97, 0.15, x["mu"], x["gamma"], seed=seed)
        s["filter"] = f
    elif kind == "two_factor":
        f = pkg.SVPF(case["n"], 8, case["nu"])
        f.configure(**{k: getattr(_config(TWO_FACTOR, 8, case["nu"]), k) for k, _ in pkg.CONFIG_FIELDS})
        f.initialize(0.995, 0.05, -3.5, 0.0, seed=seed)
        s["filter"] = f
    elif kind == "batch":
        F = case["filters"]
        cfgs = [_config(PRODUCTION, 8, float(v)) for v in x["nu"]]
        prms = [pkg.Params(float(x["rho"][k]), float(x["sz"][k]), float(x["mu"][k]), 0.0) for k in range(F)]
        if case["device"]:
            stream = torch.cuda.Stream()
            s["stream"] = stream
            b = pkg.Batch(x["n"], cfgs, prms, stream=stream.cuda_stream)
            s["y"] = torch.from_numpy(x["y"]).cuda()
            s["y_t"], s["y_prev"] = (torch.zeros(F, device="cuda") for _ in range(2))
            s["out"] = torch.zeros((F, 8), dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
        else:
            b = pkg.Batch(x["n"], cfgs, prms)
        b.initialize(seed)
        s["batch"] = b
    elif kind == "scales":
        F = case["instruments"]
        conf = pkg.lib().svpf_ms_default_config()
        conf.n_particles_reactive, conf.n_particles_inertial = case["nr"], case["ni"]
        m = pkg.MultiScale([pkg.Params(float(x["rho"][k]), float(x["sz"][k]), float(x["mu"][k]), 0.0)
                            for k in range(F)], conf)
        m.init(0.03, seed=seed)
        s["scales"] = m
    elif kind == "requests":
        cfg, prm = _config(TWO_FACTOR, 8, 6.0), pkg.Params(0.995, 0.05, -3.5, 0.0)
        floats = int(((2 * x["n"].astype(np.int64) + 15) // 16 * 16).sum()) * 4
        st = pkg.Stream(case["fleet"], floats * 4 + case["fleet"] * 4096 + 65536, int(x["n"].max()), seed=seed)
        slots = [st.admit(int(n), cfg, prm, seed=seed) for n in x["n"]]
        if slots != list(range(case["fleet"])):
            raise RuntimeError("an instrument was not admitted")
        s["loop"] = st
    elif kind == "gradient":
        ag = importlib.import_module("svpf_b200.autograd")
        s["engine"] = ag.GradEngine([case["n"]] * case["filters"], _config(GRADIENT, 8, 12.0), T_max=case["ticks"])
        s["engine"].set_objective(s["engine"].PREDICTIVE)
        s["loglik"] = ag.svpf_loglik
        s["theta"] = torch.from_numpy(x["theta"]).cuda().requires_grad_(True)
        s["y"] = torch.from_numpy(x["y"]).cuda()
        s["seed"] = seed
    else:
        es = importlib.import_module("svpf_b200.estimator")
        s["model"] = es.SVPFParamEstimator(n_particles=case["n"], n_stein_steps=case["steps"], stein_lr=0.15,
                                           nu=8.0).cuda()
        s["y"] = torch.from_numpy(x["y"]).cuda()
        s["seed"] = seed
    return s


_MS_FLOATS = ("vol_reactive", "vol_inertial", "h_reactive", "h_inertial", "loglik_reactive", "loglik_inertial",
              "vol_combined", "h_combined", "loglik_combined", "transient_magnitude", "ksd_reactive", "ksd_inertial")


def _records(out, ctype, fields):
    """An array of result records as a table of `fields`."""
    names = [f[0] for f in ctype._fields_]
    raw = np.frombuffer(out, dtype=np.int32).reshape(len(out), len(names))
    return raw[:, [names.index(f) for f in fields]]


def run(s):
    """One pass: one observation of every filter, or one training step."""
    kind, x, t = s["kind"], s["x"], s["t"]
    s["t"] = t + 1
    if kind in ("filter", "two_factor"):
        r = s["filter"].step(float(x["y"][t % OBS]))
        return np.array([r.log_lik, r.vol_mean, r.h_mean, r.mu_estimate], np.float32)
    if kind == "batch" and "stream" not in s:
        k = t % OBS
        return s["batch"].step(x["y"][k + 1], x["y"][k])
    if kind == "batch":
        k = t % OBS
        with torch.cuda.stream(s["stream"]):
            s["y_t"].copy_(s["y"][k + 1])
            s["y_prev"].copy_(s["y"][k])
        s["batch"].graph_launch(s["y_t"].data_ptr(), s["y_prev"].data_ptr(), s["out"].data_ptr())
        return s["out"][:, :6].view(torch.float32), s["out"][:, 6:]
    if kind == "scales":
        out = s["scales"].step(x["y"][t % OBS])
        ctype = type(out[0])
        return (_records(out, ctype, _MS_FLOATS).view(np.float32),
                _records(out, ctype, ("stein_steps_reactive", "stein_steps_inertial")))
    if kind == "requests":
        out = s["loop"].process(x["slots"][t % 8], x["y"][t % 8])
        raw = np.frombuffer(out, dtype=np.int32).reshape(len(out), 8)
        return raw[:, :6].view(np.float32), raw[:, 6:]
    if kind == "gradient":
        s["theta"].grad = None
        ll = s["loglik"](s["theta"], s["y"], s["engine"], s["seed"])
        ll.sum().backward()
        return ll.detach(), s["theta"].grad
    model = s["model"]
    model.zero_grad(set_to_none=True)
    nll, vol = model(s["y"], truncate_every=50, burn_in=20, seed=s["seed"])
    nll.backward()
    return nll.detach(), vol, torch.stack([model._rho_logit.grad, model._log_sigma.grad, model._mu.grad])


def work(case):
    """Particle state in and out once, and the method's sums as its equations write them: per pair of one Stein
    iteration an exponential, a reciprocal and 13 operations (vanilla transport: a reciprocal and 6)."""
    kind = case["kind"]

    def fleet(ns, flops_per_pair):
        ns = np.asarray(ns, np.float64)
        return {"bytes": float(28 * ns.sum() + 64 * len(ns)), "flops": float(flops_per_pair * (ns ** 2).sum())}

    if kind == "filter":
        its = 8 if case["knobs"] == "production" else 16
        return fleet([case["n"]], 15 * its)
    if kind == "two_factor":
        return fleet([2 * case["n"]], 7 * 40 / 2)
    if kind == "batch":
        return fleet(_inputs(case, 1)["n"], 15 * 8)
    if kind == "scales":
        a, b = fleet([case["nr"]] * case["instruments"], 9 * 5), fleet([case["ni"]] * case["instruments"], 15 * 16)
        return {k: a[k] + b[k] for k in a}
    if kind == "requests":
        x = _inputs(case, 1)
        return fleet(2 * x["n"][x["slots"][0]], 7 * 40 / 2)
    if kind == "gradient":
        pairs = case["filters"] * case["n"] ** 2 * case["ticks"] * 8.0
        return {"bytes": float(case["filters"] * (8 * case["ticks"] + 32)), "flops": pairs * (15 + 30)}
    pairs = case["paths"] * case["n"] ** 2 * case["ticks"] * float(case["steps"])
    return {"bytes": float(12 * case["paths"] * case["ticks"]), "flops": pairs * (8 + 20)}


# --------------------------------------------------------------------------- the first pass in 64 bits

_M = 0xFFFFFFFF
_D = torch.float64


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _philox(key, ctr):
    k0, k1 = key
    c0, c1, c2, c3 = ctr
    for _ in range(10):
        p0, p1 = c0 * 0xD2511F53, c2 * 0xCD9E8D57          # 64-bit products: the low words wrap as they should
        c0, c1, c2, c3 = ((p1 >> 32) & _M) ^ c1 ^ k0, p1 & _M, ((p0 >> 32) & _M) ^ c3 ^ k1, p0 & _M
        k0, k1 = (k0 + 0x9E3779B9) & _M, (k1 + 0xBB67AE85) & _M
    return c0, c1


class _Noise:
    """Draws of filters `ids` ([B]) with n particles, keyed by (seed, filter), counted by (particle, draw, tick, stream)."""

    def __init__(self, seed, ids, n):
        ids = torch.as_tensor(np.asarray(ids), dtype=torch.int64, device=_dev())[:, None]
        self.key = (torch.full_like(ids, int(seed) & _M), ((int(seed) >> 32) + 0x9E3779B9 * ids) & _M)
        self.i = torch.arange(n, dtype=torch.int64, device=_dev())[None, :].expand(ids.shape[0], n)

    def _bits(self, draw_, tick, stream):
        z = torch.zeros_like(self.i)
        return _philox(self.key, (self.i, z + draw_, z + tick, z + stream))

    def normal(self, draw_, tick, stream=0):
        a, b = self._bits(draw_, tick, stream)
        u1, u2 = ((a >> 8) + 1).to(_D) / 2 ** 24, (b >> 8).to(_D) / 2 ** 24
        return torch.sqrt(-2 * torch.log(u1)) * torch.cos(2 * math.pi * u2)

    def uniform(self, draw_, tick):
        return ((self._bits(draw_, tick, 1)[0] >> 8) + 1).to(_D) / 2 ** 24


def _f(v):
    """A value as the engine holds it (32 bits), in 64."""
    return float(np.float32(v))


def _col(v):
    return torch.as_tensor(np.asarray(v, np.float32).astype(np.float64), device=_dev()).reshape(-1, 1)


def _implied_offset(nu):
    """-E[log t_nu^2] with the asymptotic psi(nu/2)."""
    half = nu / 2
    psi = torch.where(half >= 1, torch.log(half) - 1 / (2 * half) - 1 / (12 * half * half), -0.5772156649 - 1 / half)
    return -(torch.log(nu) - 1.9635100260214235 - psi)


def _normaliser(nu):
    return torch.lgamma((nu + 1) / 2) - torch.lgamma(nu / 2) - 0.5 * torch.log(math.pi * nu)


def _clamp_h(h):
    return h.clamp(-15.0, 5.0)


def _mixture(x, m, s2):
    """Score of the mixture prior at x: -E_w[x - m] / s2, w = softmax of the Gaussian log-densities."""
    d = x[:, :, None] - m[:, None, :]
    w = torch.softmax(-d * d / (2 * s2[:, :, None]), dim=2)
    return -(w * d).sum(2) / s2


def _transport(x, g, c, bw, sign, kind, ksd):
    """Row operator of the IMQ transport (kind 0 vanilla, 2 full Newton) and the rows' KSD terms."""
    n = x.shape[1]
    b = bw[:, :, None]
    u = (x[:, :, None] - x[:, None, :]) / b
    K = 1 / (1 + u * u)
    uK2 = u * K * K
    kg, gk = (K * g[:, None, :]).sum(2), uK2.sum(2)
    phi = (kg + sign * 2 * gk / bw) / n
    if kind == 2:
        nk = (K * K * (3 * u * u - 1).abs()).sum(2)
        H = ((K * c[:, None, :]).sum(2) + 2 * nk / bw ** 2) / K.sum(2).clamp(min=1e-6)
        phi = phi / H.clamp(0.1, 100.0) * 0.7
    rows = None
    if ksd:
        gdk, hs = (uK2 * g[:, None, :]).sum(2), (K * K * (3 - 4 * K)).sum(2)
        rows = g * kg + 2 / bw * (g * gk - gdk) + 2 / bw ** 2 * hs
    return phi, rows


def _iteration(x, v, m, s2, bw, p, c, y2, beta, es, z, last):
    """One Stein iteration: gradient pass, transport, RMSProp and diffusion; the log-weights and KSD rows."""
    nu = p["nu"]
    gp = _mixture(x, m, s2)
    A = y2 / (torch.exp(x.clamp(max=20.0)) + 1e-8) / nu
    lw = p["stc"] - 0.5 * x - (nu + 1) * 0.5 * torch.log1p(A)
    if c["use_exact_gradient"]:
        glik = -0.5 + 0.5 * (nu + 1) * A / (1 + A) - _f(c["lik_offset"])
    else:
        glik = (torch.log(y2 + 1e-10) - x + _f(c["lik_offset"])) / 1.4
    g = (gp + beta * glik).clamp(-10.0, 10.0)
    curv = (0.5 * (nu + 1) * A / (1 + A) ** 2 + 1 / s2).clamp(0.1, 100.0)
    phi, rows = _transport(x, g, curv, bw, 1.0 if c["stein_repulsive_sign"] else -1.0, 2 if c["use_full_newton"] else 0,
                           last)
    v = _f(c["rmsprop_rho"]) * v + (1 - _f(c["rmsprop_rho"])) * phi * phi
    x = _clamp_h(x + es * phi * torch.rsqrt(v + _f(c["rmsprop_eps"])) + math.sqrt(2 * es * _f(c["temperature"])) * z)
    return x, v, lw, rows


def _schedule(c):
    """Iterations of a tick whose previous KSD is unknown (the full budget): (beta, step) each."""
    budget, na = c["stein_max_steps"], c["n_anneal_steps"] if c["use_annealing"] else 1
    base = budget // na
    out = []
    for it in range(budget):
        a = na - 1 if base == 0 else min(it // base, na - 1)
        if not c["use_annealing"]:
            beta = 1.0
        elif c["use_adaptive_beta"]:
            beta = 1.0 if a == na - 1 else min(max(0.30 * (0.5 + 0.5 * (a + 1) / na), 0.1), 1.0)
        else:
            beta = (0.30, 0.65, 1.0)[a % 3]
        beta = _f(beta)
        out.append((beta, 0.1 * (0.5 if c["use_guide"] else 1.0) * math.sqrt(beta)))
    return out


def _start(p, noise):
    """Particles and scalar state of a freshly initialised filter."""
    var = p["sz0"] ** 2 / (1 - p["rho0"] ** 2 + 1e-6)
    x = _clamp_h(p["mu"] + torch.sqrt(var) * noise.normal(0, 0, 2))
    one = torch.ones_like(p["mu"])
    return {"x": x, "v": torch.zeros_like(x), "hbar": -3.5 * one, "bw2": None, "ema": None, "m": p["mu"] * one,
            "P": p["sz"] ** 2 / (1 - p["rho"] ** 2) * one}


def _tick(c, p, s, y, y_prev, noise, t, step):
    """One tick of B filters with a common n: the new state, and its outputs.  p: [B, 1] parameters."""
    x, n = s["x"], s["x"].shape[1]
    mu, rho, sz = p["mu"], p["rho"], p["sz"]
    y2 = y * y
    log_y2 = torch.log(y2 + 1e-8)
    m, P = s["m"], s["P"]
    if c["use_guide"]:
        mp, Pp = mu + rho * (m - mu), rho * rho * P + sz * sz
        K = Pp / (Pp + 6.93 + 1e-8)
        m, P = mp + K * (log_y2 - (mp - p["off"])), (1 - K) * Pp
    lev = p["gamma"] * y_prev / (torch.exp(x / 2) + 1e-8)
    z = noise.normal(0, t)
    means = mu + rho * (x - mu) + lev
    jump = torch.where(noise.uniform(0, t) < _f(c["mim_jump_prob"]), _f(c["mim_jump_scale"]), 1.0)
    up = rho
    if c["use_asymmetric_rho"]:   # no particle has moved before the first tick: h > h_prev nowhere
        up = torch.full_like(rho, _f(c["rho_down"]))
    move = mu + up.clamp(0.0, 0.999) * (x - mu) + lev
    if c["use_guided"]:
        implied = (torch.log(y2 + 1e-10) + p["off"]).clamp(min=-5.0)
        zz = (implied - move) / 2.5 - _f(c["guided_innovation_threshold"])
        ga = _f(c["guided_alpha_base"]) + (_f(c["guided_alpha_shock"]) - _f(c["guided_alpha_base"])) * torch.where(
            zz > 0, torch.tanh(zz), 0.0)
        move = (1 - ga) * move + ga * implied
    x = _clamp_h(move + sz * jump * z)
    lp = p["stc"] - 0.5 * x - (p["nu"] + 1) / 2 * torch.log1p(y2 / (torch.exp(x) + 1e-8) / p["nu"])
    predictive = torch.logsumexp(lp, 1, keepdim=True) - math.log(n)
    if c["use_guide"]:
        gs = _f(c["guide_strength_base"])
        x = _clamp_h((1 - gs) * s["hbar"] + gs * m + (x - s["hbar"]))
    mean = x.mean(1, keepdim=True)
    var = (x * x).mean(1, keepdim=True) - mean * mean
    fresh = (2 * var / math.log(n + 1)).clamp(min=1e-6)
    bw2 = fresh if s["bw2"] is None else 0.3 * fresh + 0.7 * s["bw2"]
    a = y.abs()
    ema = a if s["ema"] is None else 0.05 * a + 0.95 * s["ema"]
    spread = (x.amax(1, keepdim=True) - x.amin(1, keepdim=True)) / 2
    comb = torch.maximum(a / ema.clamp(min=1e-8), spread.clamp(max=2.0))
    bw2 = bw2 * (1 - 0.25 * (comb - 1).clamp(max=2.0)).clamp(0.5, 1.0)
    bw = torch.sqrt(bw2).clamp(0.01, 2.0)
    v, lw, rows = s["v"], None, None
    schedule = _schedule(c)
    for it, (beta, es) in enumerate(schedule):
        x, v, lw, rows = step(x, v, means, sz * sz, bw, p, c, y2, beta, es, noise.normal(1 + it, t),
                              it == len(schedule) - 1)
    hm = x.mean(1, keepdim=True)
    new = {"x": x, "v": v, "hbar": hm, "bw2": bw2, "ema": ema, "m": m, "P": P}
    return new, {"loglik": torch.logsumexp(lw, 1) - math.log(n), "vol": torch.exp(x / 2).mean(1), "h_mean": hm[:, 0],
                 "bw": bw[:, 0], "ksd": torch.sqrt((rows.sum(1) / n ** 2).clamp(min=0.0)),
                 "predictive": predictive[:, 0]}


def _first_tick(c, ids, n, seed, y, y_prev, rho, sz, mu, gamma, nu, rho0=None, sz0=None):
    """The outputs of the first tick of filters `ids`, n particles each."""
    got = []
    most = max(1, int(6e7 // n ** 2))
    for k in range(0, len(ids), most):
        part = slice(k, k + most)
        noise = _Noise(seed, ids[part], n)
        p = {"rho": _col(rho[part]), "sz": _col(sz[part]), "mu": _col(mu[part]), "gamma": _col(gamma[part]),
             "nu": _col(nu[part]), "rho0": _col((rho if rho0 is None else rho0)[part]),
             "sz0": _col((sz if sz0 is None else sz0)[part])}
        p["off"], p["stc"] = _implied_offset(p["nu"]), _normaliser(p["nu"])
        with torch.no_grad():
            got.append(_tick(c, p, _start(p, noise), _col(y[part]), _col(y_prev[part]), noise, 0, _iteration)[1])
    return {k: torch.cat([g[k] for g in got]) for k in got[0]}


def _first_tick_2f(c, ids, n, seed, y, mu, nu):
    """The outputs of a two-factor filter's first tick."""
    got = []
    most = max(1, int(1.2e8 // n ** 2))
    for k in range(0, len(ids), most):
        part = slice(k, k + most)
        noise = _Noise(seed, ids[part], n)
        yt = _col(y[part])
        mu_, nu_ = torch.full_like(yt, _f(mu)), torch.full_like(yt, _f(nu))
        y2 = yt * yt
        rho, sig = [_f(c["rho_fast"]), _f(c["rho_slow"])], [_f(c["sigma_fast"]), _f(c["sigma_slow"])]
        var = [sig[q] ** 2 + rho[q] ** 2 * sig[q] ** 2 / (1 - rho[q] ** 2) for q in range(2)]
        innov = torch.log(y2 + 1e-8) + _implied_offset(nu_) - mu_
        gs = _f(c["guide_strength"])
        prev, x = [], []
        for q in range(2):
            sd = sig[q] / math.sqrt(1 - rho[q] ** 2 + 1e-8)
            prev.append(_clamp_h(sd * noise.normal(1 + q, 0, 2)))
            z = noise.normal(q, 0)
            if q == 0:
                z = z * torch.where(noise.uniform(0, 0) < _f(c["mim_jump_prob"]), _f(c["mim_jump_scale"]), 1.0)
            guide = gs * var[q] / (var[0] + var[1] + 6.93 + 1e-8) * innov   # the previous factor means are zero
            x.append(_clamp_h(guide + _clamp_h(rho[q] * prev[q] + sig[q] * z)))
        bw = []
        for q in range(2):
            mean = x[q].mean(1, keepdim=True)
            sd = torch.sqrt(((x[q] * x[q]).mean(1, keepdim=True) - mean * mean).clamp(min=1e-8))
            bw.append((1.06 * sd * n ** -0.2).clamp(min=_f((c["bw_floor_fast"], c["bw_floor_slow"])[q])))
        v = [torch.zeros_like(x[0]), torch.zeros_like(x[0])]
        s2 = [sig[q] ** 2 + 1e-8 for q in range(2)]
        share = [s2[0] / (s2[0] + s2[1]), 1 - s2[0] / (s2[0] + s2[1])]
        kn, lw = 2, None
        na, steps = c["n_anneal_steps"], 8
        es0 = 0.5 / steps
        sign = 1.0 if c["stein_repulsive_sign"] else -1.0
        for a in range(na):
            beta = (a + 1) / na
            for _ in range(steps):
                h = mu_ + x[0] + x[1]
                ratio = y2 / (nu_ * torch.exp(h) + 1e-8)
                lg = -0.5 + 0.5 * (nu_ + 1) * ratio / (1 + ratio + 1e-8)
                lw = _normaliser(nu_) - 0.5 * h - 0.5 * (nu_ + 1) * torch.log(1 + ratio)
                new = []
                for q in range(2):
                    g = -(x[q] - rho[q] * prev[q]) / s2[q] + beta * share[q] * lg
                    phi = _transport(x[q], g, None, bw[q], sign, 0, False)[0]
                    v[q] = _f(c["rmsprop_rho"]) * v[q] + (1 - _f(c["rmsprop_rho"])) * phi * phi
                    es = es0 * beta
                    new.append(_clamp_h(x[q] + es * phi * torch.rsqrt(v[q] + _f(c["rmsprop_eps"])) +
                                        math.sqrt(2 * es * _f(c["temperature"])) * noise.normal(kn + q, 0)))
                x = new
                kn += 2
        hm = (mu_ + x[0].mean(1, keepdim=True) + x[1].mean(1, keepdim=True))[:, 0]
        got.append({"loglik": torch.logsumexp(lw, 1) - math.log(n), "vol": torch.exp((mu_ + x[0] + x[1]) / 2).mean(1),
                    "h_mean": hm, "bw": bw[0][:, 0], "ksd": torch.zeros_like(hm)})
    return {k: torch.cat([g[k] for g in got]) for k in got[0]}


def _by_count(ns, one):
    """Outputs of filters with different particle counts: one(indices, n) per count, back in order."""
    out = None
    for n in np.unique(ns):
        idx = np.where(ns == n)[0]
        got = one(idx, int(n))
        if out is None:
            out = {k: torch.zeros(len(ns), dtype=_D, device=_dev()) for k in got}
        for k in got:
            out[k][torch.from_numpy(idx).to(_dev())] = got[k]
    return out


def _gradient(case, x, seed):
    """Log-likelihoods and gradient by autograd, each Stein iteration recomputed in the backward."""
    from torch.utils.checkpoint import checkpoint

    def step(*args):
        return checkpoint(_iteration, *args, use_reentrant=False)

    F, n, T = case["filters"], case["n"], case["ticks"]
    lls, grads = [], []
    most = max(1, int(3e7 // n ** 2))
    for k in range(0, F, most):
        part = slice(k, k + most)
        theta = torch.from_numpy(x["theta"][part].astype(np.float64)).to(_dev()).requires_grad_(True)
        y = torch.from_numpy(x["y"][part].astype(np.float64)).to(_dev())
        noise = _Noise(seed, np.arange(F)[part], n)
        p = {"mu": theta[:, 0:1], "rho": theta[:, 1:2], "sz": theta[:, 2:3], "nu": theta[:, 3:4]}
        p.update(rho0=p["rho"], sz0=p["sz"], gamma=torch.zeros_like(p["mu"]), stc=_normaliser(p["nu"]),
                 off=_implied_offset(torch.full_like(p["mu"], 12.0)).detach())
        s, ll = _start(p, noise), []
        for t in range(T):
            s, out = _tick(GRADIENT, p, s, y[:, t:t + 1], y[:, t - 1:t] if t else torch.zeros_like(y[:, :1]), noise, t,
                           step)
            ll.append(out["predictive"])
        ll = torch.stack(ll, 1)
        grads.append(torch.autograd.grad(ll.sum(), theta)[0])
        lls.append(ll.detach())
    return torch.cat(lls), torch.cat(grads)


def _estimator(case, x, seed):
    """The torch estimator's training step, backpropagated window by window (its path is cut every 50 ticks)."""
    P, n, T, S, nu, lr, burn = case["paths"], case["n"], case["ticks"], case["steps"], 8.0, 0.15, 20
    raw = [torch.tensor(v, dtype=torch.float32).to(_dev(), _D).requires_grad_(True)
           for v in (math.log(0.9 / (1 - 0.9 + 1e-8) + 1e-8), math.log(0.15), -3.5)]
    # the parameters' values as the engine gets them, in 32 bits; their derivatives in 64
    rho64, sz64 = 0.5 + 0.499 * torch.sigmoid(raw[0]), torch.nn.functional.softplus(raw[1]) + 0.001
    r32 = [v.detach().float() for v in raw]
    rho32 = (0.5 + 0.499 * torch.sigmoid(r32[0])).to(_D)
    sz32 = (torch.nn.functional.softplus(r32[1]) + 0.001).to(_D)
    leaf = [rho32.clone().requires_grad_(True), sz32.clone().requires_grad_(True), raw[2].detach().clone().requires_grad_(True)]
    rho, sz, mu = leaf
    y = torch.from_numpy(x["y"].astype(np.float64)).to(_dev())
    noise, half = _Noise(seed, np.arange(P), n), _Noise(seed, np.arange(P), n // 2)
    C = math.lgamma((nu + 1) / 2) - math.lgamma(nu / 2) - 0.5 * math.log(nu * math.pi)
    h = mu + sz / torch.sqrt(1 - rho ** 2 + 1e-6) * noise.normal(0, 0, 2)
    nll, vols, grads = 0.0, [], [0.0, 0.0, 0.0]
    window = 0.0

    def close(total):
        if torch.is_tensor(total):
            for q, g in enumerate(torch.autograd.grad(total, leaf, allow_unused=True)):
                if g is not None:
                    grads[q] = grads[q] + g

    for t in range(T):
        if t and t % 50 == 0:
            close(window)
            window, h = 0.0, h.detach()
        e = half.normal(0, t)
        e = torch.cat([e, -e], 1)
        m = mu + rho * (h - mu)
        h = m + sz * e
        yt = y[:, t:t + 1]
        sc = torch.exp(h / 2) + 1e-8
        lp = C - torch.log(sc) - (nu + 1) / 2 * torch.log1p((yt / sc) ** 2 / nu)
        if t >= burn:
            part = -(torch.logsumexp(lp, 1) - math.log(n)).sum() / (P * (T - burn))
            nll, window = nll + part.detach(), window + part
        b = ((h.detach().std(1, unbiased=False, keepdim=True) + 0.1) ** 2 + 1e-8)
        for _ in range(S):
            A = yt * yt / (torch.exp(h) * nu + 1e-8)
            g = (-(h - m) / (sz ** 2 + 1e-8) - 0.5 + (nu + 1) / 2 * A / (1 + A)).clamp(-10, 10)
            d = h[:, :, None] - h[:, None, :]
            K = torch.rsqrt(1 + d * d / b[:, :, None])
            h = h + lr / n * ((K * g[:, None, :]).sum(2) - (d * K ** 3).sum(2) / b)
        vols.append(torch.exp(h / 2).mean(1).detach())
    close(window)
    raw_grads = torch.autograd.grad([rho64, sz64], raw[:2], grad_outputs=[grads[0], grads[1]])
    return nll, torch.stack(vols, 1), torch.stack([raw_grads[0], raw_grads[1], grads[2]])


def exact(case, seed):
    x, kind = _inputs(case, seed), case["kind"]
    names = ("loglik", "vol", "h_mean")
    if kind == "filter":
        c = PRODUCTION if case["knobs"] == "production" else BINDING
        o = _first_tick(c, np.array([0]), case["n"], seed, x["y"][:1], np.zeros(1), np.array([0.97]), np.array([0.15]),
                        np.array([x["mu"]]), np.array([x["gamma"]]), np.array([case["nu"]]))
        mu_est = torch.tensor([x["mu"]], dtype=_D, device=_dev())
        return torch.cat([o[k] for k in names] + [mu_est])
    if kind == "two_factor":
        o = _first_tick_2f(TWO_FACTOR, np.array([0]), case["n"], seed, x["y"][:1], -3.5, case["nu"])
        return torch.cat([o[k] for k in names] + [torch.tensor([-3.5], dtype=_D, device=_dev())])
    if kind == "batch":
        if 8 * (x["n"].astype(np.float64) ** 2).sum() > 4e10:
            return None   # some tens of seconds
        zero = np.zeros(case["filters"])
        o = _by_count(x["n"], lambda i, n: _first_tick(PRODUCTION, i, n, seed, x["y"][1][i], x["y"][0][i], x["rho"][i],
                                                       x["sz"][i], x["mu"][i], zero[i], x["nu"][i]))
        if case["device"]:
            return torch.stack([o[k] for k in ("loglik", "vol", "h_mean", "h_mean", "bw", "ksd")], 1), None
        return [o[k] for k in names]
    if kind == "scales":
        F = case["instruments"]
        ids, one, zero, nu = np.arange(F), np.ones(F), np.zeros(F), np.full(F, 5.0)
        r = _first_tick(REACTIVE, ids, case["nr"], seed, x["y"][0], zero, 0.92 * one, 0.18 * one, x["mu"], zero, nu)
        i = _first_tick(INERTIAL, F + ids, case["ni"], seed, x["y"][0], zero, x["rho"], x["sz"], x["mu"], zero, nu,
                        0.98 * one, 0.10 * one)
        cols = [r["vol"], i["vol"], r["h_mean"], i["h_mean"], r["loglik"], i["loglik"], i["vol"], i["h_mean"],
                i["loglik"], r["vol"] - i["vol"], r["ksd"], i["ksd"]]
        return torch.stack(cols, 1), None
    if kind == "requests":
        slots = x["slots"][0]
        o = _by_count(x["n"][slots], lambda i, n: _first_tick_2f(TWO_FACTOR, slots[i], n, seed, x["y"][0][i], -3.5, 6.0))
        return torch.stack([o[k] for k in ("loglik", "vol", "h_mean", "h_mean", "bw", "ksd")], 1), None
    if kind == "gradient":
        return _gradient(case, x, seed)
    return _estimator(case, x, seed)
