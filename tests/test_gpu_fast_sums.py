"""The batch tick's fast sums (csrc/svpf_fast.cuh) against the FP64 oracle.

A filter of 257 particles or more that has no forced tile takes its Stein
iterations through interpolated panels instead of the sweeps over all pairs.
One tick from made states, at sizes around the tiles' and bins' edges, where
that path branches: a smooth cloud, one point (a single panel, equal
particles), two clusters many sigma apart (mixture sums that do not
interpolate), far outliers and particles at the position clamp (the shared
edge panels), a shock that moves the particles away from the prior means (far
points), and a spread that does not fit the tables (the sweeps finish the
tick).  Tolerance as in the randomised runs: 1e-4 relative (floor 1; KSD
1e-3), or four times what the oracle's own FP32 mirror deviates on the same
state and on that state moved by two FP32 ulps.
"""
import concurrent.futures as cf
import os

import numpy as np
import pytest

import tape
from test_gpu_batch_parity import _twin
from test_oracle import TOL, rel_err

pytestmark = pytest.mark.gpu

STATES = ["cloud", "point", "clusters", "outliers", "clamped", "shock", "spread"]
SIZES = [257, 300, 512, 777, 1025, 2049, 4096]


def _state(kind, n, rng, mu):
    if kind == "point":
        h = np.full(n, mu)
    elif kind == "clusters":
        h = np.where(np.arange(n) % 3 == 0, mu + 2.0, mu - 1.0) + 0.02 * rng.standard_normal(n)
    elif kind == "spread":
        h = rng.uniform(-15.0, 5.0, n)
    else:
        h = mu + (0.1 if kind == "shock" else 0.5) * rng.standard_normal(n)
        if kind == "outliers":
            h[:: 23] = rng.uniform(-14.0, 4.5, len(h[:: 23]))
        if kind == "clamped":
            h[:: 3] = -15.0
    return np.clip(h, -15.0, 5.0).astype(np.float32)


@pytest.mark.parametrize("newton", [1, 0])
@pytest.mark.parametrize("sigma", [0.05, 0.3])
def test_fast_sums_match_oracle(pkg, oracle_mod, newton, sigma):
    ns = [n for n in SIZES for _ in STATES] + [8192]
    kinds = STATES * len(SIZES) + ["spread"]
    F, n_max = len(ns), max(ns)
    cfg = pkg.production_config(8.0, 5)
    cfg.update(use_newton=newton, use_full_newton=newton, stein_min_steps=4, stein_max_steps=5)
    params = [(0.95, sigma, -1.0, -0.2 if f % 2 else 0.0) for f in range(F)]
    b = pkg.Batch(ns, [cfg] * F, [pkg.Params(*p) for p in params])
    b.initialize(seed=3)
    rng = np.random.default_rng(17)
    y = np.empty(F, np.float32)
    for f in range(F):
        ctl = b.get_state(f)[0]
        ctl.timestep, ctl.ksd_prev, ctl.ksd_last, ctl.vol_prev = 12, 0.6, 0.6, 0.6
        ctl.guide_initialized, ctl.h_mean_prev, ctl.bw_sq = 1, -1.0, 0.04
        ctl.return_ema, ctl.return_var = 0.5, 0.3
        h = _state(kinds[f], ns[f], rng, -1.0)
        v = rng.uniform(0.05, 0.5, ns[f]).astype(np.float32)
        b.set_state(f, ctl, h, (h - 0.1).astype(np.float32), v, np.zeros(ns[f], np.float32))
        y[f] = 25.0 if kinds[f] == "shock" else 0.4 + 0.05 * (f % 7)
    nrm, uni = tape.tape(5, 0, n_max, 16, 2)
    b.set_noise_tape(nrm, uni)
    yp = np.full(F, 0.3, np.float32)
    twins = [_twin(oracle_mod, b, f, cfg, params[f]) for f in range(F)]
    mirrors = []
    for nudge in (0.0, 2.0 ** -22, -(2.0 ** -22)):
        m = [_twin(oracle_mod, b, f, cfg, params[f], 1) for f in range(F)]
        for o in m:
            o.h = o.h * (1.0 + nudge)
        mirrors.append(m)
    ll, vol, hm = b.step(y, yp)
    ctl = b.ctl()
    with cf.ThreadPoolExecutor(max_workers=min(16, os.cpu_count() or 1)) as pool:
        def step(m):
            return list(pool.map(lambda f: m[f].step(y[f], yp[f], nrm[:, :ns[f]], uni[:, :ns[f]]), range(F)))
        want, around = step(twins), [step(m) for m in mirrors]
    for f in range(F):
        tag = (kinds[f], ns[f])
        assert ctl[f].status == 0 and ctl[f].stein_steps_used == want[f].steps_used, tag
        dev = max(rel_err(m[f].h, twins[f].h) for m in mirrors)
        got = b.get_particles(f)
        assert rel_err(got, twins[f].h) < max(TOL, 4 * dev), (tag, rel_err(got, twins[f].h), dev)
        for name, value, base in (("loglik", ll[f], TOL), ("vol", vol[f], TOL), ("h_mean", hm[f], TOL),
                                  ("ksd", ctl[f].ksd_last, 1e-3)):
            w = getattr(want[f], name)
            dev = max(abs(getattr(a[f], name) - w) for a in around) / max(1.0, abs(w))
            assert abs(value - w) < max(base, 4 * dev) * max(1.0, abs(w)), (tag, name, value, w, dev)
    b.close()


@pytest.mark.parametrize("newton", [1, 0])
@pytest.mark.parametrize("kind", STATES)
def test_single_filter_fast_sums_match_oracle(pkg, oracle_mod, newton, kind):
    """The same for a single filter, whose cluster shares the sums: sizes
    around the first that takes them, ones that leave a member fewer slots
    than the others, and a spread that makes all members turn to the sweeps."""
    ns = [2047, 2048, 2049, 3001, 4096] + ([8192] if kind in ("cloud", "spread") else [])
    cfg = pkg.production_config(8.0, 5)
    cfg.update(use_newton=newton, use_full_newton=newton, stein_min_steps=4, stein_max_steps=5)
    for n in ns:
        rng = np.random.default_rng(n)
        f = pkg.SVPF(n, 5, 8.0)
        f.configure(**cfg.to_dict())
        f.initialize(0.95, 0.05, -1.0, -0.2, seed=3)
        ctl = f.get_state()[0]
        ctl.timestep, ctl.ksd_prev, ctl.ksd_last, ctl.vol_prev = 12, 0.6, 0.6, 0.6
        ctl.guide_initialized, ctl.h_mean_prev, ctl.bw_sq = 1, -1.0, 0.04
        ctl.return_ema, ctl.return_var = 0.5, 0.3
        h = _state(kind, n, rng, -1.0)
        v = rng.uniform(0.05, 0.5, n).astype(np.float32)
        f.set_state(ctl, h, (h - 0.1).astype(np.float32), v, np.zeros(n, np.float32))
        nrm, uni = tape.tape(5, 0, n, 16, 2)
        f.set_noise_tape(nrm, uni)
        twin = _twin(oracle_mod, _One(f), 0, cfg, (0.95, 0.05, -1.0, -0.2))
        mirrors = []
        for nudge in (0.0, 2.0 ** -22, -(2.0 ** -22)):
            o = _twin(oracle_mod, _One(f), 0, cfg, (0.95, 0.05, -1.0, -0.2), 1)
            o.h = o.h * (1.0 + nudge)
            mirrors.append(o)
        y = 25.0 if kind == "shock" else 0.4
        rc, out = f.step_raw(y, 0.3)
        with cf.ThreadPoolExecutor(max_workers=4) as pool:
            want, *around = pool.map(lambda o: o.step(y, 0.3, nrm, uni), [twin] + mirrors)
        ctl, got = f.get_state()[:2]
        assert rc == 0 and ctl.status == 0 and ctl.stein_steps_used == want.steps_used, n
        dev = max(rel_err(m.h, twin.h) for m in mirrors)
        assert rel_err(got, twin.h) < max(TOL, 4 * dev), (n, rel_err(got, twin.h), dev)
        for name, value, base in (("loglik", out.loglik, TOL), ("vol", out.vol, TOL), ("h_mean", out.h_mean, TOL),
                                  ("ksd", ctl.ksd_last, 1e-3)):
            w = getattr(want, name)
            dev = max(abs(getattr(a, name) - w) for a in around) / max(1.0, abs(w))
            assert abs(value - w) < max(base, 4 * dev) * max(1.0, abs(w)), (n, name, value, w, dev)
        f.close()


class _One:
    """A single filter's state in the form that a batch gives it."""

    def __init__(self, f):
        self.f = f

    def get_state(self, _):
        return self.f.get_state()


@pytest.mark.parametrize("exact", [1, 0])
def test_two_factor_fast_sums_match_oracle(pkg, oracle_mod, exact):
    """The same for the two-factor tick's transports: both factors of made
    states, a spread of the slow factor over its floored bandwidth included
    (its step sweeps over the pairs)."""
    sizes = [257, 300, 513, 1025, 2048]
    kinds2 = ["cloud", "point", "outliers", "clamped", "spread"]
    ns = [n for n in sizes for _ in kinds2] + [4096]
    kinds = kinds2 * len(sizes) + ["outliers"]
    F, n_max = len(ns), max(ns)
    cfg = pkg.default_config(2, 6.0)
    cfg.update(use_two_factor=1, rho_fast=0.80, sigma_fast=0.30, rho_slow=0.97, sigma_slow=0.10, bw_floor_fast=0.01,
               bw_floor_slow=0.05, use_svld=1, use_annealing=1, n_anneal_steps=3, temperature=0.45, use_mim=1,
               mim_jump_prob=0.25, mim_jump_scale=9.0, use_guide=1, guide_strength=0.12, use_exact_gradient=exact)
    params = [(0.95, 0.1, -3.0, 0.0)] * F
    b = pkg.Batch(ns, [cfg] * F, [pkg.Params(*p) for p in params])
    b.initialize(seed=3)
    rng = np.random.default_rng(23)
    for f in range(F):
        ctl = b.get_state(f)[0]
        h = np.concatenate([_state(kinds[f], ns[f], rng, 0.0), _state(kinds[f], ns[f], rng, 0.2)])
        v = rng.uniform(0.05, 0.5, 2 * ns[f]).astype(np.float32)
        b.set_state(f, ctl, h, (h - 0.1).astype(np.float32), v, np.zeros(ns[f], np.float32))
    y = (0.2 + 0.02 * np.arange(F)).astype(np.float32)
    nrm, uni = tape.tape(9, 0, n_max, 24, 2)
    b.set_noise_tape(nrm, uni)
    yp = np.zeros(F, np.float32)
    twins = [_twin(oracle_mod, b, f, cfg, params[f]) for f in range(F)]
    mirrors = []
    for nudge in (0.0, 2.0 ** -22, -(2.0 ** -22)):
        m = [_twin(oracle_mod, b, f, cfg, params[f], 1) for f in range(F)]
        for o in m:
            o.h = o.h * (1.0 + nudge)
        mirrors.append(m)
    ll, vol, hm = b.step(y, yp)
    ctl = b.ctl()
    with cf.ThreadPoolExecutor(max_workers=min(16, os.cpu_count() or 1)) as pool:
        def step(m):
            return list(pool.map(lambda f: m[f].step(y[f], yp[f], nrm[:, :ns[f]], uni[:, :ns[f]]), range(F)))
        want, around = step(twins), [step(m) for m in mirrors]
    for f in range(F):
        tag = (kinds[f], ns[f])
        assert ctl[f].status == 0, tag
        dev = max(rel_err(m[f].h, twins[f].h) for m in mirrors)
        got = b.get_particles(f)
        assert rel_err(got, twins[f].h) < max(TOL, 4 * dev), (tag, rel_err(got, twins[f].h), dev)
        for name, value in (("loglik", ll[f]), ("vol", vol[f]), ("h_mean", hm[f])):
            w = getattr(want[f], name)
            dev = max(abs(getattr(a[f], name) - w) for a in around) / max(1.0, abs(w))
            assert abs(value - w) < max(TOL, 4 * dev) * max(1.0, abs(w)), (tag, name, value, w, dev)
    b.close()
